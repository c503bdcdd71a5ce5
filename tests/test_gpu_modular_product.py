"""The modular tensor-core product at the edges of its tiles (128 x 128), K slices (64) and
exact chunks (512), through a two-site contraction with local dimension one: the FP64 path
takes it from 2.5 M multiply-adds.

Tolerance: its stated bound, 4 K max_k |a_ik| max_k |b_kj| 2^-T in either part with
T = min(57, (122 - ceil log2 K) // 2), and one rounding of the result."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


@pytest.fixture(scope="module")
def ctx():
    import tngpu
    return tngpu.context()


def product(ctx, A, B):
    (m, k), n = A.shape, B.shape[1]
    Af, Bf = np.asfortranarray(A.astype(complex)), np.asfortranarray(B.astype(complex))
    one, out = np.ones(1, complex), np.zeros((m, n), dtype=np.complex128, order="F")
    ctx.check(ctx.lib.tn_gate2_apply(ctx.h, m, k, n, 1, dp(Af), dp(Bf), dp(one), dp(out)))
    return out


def check(ctx, A, B):
    k = A.shape[1]
    T = min(57, (122 - int(np.ceil(np.log2(k)))) // 2)
    big = lambda x, ax: np.maximum(abs(x.real), abs(x.imag)).max(axis=ax)  # noqa: E731
    ref = A.astype(np.clongdouble) @ B.astype(np.clongdouble)
    got = product(ctx, A, B)
    tol = 4 * k * np.outer(big(A, 1), big(B, 0)) * 2.0 ** -T + 2.0 ** -52 * abs(ref) + 1e-300
    assert np.all(abs((got - ref).real) <= tol) and np.all(abs((got - ref).imag) <= tol)


@pytest.mark.parametrize("m,n,k", [(127, 129, 153), (128, 128, 153), (129, 257, 80), (130, 200, 512), (200, 131, 513),
                                   (64, 96, 1100), (300, 40, 700), (16, 4100, 40), (513, 300, 17), (16, 16, 10000)])
def test_random(ctx, m, n, k):
    r = np.random.default_rng(m + n + k)
    z = lambda *s: r.standard_normal(s) + 1j * r.standard_normal(s)  # noqa: E731
    check(ctx, z(m, k), z(k, n))


@pytest.mark.parametrize("k", [128, 512, 513, 1300])
def test_constant_operands(ctx, k):
    """Residue products of one sign: the largest sums the exact accumulation has to hold."""
    r = np.random.default_rng(k)
    for _ in range(4):
        a, b, c, d = (float(x) for x in r.integers(1, 1 << 50, 4))
        check(ctx, np.full((140, k), a + 1j * b), np.full((k, 150), c - 1j * d))


def test_rows_over_the_range(ctx):
    r = np.random.default_rng(3)
    m, n, k = 150, 140, 160
    A = r.standard_normal((m, k)) * 10.0 ** r.uniform(-120, 120, (m, 1)) * 10.0 ** r.uniform(-12, 0, (m, k)) + 0j
    B = r.standard_normal((k, n)) * 10.0 ** r.uniform(-120, 120, (1, n)) * (1 + 1j)
    A[7], B[:, 5] = 0.0, 0.0
    check(ctx, A, B)
    D = np.full((m, k), 2.0 ** -1070 + 0j)
    assert np.all(product(ctx, D, np.full((k, n), 2.0 ** 60 + 0j)) == k * 2.0 ** -1010)


def test_infinities_and_nan_stay_in_their_row_and_column(ctx):
    r = np.random.default_rng(4)
    m, n, k = 150, 140, 160
    A, B = r.standard_normal((m, k)) + 0j, r.standard_normal((k, n)) + 0j
    clean = product(ctx, A, B)
    A[3, 8], B[9, 11] = np.inf, np.nan
    got = product(ctx, A, B)
    assert not np.isfinite(got[3]).any() and np.isnan(got[:, 11]).all()
    keep = np.ones((m, n), bool)
    keep[3], keep[:, 11] = False, False
    assert np.array_equal(got[keep], clean[keep])
