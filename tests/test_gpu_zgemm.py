"""The FP64 complex product (tn_gemm) at the edges of its three kernels: the
per-output one, the modular tensor-core one (tiles of 128 x 128, K slices of
64, exact chunks of 512) and their dispatch, against extended-precision sums.

Tolerance: the tensor-core path rounds every entry to T bits below its row's
(column's) largest power of two, T = min(57, (122 - ceil log2 K) // 2), forms
the product of those integers exactly and rounds once, so an output is within
4 K amax bmax 2^-T + 2^-52 |C| (two operands, two products per part); the
per-output kernel sums K terms, K 2^-52 sum |a||b| at most."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import tngpu
    return tngpu.context()


def gemm(ctx, A, B, conj_a):
    m, k = (A.shape[1], A.shape[0]) if conj_a else A.shape
    n = B.shape[1]
    dp = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    Af, Bf = (np.asfortranarray(x.astype(np.complex128)) for x in (A, B))
    out = np.zeros((m, n), dtype=np.complex128, order="F")
    ctx.check(ctx.lib.tn_gemm(ctx.h, m, n, k, dp(Af), int(conj_a), dp(Bf), dp(out), 0))
    return out


def check(ctx, A, B, conj_a):
    opA = A.conj().T if conj_a else A
    k = opA.shape[1]
    ref = opA.astype(np.clongdouble) @ B.astype(np.clongdouble)
    got = gemm(ctx, A, B, conj_a)
    T = min(57, (122 - int(np.ceil(np.log2(k)))) // 2)
    big = lambda x, ax: np.maximum(abs(x.real), abs(x.imag)).max(axis=ax)  # noqa: E731
    tc = 4 * k * np.outer(big(opA, 1), big(B, 0)) * 2.0 ** -T + 2.0 ** -52 * abs(ref)
    simt = k * 2.0 ** -52 * (abs(opA) @ abs(B))
    err = np.abs(got - ref).astype(float)
    assert np.all(err <= np.maximum(tc, simt) + 1e-300), float((err / (np.maximum(tc, simt) + 1e-300)).max())


SIZES = [(1, 1, 1), (3, 5, 2), (4, 4, 4000), (16, 16, 1024), (47, 64, 64), (127, 129, 153),
         (128, 128, 153), (129, 257, 65), (130, 200, 512), (200, 131, 513), (64, 96, 1100),
         (300, 40, 700), (16, 4100, 40), (513, 300, 17)]


@pytest.mark.parametrize("m,n,k", SIZES)
@pytest.mark.parametrize("conj_a", [False, True])
def test_gemm_random(ctx, m, n, k, conj_a):
    r = np.random.default_rng(m + 7 * n + k)
    z = lambda *s: r.standard_normal(s) + 1j * r.standard_normal(s)  # noqa: E731
    check(ctx, z(k, m) if conj_a else z(m, k), z(k, n), conj_a)


@pytest.mark.parametrize("k", [64, 512, 513, 1300])
def test_gemm_constant_operands(ctx, k):
    """Equal entries give every residue product one sign: the largest sums
    the exact accumulation has to hold."""
    r = np.random.default_rng(k)
    for _ in range(6):
        a, b, c, d = (float(x) for x in r.integers(1, 1 << 50, 4))
        check(ctx, np.full((140, k), a + 1j * b), np.full((k, 150), c - 1j * d), False)


def test_gemm_graded_and_extreme_rows(ctx):
    """Rows and columns over the FP64 range, zero rows, entries graded inside
    a row, denormals."""
    r = np.random.default_rng(3)
    m, n, k = 150, 140, 160
    A = r.standard_normal((m, k)) * 10.0 ** r.uniform(-120, 120, (m, 1)) * 10.0 ** r.uniform(-12, 0, (m, k)) + 0j
    B = r.standard_normal((k, n)) * 10.0 ** r.uniform(-120, 120, (1, n)) * (1 + 1j)
    A[7] = 0.0
    B[:, 5] = 0.0
    A[9, 1:] = 0.0
    check(ctx, A, B, False)
    got = gemm(ctx, A, B, False)
    assert np.all(got[7] == 0) and np.all(got[:, 5] == 0)
    D = np.full((m, k), 2.0 ** -1070 + 0j)
    assert np.all(gemm(ctx, D, np.full((k, n), 2.0 ** 60 + 0j), False) == k * 2.0 ** -1010)


def test_gemm_infinities_and_nan_stay_in_their_row_and_column(ctx):
    r = np.random.default_rng(4)
    m, n, k = 150, 140, 160
    A, B = r.standard_normal((m, k)) + 0j, r.standard_normal((k, n)) + 0j
    clean = gemm(ctx, A, B, False)
    A[3, 8], B[9, 11] = np.inf, np.nan
    got = gemm(ctx, A, B, False)
    assert not np.isfinite(got[3]).any() and np.isnan(got[:, 11]).all()
    keep = np.ones((m, n), bool)
    keep[3], keep[:, 11] = False, False
    assert np.array_equal(got[keep], clean[keep])
