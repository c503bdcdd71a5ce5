"""Products and splits of graded operands on both sides of the size from which the
tensor cores take them.

tn_gemm in FP64: every output within K 2^-52 of sum_k |a_ik| |b_kj| (two roundings a
term), also where large entries of one side meet small ones of the other along K.

The truncated split of D Q, D diagonal over up to twelve decades and Q unitary: every
singular value to 64 n 2^-52, as the vectors are unit vectors to rounding and the product of
them with the matrix is what has to keep the small ones."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


@pytest.fixture(scope="module")
def ctx():
    import tngpu
    return tngpu.context()


@pytest.mark.parametrize("m,n,k", [(5, 7, 300), (64, 48, 40), (150, 140, 256), (513, 300, 65), (100, 90, 2000)])
@pytest.mark.parametrize("decades", [4, 12])
@pytest.mark.parametrize("conj_a", [False, True])
def test_gemm_graded_along_k(ctx, m, n, k, decades, conj_a):
    r = np.random.default_rng(m + k)
    z = lambda *s: r.standard_normal(s) + 1j * r.standard_normal(s)  # noqa: E731
    lam = 10.0 ** (decades * (r.random(k) - 0.5))
    A, B = z(m, k) * lam, z(k, n) / lam[:, None]
    Af, Bf = np.asfortranarray(A.conj().T if conj_a else A), np.asfortranarray(B)
    out = np.zeros((m, n), dtype=np.complex128, order="F")
    ctx.check(ctx.lib.tn_gemm(ctx.h, m, n, k, dp(Af), int(conj_a), dp(Bf), dp(out), 0))
    ref = A.astype(np.clongdouble) @ B.astype(np.clongdouble)
    assert np.all(abs(out - ref) <= k * EPS * (abs(A) @ abs(B)))


@pytest.mark.parametrize("n", [33, 129, 160, 200, 406])
@pytest.mark.parametrize("decades", [4, 8, 12])
@pytest.mark.parametrize("left", [0, 1])
def test_truncate_graded(ctx, n, decades, left):
    import tngpu
    r = np.random.default_rng(n)
    D = r.permutation(10.0 ** (-decades * np.arange(n) / n))
    Q = np.linalg.qr(r.standard_normal((n, n)) + 1j * r.standard_normal((n, n)))[0]
    A = D[:, None] * Q
    # the vectors of the graded side: its rows, or the transpose's columns
    th = np.asfortranarray(A.T if left else A)
    X, Y = (np.zeros((n, n), dtype=np.complex128, order="F") for _ in range(2))
    S, k = np.zeros(n), C.c_int64(n)
    t = tngpu._lib.trunc(0.0, 0, 1)
    ctx.check(ctx.lib.tn_truncate(ctx.h, n, n, dp(th), C.byref(t), left, dp(X), dp(Y), dp(S), C.byref(k)))
    assert k.value == n
    iso = Y.conj().T if left else X
    assert np.abs(iso.conj().T @ iso - np.eye(n)).max() <= 64 * n * EPS
    assert np.abs(S / np.sort(D)[::-1] - 1).max() <= 64 * n * EPS
    assert np.abs(X @ Y - th).max() <= 64 * n * EPS
