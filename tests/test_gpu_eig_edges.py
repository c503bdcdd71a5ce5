"""The Hermitian eigensolver at the edges of its forms: cluster sizes 1, 4, 8
and 16 of the reduction (orders 16, 32, 64 and 208), the divide and conquer's
levels (powers of two) and its two forms (128), the panel widths of the
back-transformation (64, 128) and its form for small orders (32, 48).

tn_eigh_top is checked on indefinite, rank-deficient, diagonal and zero-padded
matrices: residual and orthogonality are within 64 n 2^-52, a backward error of
64 roundings in each of n reflections.  tn_truncate's Gram path is graded: the
singular values of D M, M well conditioned, are good to 64 n 2^-52 each,
however small, against one-sided Jacobi (LAPACK dgejsv, which has that
property)."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52
SIZES = [1, 2, 3, 5, 8, 9, 16, 17, 31, 32, 33, 48, 49, 63, 64, 65, 127, 128, 129, 192, 193, 208, 209, 256, 257, 405, 406, 1100, 1200]


def dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


@pytest.fixture(scope="module")
def ctx():
    import tngpu
    return tngpu.context()


def matrices(n):
    r = np.random.default_rng(n)
    z = lambda *s: r.standard_normal(s) + 1j * r.standard_normal(s)  # noqa: E731
    A = z(n, n)
    yield "indefinite", (A + A.conj().T) * 10.0 ** r.uniform(-150, 150)
    M = z(n, max(1, n // 4))
    yield "rank n/4", M @ M.conj().T
    yield "diagonal", np.diag(np.arange(n) % 3 - 1.0) + 0j
    B = np.zeros((n, n), complex)
    h = n // 2
    B[:h, :h] = (A + A.conj().T)[:h, :h]
    yield "padded", B


@pytest.mark.parametrize("n", SIZES)
def test_eigh_top_edges(ctx, n):
    for name, G in matrices(n):
        for want in sorted({1, (n + 1) // 2, n}):
            Gf = np.asfortranarray(G)
            lam, V = np.zeros(want), np.zeros((n, want), dtype=np.complex128, order="F")
            ctx.check(ctx.lib.tn_eigh_top(ctx.h, n, dp(Gf), want, dp(lam), dp(V)))
            top = max(np.abs(np.linalg.eigvalsh(G)).max(), 1e-300)
            ref = np.linalg.eigvalsh(G)[::-1][:want]
            assert np.abs(lam - ref).max() <= 64 * n * EPS * top, (name, want)
            assert np.abs(V.conj().T @ V - np.eye(want)).max() <= 64 * n * EPS, (name, want)
            assert np.abs(G @ V - V * lam).max() <= 64 * n * EPS * top, (name, want)


@pytest.mark.parametrize("n", [2, 17, 33, 65, 129, 257, 406])
@pytest.mark.parametrize("order", ["down", "up", "mixed"])
def test_truncate_graded(ctx, n, order):
    import tngpu
    lapack = pytest.importorskip("scipy.linalg").lapack
    r = np.random.default_rng(n)
    M = np.eye(n) + 0.2 / np.sqrt(n) * r.standard_normal((n, n))
    D = 10.0 ** (-5 * np.arange(n) / n)
    D = {"down": D, "up": D[::-1], "mixed": r.permutation(D)}[order]
    A = D[:, None] * M
    s = lapack.dgejsv(A.T)
    ref = s[0] * (s[3][1] / s[3][0])
    th = np.asfortranarray(A.astype(np.complex128))
    X, Y = (np.zeros((n, n), dtype=np.complex128, order="F") for _ in range(2))
    S, k = np.zeros(n), C.c_int64(n)
    t = tngpu._lib.trunc(0.0, 0, 1)
    ctx.check(ctx.lib.tn_truncate(ctx.h, n, n, dp(th), C.byref(t), 0, dp(X), dp(Y), dp(S), C.byref(k)))
    assert k.value == n
    assert np.abs(S / ref - 1).max() <= 64 * n * EPS
    assert np.abs(X.conj().T @ X - np.eye(n)).max() <= 64 * n * EPS
    assert np.abs(X @ Y - A).max() <= 64 * n * EPS


def test_not_finite(ctx):
    """A NaN gives NaN eigenvalues or an error, and the next call is clean."""
    n = 40
    G = np.asfortranarray(np.eye(n) + 0j)
    G[3, 3] = np.nan
    lam, V = np.zeros(4), np.zeros((n, 4), dtype=np.complex128, order="F")
    if ctx.lib.tn_eigh_top(ctx.h, n, dp(G), 4, dp(lam), dp(V)) == 0:
        assert np.isnan(lam).all()
    G = np.asfortranarray(np.diag(np.arange(n) + 1.0) + 0j)
    ctx.check(ctx.lib.tn_eigh_top(ctx.h, n, dp(G), 4, dp(lam), dp(V)))
    assert np.allclose(lam, [40, 39, 38, 37])
