"""The Hermitian eigensolver at the orders of large truncated splits and up to its largest,
4096, where the reduction keeps its rows in global memory."""

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


def top(ctx, G, want):
    n = len(G)
    Gf = np.asfortranarray(G, dtype=np.complex128)
    lam, V = np.zeros(want), np.zeros((n, want), dtype=np.complex128, order="F")
    ctx.check(ctx.lib.tn_eigh_top(ctx.h, n, dp(Gf), want, dp(lam), dp(V)))
    return lam, V


@pytest.mark.parametrize("n,want", [(1500, 64), (2048, 1024), (4096, 40)])
def test_known_spectrum(ctx, n, want):
    """Reflections of a diagonal matrix: within 64 n 2^-52 as at the smaller orders."""
    r = np.random.default_rng(n)
    d = r.standard_normal(n)
    G = np.diag(d).astype(complex)
    for _ in range(3):
        v = r.standard_normal(n) + 1j * r.standard_normal(n)
        v /= np.linalg.norm(v)
        G -= np.outer(2 * v, v.conj() @ G)
        G -= np.outer(G @ v, 2 * v.conj())
    G = (G + G.conj().T) / 2
    lam, V = top(ctx, G, want)
    big = np.abs(d).max()
    assert np.abs(lam - np.sort(d)[::-1][:want]).max() <= 64 * n * EPS * big
    assert np.abs(V.conj().T @ V - np.eye(want)).max() <= 64 * n * EPS
    assert np.abs(G @ V - V * lam).max() <= 64 * n * EPS * big

