"""Truncated splits of matrices with sectors, exact zeros, rank deficiency, graded rows and
columns and rounding-size entries where exact arithmetic has zeros: what a symmetric
evolution from a product state brings.

The isometry is orthonormal and the other factor the matrix seen through it, to 64 n 2^-52 of
the norm; what is left out is no more than the smallest squared singular values, plus 2 k
times the Gram eigenproblem's 64 n 2^-52 (the sum of the k largest eigenvalues moves by that
much at most: K. Fan).

Quenches from product states with random phases, whose splits are of that kind, against the
oracle's, to its 1e-9."""

import ctypes as C

import numpy as np
import oracle as O
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


@pytest.fixture(scope="module")
def tn():
    import tngpu
    return tngpu


def matrix(r, kind, m, n):
    A = r.standard_normal((m, n)) + 1j * r.standard_normal((m, n))
    if kind % 2 == 0:  # sectors
        A = A * (r.integers(0, 3, m)[:, None] == r.integers(0, 3, n)[None])
    if kind in (1, 2, 4):
        A = 10.0 ** (-r.uniform(0, 20) * np.sort(r.random(m)))[:, None] * A
    if kind in (2, 3):
        A = A * 10.0 ** (-r.uniform(0, 15) * r.random(n))
    if kind == 5:
        A = A * (r.random((m, n)) < 0.3)
    if kind == 6:
        A = A[:, :1] @ A[:1]
    if r.random() < 0.6:
        lev = 10.0 ** r.uniform(-22, -15) * max(np.abs(A).max(), 1e-30)
        z = r.standard_normal((m, n)) + 1j * r.standard_normal((m, n))
        A = A + (r.random((m, n)) < r.random()) * lev * 10.0 ** r.uniform(-6, 0, (m, n)) * z
    return A


@pytest.mark.parametrize("lo,hi,count", [(2, 13, 1500), (13, 48, 300), (48, 140, 40), (210, 300, 6)])
@pytest.mark.parametrize("direction", [0, 1])
def test_splits(tn, lo, hi, count, direction):
    ctx = tn.context()
    r = np.random.default_rng([lo, direction])
    for it in range(count):
        m, n = (int(v) for v in r.integers(lo, hi, 2))
        A = matrix(r, it % 7, m, n)
        top = np.linalg.norm(A)
        if top == 0:
            continue
        k0 = min(m, n)
        keep = int(r.integers(1, k0 + 1))
        th = np.asfortranarray(A)
        X, Y, S, k = np.zeros(m * k0, complex), np.zeros(k0 * n, complex), np.zeros(k0), C.c_int64(k0)
        t = tn._lib.trunc(0.0, keep, 1)
        ctx.check(ctx.lib.tn_truncate(ctx.h, m, n, dp(th), C.byref(t), direction, dp(X), dp(Y), dp(S), C.byref(k)))
        k = k.value
        assert k == keep
        X, Y = X[:m * k].reshape((m, k), order="F"), Y[:k * n].reshape((k, n), order="F")
        iso, other, seen = (X, Y, X.conj().T @ A) if direction == 0 else (Y.conj().T, X, A @ Y.conj().T)
        tol = 64 * max(m, n) * EPS
        assert np.abs(iso.conj().T @ iso - np.eye(k)).max() <= tol, (it, m, n)
        assert np.abs(other - seen).max() <= tol * top, (it, m, n)
        tail = (np.linalg.svd(A, compute_uv=False)[k:] ** 2).sum()
        assert np.linalg.norm(A - X @ Y) ** 2 <= tail + 2 * k * tol * top ** 2, (it, m, n, k)


@pytest.mark.parametrize("n", [3, 20, 60, 150, 300, 1200])
@pytest.mark.parametrize("s", [1e-1, 1e-2, 1e-4])
def test_equal_rows(tn, n, s):
    """Rows that are all alike beside a larger one: two singular values, each to 64 n 2^-52."""
    ctx = tn.context()
    A = np.zeros((n, 2), complex)
    A[0, 0], A[1:, 1] = np.sqrt(n), s
    th = np.asfortranarray(A)
    X, Y, S, k = np.zeros(2 * n, complex), np.zeros(4, complex), np.zeros(2), C.c_int64(2)
    t = tn._lib.trunc(0.0, 2, 1)
    ctx.check(ctx.lib.tn_truncate(ctx.h, n, 2, dp(th), C.byref(t), 0, dp(X), dp(Y), dp(S), C.byref(k)))
    assert k.value == 2
    tol = 64 * n * EPS
    assert np.abs(S - [np.sqrt(n), s * np.sqrt(n - 1)]).max() <= tol * np.sqrt(n)
    assert np.abs(X.reshape((n, 2), order="F") @ Y.reshape((2, 2), order="F") - A).max() <= tol * np.sqrt(n)


@pytest.mark.parametrize("seed", range(8))
def test_quench_from_a_product_state(tn, seed):
    N, dt, steps = 10, 0.05, 6
    r = np.random.default_rng(seed)
    up, ph = r.permutation(N) < N // 2, np.exp(2j * np.pi * r.random(N))
    ts = [np.asfortranarray(np.reshape([1.0, 0] if u else [0, 1.0], (1, 2, 1)) * p) for u, p in zip(up, ph)]

    def run(mod, psi):
        st, H, Z = mod.spinhalf(), mod.OpList(N), mod.OpList(N)
        for i in range(1, N):
            for o, c in (("x", 1.0), ("y", 1.0), ("z", 0.5)):
                H.add([o, o], [i, i + 1], c)
        for i in range(1, N + 1):
            H.add("z", i, 0.2 * (-1) ** i)
            Z.add("z", i, 1.0)
        psi, E = mod.tebd(st, psi, H, dt, steps * dt, steps * dt, cutoff=1e-10, maxdim=32, evol="real")
        return np.real(E), np.real(mod.inner(st, psi, Z, psi))

    E, z = run(tn, tn.GMPS.from_tensors(ts))
    E0, z0 = run(O, O.GMPS(1, 2, [t.copy() for t in ts], 0))
    assert abs(E - E0) <= 1e-9 and np.abs(z - z0).max() <= 1e-9
