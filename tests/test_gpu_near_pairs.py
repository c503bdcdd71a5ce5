"""Truncated splits whose cut passes between two Schmidt vectors of nearly equal
weight: the kept one has to be the right one as far as the matrix determines it.

For a matrix with graded rows, D M with M well conditioned, a relative change of every
entry by 2^-52 turns the vectors of a pair by about 2^-52 over its relative gap, whatever
its weight (J. Barlow and J. Demmel, SIAM J. Numer. Anal. 27, 1990); n reflections of some
roundings give 64 n of that."""

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


def jacobi(A):
    """Left singular vectors of a real A, descending, by one-sided Jacobi in 64-bit-mantissa floats."""
    B = A.T.astype(np.longdouble)
    n = B.shape[1]
    V = np.eye(n, dtype=np.longdouble)
    for _ in range(30):
        off = np.longdouble(0)
        for p in range(n - 1):
            for q in range(p + 1, n):
                a, b, c = B[:, p] @ B[:, p], B[:, q] @ B[:, q], B[:, p] @ B[:, q]
                off = max(off, abs(c) / np.sqrt(a * b))
                if abs(c) <= 1e-19 * np.sqrt(a * b):
                    continue
                z = (b - a) / (2 * c)
                t = (1 if z >= 0 else -1) / (abs(z) + np.sqrt(1 + z * z))
                cs = 1 / np.sqrt(1 + t * t)
                for M in (B, V):
                    x, y = M[:, p].copy(), M[:, q].copy()
                    M[:, p], M[:, q] = cs * (x - t * y), cs * (t * x + y)
        if off < 1e-18:
            break
    s = np.sqrt((B * B).sum(0))
    return V[:, np.argsort(-s)]


def weights(n, weight, gap):
    """Singular values over nine decades with a pair of this weight and relative gap at n / 2."""
    s = 10.0 ** (-9 * np.arange(n) / n)
    k = n // 2
    s[:k] = np.geomspace(1, 3 * np.sqrt(weight), k)
    s[k - 1], s[k] = np.sqrt(weight) * (1 + gap / 2), np.sqrt(weight)
    s[k + 1:] = np.sqrt(weight) * np.geomspace(0.3, 1e-4, n - k - 1)
    return s, k


@pytest.mark.parametrize("kind,n", [("diagonal", n) for n in (20, 33, 72, 130, 260)] + [("dense", n) for n in (20, 33)])
@pytest.mark.parametrize("weight,gap", [(1e-8, 1e-9), (1e-10, 1e-6), (1e-10, 1e-8), (1e-12, 1e-7)])
def test_pair_at_the_cut(tn, kind, n, weight, gap):
    ctx = tn.context()
    r = np.random.default_rng(n)
    s, k = weights(n, weight, gap)
    if kind == "diagonal":
        p, q = r.permutation(n), r.permutation(n)
        A = np.zeros((n, n), complex)
        A[p, q] = s * np.exp(2j * np.pi * r.random(n))
        U = np.zeros((n, n))
        U[p, np.arange(n)] = 1
    else:
        A = s[:, None] * (np.eye(n) + 0.02 / np.sqrt(n) * r.standard_normal((n, n))) + 0j
        U = jacobi(A.real)
    th = np.asfortranarray(A)
    X, Y = (np.zeros((n, n), dtype=np.complex128, order="F") for _ in range(2))
    S, kk = np.zeros(n), C.c_int64(n)
    t = tn._lib.trunc(0.0, k, 1)
    ctx.check(ctx.lib.tn_truncate(ctx.h, n, n, dp(th), C.byref(t), 0, dp(X), dp(Y), dp(S), C.byref(kk)))
    assert kk.value == k
    Xk = np.reshape(X.ravel(order="F")[:n * k], (n, k), order="F")
    out = Xk - U[:, :k] @ (U[:, :k].conj().T @ Xk)  # what was kept of the vectors to leave
    assert np.linalg.norm(out, axis=0)[k - 1] <= 64 * n * EPS / gap


def test_chain_against_svd(tn):
    """One sweep of the 30-site XXZ chain at bond dimension 100 from a random state, cut by
    the dimension at weights of about 1e-9: energy and observables as with LAPACK's SVD in
    every split, to the 1e-9 that this library states against its oracle."""
    N, D = 30, 100
    r = np.random.default_rng([1, N, D])
    dims = [int(min(D, 2.0 ** min(i, N - i))) for i in range(N + 1)]
    ts = []
    for i in range(N):
        a = r.standard_normal((dims[i], 2, dims[i + 1]))
        lam = 10.0 ** (-0.75 * np.arange(dims[i + 1]) / max(dims[i + 1], 2))
        ts.append(np.asfortranarray(a * (lam / np.linalg.norm(lam) / np.sqrt(2.0)), dtype=np.complex128))

    def run(mod, psi, mpo, **kw):
        st = mod.spinhalf()
        psi.movecenter(1)
        psi.normalize()
        H, X = mod.OpList(N), mod.OpList(N)
        for i in range(1, N):
            for o in "xyz":
                H.add([o, o], [i, i + 1], 1.0)
        for i in range(1, N + 1):
            X.add("x", i, 1.0)
        psi, E = mod.dmrg(psi, mpo(st, H), krylovdim=3, maxsweeps=1, cutoff=1e-10, maxdim=D, verbose=False)
        return np.real(E), np.real(mod.inner(st, psi, X, psi))

    ref = run(O, O.GMPS(1, 2, [t.copy() for t in ts], 0), O.mpo_from_oplist)
    got = run(tn, tn.GMPS.from_tensors(ts), tn.MPO)
    assert abs(got[0] - ref[0]) <= 1e-9 * abs(ref[0])
    assert np.abs(got[1] - ref[1]).max() <= 1e-9 * np.abs(ref[1]).max()
