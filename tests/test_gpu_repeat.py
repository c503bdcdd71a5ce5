"""The same calls on the same inputs, again and again with other calls between them, give
the same bits: norms, splits, sums of operator products, Lanczos steps and quenches
(their small results come back through one pinned buffer, and blocks of a cluster or a
grid pass theirs to one another)."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROUNDS = 25


def dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def state(tn, N, D, seed):
    r = np.random.default_rng([N, D, seed])
    b = [min(D, 2 ** min(i, N - i)) for i in range(N + 1)]
    psi = tn.GMPS.from_tensors([np.asfortranarray(r.standard_normal(s) + 1j * r.standard_normal(s))
                                for s in zip(b[:-1], [2] * N, b[1:])])
    psi.movecenter(1)
    psi.normalize()
    return psi


def calls(tn):
    st = tn.spinhalf()

    def ham(N):
        H = tn.OpList(N)
        for i in range(1, N):
            for o in "xyz":
                H.add([o, o], [i, i + 1], 1.0)
        for i in range(1, N + 1):
            H.add("z", i, 0.3)
        return H

    def quench(N, D):
        psi = state(tn, N, D, 1)
        obs = tn.TEBDOperators(st, ham(N))
        psi, E = tn.tebd(st, psi, ham(N), 0.05, 0.1, 0.1, observers=[obs], cutoff=1e-10, maxdim=D, evol="real")
        return [np.asarray(E), np.asarray(obs.measurements), np.asarray(psi.bonddims())]

    def sums(N, D, seed):
        psi = state(tn, N, D, seed)
        return [np.asarray(tn.inner(st, psi, ham(N), psi)), np.asarray(psi.norm())]

    def ground(N, D):
        psi, E = tn.dmrg(state(tn, N, D, 2), tn.MPO(st, ham(N)), krylovdim=3, maxsweeps=1, cutoff=1e-10, maxdim=D,
                         verbose=False)
        return [np.asarray(E), np.asarray(psi.bonddims())]

    def split(n):
        ctx = tn.context()
        r = np.random.default_rng(n)
        th = np.asfortranarray(r.standard_normal((n, n)) + 1j * r.standard_normal((n, n)))
        X, Y = (np.zeros((n, n), dtype=np.complex128, order="F") for _ in range(2))
        S, k = np.zeros(n), C.c_int64(n)
        t = tn._lib.trunc(1e-10, 3 * n // 4, 1)
        ctx.check(ctx.lib.tn_truncate(ctx.h, n, n, dp(th), C.byref(t), 0, dp(X), dp(Y), dp(S), C.byref(k)))
        return [X, Y, S, np.asarray(k.value)]

    for N, D in ((6, 8), (10, 16), (8, 12)):
        yield f"quench {N} {D}", lambda N=N, D=D: quench(N, D)
    for N, D, s in ((4, 2, 1), (9, 8, 2), (12, 40, 3)):
        yield f"sums {N} {D}", lambda N=N, D=D, s=s: sums(N, D, s)
    yield "ground 8 8", lambda: ground(8, 8)
    yield "ground 12 40", lambda: ground(12, 40)
    for n in (3, 17, 40, 90, 150, 230):
        yield f"split {n}", lambda n=n: split(n)


def test_bits():
    import tngpu as tn
    every = list(calls(tn))
    first = {name: f() for name, f in every}
    r = np.random.default_rng(0)
    for _ in range(ROUNDS):
        for i in r.permutation(len(every)):
            name, f = every[i]
            for a, b in zip(first[name], f()):
                assert np.array_equal(a, b), name
