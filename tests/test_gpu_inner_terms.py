"""Sums of operator products (inner): every length of a term, operators shared by
terms or not, bra and ket of different bond dimensions, and blocks too large to be
kept together, against the oracle.  Tolerance: 64 n 2^-52 of the product of norms for
chains of n sites, a few roundings a product."""

import numpy as np
import oracle as O
import pytest

pytestmark = pytest.mark.gpu


def state(mod, N, D, d, seed):
    r = np.random.default_rng(seed)
    b = [min(D, d ** min(i, N - i)) for i in range(N + 1)]
    ts = [np.asfortranarray((r.standard_normal(s) + 1j * r.standard_normal(s)) / np.sqrt(d * s[0]))
          for s in zip(b[:-1], [d] * N, b[1:])]
    return ts


def norm(ts):
    E = np.ones((1, 1))
    for t in ts:
        E = np.tensordot(t.conj(), np.tensordot(E, t, (1, 0)), ((0, 1), (0, 1)))
    return np.sqrt(abs(E[0, 0]))


@pytest.mark.parametrize("N,Db,Dk", [(1, 1, 1), (2, 1, 2), (3, 2, 2), (6, 4, 3), (9, 5, 16), (10, 17, 8), (7, 8, 8)])
def test_terms_of_every_length(N, Db, Dk):
    import tngpu as tn
    names = ["x", "y", "z", "s+", "s-"]

    def ops(mod):
        g = np.random.default_rng(N + Dk)
        H = mod.OpList(N)
        for i in range(1, N + 1):
            for ln in (1, 1, 2, 2, 3, 4):
                if i + ln - 1 <= N:
                    H.add([names[g.integers(5)] for _ in range(ln)], list(range(i, i + ln)), float(g.standard_normal()))
        return H

    tb, tk = state(O, N, Db, 2, 1), state(O, N, Dk, 2, 2)
    got = np.asarray(tn.inner(tn.spinhalf(), tn.GMPS.from_tensors(tb), ops(tn), tn.GMPS.from_tensors(tk)))
    ref = np.asarray(O.inner(O.spinhalf(), O.GMPS(1, 2, tb, 0), ops(O), O.GMPS(1, 2, tk, 0)))
    assert got.shape == ref.shape
    assert np.abs(got - ref).max() <= 64 * N * 2.0 ** -52 * 4 * norm(tb) * norm(tk)


def test_all_terms_and_one_by_one():
    """Together the blocks of these terms are beyond what is kept at once."""
    import tngpu as tn
    N, D = 22, 700
    ts = state(O, N, D, 2, 3)
    psi = tn.GMPS.from_tensors(ts)
    names = ["x", "y", "z", "s+", "s-", "n", "id"]
    terms = [([names[(i + k) % 5]], [i]) for i in range(9, 14) for k in range(5)]
    terms += [([names[k], names[(k + 1) % 5]], [i, i + 1]) for i in range(8, 14) for k in range(5)]

    def run(sel):
        H = tn.OpList(N)
        for o, s in sel:
            H.add(o, s, 1.0)
        return np.asarray(tn.inner(tn.spinhalf(), psi, H, psi))

    together = run(terms)
    alone = np.concatenate([run([t]) for t in terms[::11]])
    assert np.abs(together[::11] - alone).max() <= 64 * N * 2.0 ** -52 * 4 * norm(ts) ** 2
