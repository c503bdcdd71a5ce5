"""The Lanczos step's kernels: the operator on the middle legs (small_apply, with its
lists of real, imaginary and other entries) and the orthogonalisation, at the edges
of their tiles and groups (128 threads a block, 8 vectors a group)."""

import ctypes as C

import numpy as np
import oracle as O
import pytest

pytestmark = pytest.mark.gpu


def dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


@pytest.fixture(scope="module")
def tn():
    import tngpu
    return tngpu


def gates(r, d):
    z = lambda: r.standard_normal((d,) * 4) + 1j * r.standard_normal((d,) * 4)  # noqa: E731
    yield "dense", z()
    yield "zero", 0 * z()
    yield "real sparse", np.where(r.random((d,) * 4) < 0.3, z().real, 0) + 0j
    mixed = z()
    mixed.real[r.random((d,) * 4) < 0.5] = 0
    mixed.imag[r.random((d,) * 4) < 0.5] = 0
    yield "mixed", mixed


@pytest.mark.parametrize("d,cl,cm,cr", [(2, 1, 1, 1), (2, 1, 2, 3), (2, 127, 3, 1), (3, 16, 4, 8), (2, 43, 5, 129),
                                        (3, 7, 20, 19), (2, 200, 2, 260), (7, 3, 2, 2)])
def test_operator_on_the_middle_legs(tn, d, cl, cm, cr):
    """Within 64 roundings of the exact sums of d^2 products of sums of cm; an
    infinity or NaN reaches what the full sums bring it to."""
    ctx = tn.context()
    r = np.random.default_rng(cl + cr)
    A1 = np.asfortranarray(r.standard_normal((cl, d, cm)) + 1j * r.standard_normal((cl, d, cm)))
    A2 = np.asfortranarray(r.standard_normal((cm, d, cr)) + 1j * r.standard_normal((cm, d, cr)))
    for name, G in gates(r, d):
        Gf = np.asfortranarray(G)
        out = np.zeros((cl, d, d, cr), dtype=np.complex128, order="F")
        ctx.check(ctx.lib.tn_gate2_apply(ctx.h, cl, cm, cr, d, dp(A1), dp(A2), dp(Gf), dp(out)))
        ref = np.einsum("aijb,piqj->apqb", np.tensordot(A1, A2, axes=([2], [0])), G)
        mod = np.einsum("aijb,piqj->apqb", np.tensordot(abs(A1), abs(A2), axes=([2], [0])), abs(G))
        assert np.all(abs(out - ref) <= 2.0 ** -46 * mod + 1e-300), name
        bad = A1.copy(order="F")
        bad[-1, 0, 0] = np.nan
        ctx.check(ctx.lib.tn_gate2_apply(ctx.h, cl, cm, cr, d, dp(bad), dp(A2), dp(Gf), dp(out)))
        assert np.isnan(out[-1]).all() and np.isfinite(out[:-1]).all(), name


@pytest.mark.parametrize("N,D,krylovdim", [(2, 1, 4), (4, 2, 3), (8, 4, 2), (8, 4, 8), (8, 4, 9), (8, 4, 17),
                                           (12, 8, 5)])
def test_lowest_energy(tn, N, D, krylovdim):
    """Full bond dimension, six sweeps: the energy of the oracle's DMRG, to 1e-9 (the
    same Krylov spaces in exact arithmetic)."""
    r = np.random.default_rng(N)
    shapes = [((1 if i == 0 else D), 2, (1 if i == N - 1 else D)) for i in range(N)]
    ts = [np.asfortranarray(r.standard_normal(s) + 1j * r.standard_normal(s)) for s in shapes]
    psi = tn.GMPS.from_tensors(ts, 1)
    def ham(mod):
        H = mod.OpList(N)
        for i in range(1, N + 1):
            H.add("x", i, 0.7)
            if i < N:
                H.add(["z", "z"], [i, i + 1], 1.0)
        return H

    kw = dict(maxdim=64, cutoff=1e-14, minsweeps=6, maxsweeps=6, krylovdim=krylovdim, kryloviter=3)
    _, E = tn.dmrg(psi, tn.MPO(tn.spinhalf(), ham(tn)), verbose=False, **kw)
    po = O.GMPS(1, 2, [t.copy() for t in ts], 1)
    _, ref = O.dmrg(po, O.mpo_from_oplist(O.spinhalf(), ham(O)), numconverges=np.inf, **kw)
    assert abs(E - np.real(ref)) <= 1e-9 * abs(ref)
