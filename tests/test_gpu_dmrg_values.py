"""Two sweeps of DMRG of the 20-site Ising chain (ordered side) from random states of
bond dimension 4: the six of the first 200 whose results depend most on which of two
nearly equal Schmidt vectors a cut at 1e-10 keeps.

Energies, bond dimensions and <x_i> or <z_i z_{i+1}> are those of the FP64 solver
(csrc/eig_fp64.cu), recorded when it was the only one.  The operations and their
order are the same, so the energies have to agree to a few units in the last place;
the observables come from other sums (16 roundings)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, EPS = 20, 2.0 ** -52
RECORDED = {
    6: (-20.40021714775875, [2, 4, 5, 5, 5, 4, 4, 3, 3, 3, 3, 3, 3, 4, 5, 5, 5, 4, 2],
        [0.2586591356904593, 0.2586744199807438, 0.2589741872191972, 0.2931729042004508, 0.48383952849403844]),
    44: (-20.400217148406234, [2, 4, 5, 5, 5, 4, 4, 3, 4, 4, 3, 4, 4, 4, 5, 5, 5, 4, 2],
         [0.2586585606286634, 0.25867336705951943, 0.25897338856775937, 0.2931748527595072, 0.4838387879023289]),
    53: (-20.399388767193795, [2, 4, 5, 5, 7, 10, 15, 16, 9, 8, 14, 8, 4, 4, 5, 5, 5, 4, 2],
         [0.2597739975751477, 0.2582765984827703, 0.25926901200507263, 0.2932531619468961, 0.4839043576377278]),
    54: (-20.386579669420335, [2, 4, 5, 5, 5, 8, 7, 5, 5, 11, 15, 10, 5, 4, 7, 6, 5, 4, 2],
         [0.25836364058268513, 0.25440479017717543, 0.24586475838306265, 0.33395034716301875, 0.5356791926142956]),
    108: (-20.399518729399176, [2, 4, 5, 6, 5, 3, 4, 4, 4, 4, 5, 10, 6, 6, 7, 6, 5, 4, 2],
          [0.2586579147970998, 0.257101327976639, 0.2588845736341314, 0.3035165091944274, 0.49522122669090235]),
    178: (-20.400217148603808, [2, 4, 5, 5, 5, 4, 4, 4, 3, 3, 3, 4, 4, 4, 5, 5, 5, 4, 2],
          [0.2586590516090896, 0.2586746985789488, 0.2589742217434838, 0.2931779671125798, 0.4838311379055821]),
}
SITES = (12, 14, 16, 19, 20)  # of <x_i>


def start(seed):
    r = np.random.default_rng([seed, N, 4])
    dims = [min(4, 2 ** min(i, N - i)) for i in range(N + 1)]
    out = []
    for i in range(N):
        a = r.standard_normal((dims[i], 2, dims[i + 1]))
        lam = 10.0 ** (-0.75 * np.arange(dims[i + 1]) / max(dims[i + 1], 2))
        out.append(np.asfortranarray(a * (lam / np.linalg.norm(lam) / np.sqrt(2.0)), dtype=np.complex128))
    return out


@pytest.mark.parametrize("seed", sorted(RECORDED))
def test_recorded_values(seed):
    import tngpu as tn
    st = tn.spinhalf()
    H = tn.OpList(N)
    for i in range(1, N):
        H.add(["z", "z"], [i, i + 1], -1.0)
    for i in range(1, N + 1):
        H.add("x", i, -0.5)
    psi = tn.GMPS.from_tensors(start(seed))
    psi.movecenter(1)
    psi.normalize()
    psi, E = tn.dmrg(psi, tn.MPO(st, H), krylovdim=8, maxsweeps=2, cutoff=1e-10, maxdim=64, verbose=False)
    X = tn.OpList(N)
    for i in SITES:
        X.add("x", i, 1.0)
    energy, dims, xs = RECORDED[seed]
    assert [int(b) for b in psi.bonddims()][1:20] == dims
    assert abs(E - energy) <= 4 * EPS * abs(energy)
    assert np.abs(np.real(tn.inner(st, psi, X, psi)) - xs).max() <= 16 * EPS
