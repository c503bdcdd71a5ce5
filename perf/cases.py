"""Performance cases of the framework: the calls a program makes through the
public Python API (tngpu), over the range of sizes of this repository's
configurations, tests and benchmark, each direction and precision included.

A case is a dict with a ``kind``:

  measure     inner: energy terms and local observables of a state, as the
              TEBD energy observer and every DMRG script evaluate them
  canonical   gauge sweeps: a non-truncating one to the right end, a
              truncating one back, and the spectrum of the middle bond
  tebd        real-time quench of the XXZ chain in a staggered field (the
              TEBD configuration) with its operator observer, FP64 or mixed
  dmrg        two-site DMRG sweeps, TFIM or XXZ, FP64 or mixed-env64
  fit         applyMPO and the variational fit of a sum of states (vmps)
  trajectory  one quantum-jump trajectory of the single-trajectory driver
  ensemble    a trajectory ensemble in the persistent engine
  grad        gradient of a TEBD evolution (forward and backward)

MPS tensors carry a gauge freedom (phases and rotations of the bond bases), so
states come back as what does not depend on it: observables on every site and
bond, spectra, bond dimensions, norms.  A mixed-precision run's results carry
FP32-class rounding (3xTF32 products) and come back in single precision.
"""

from __future__ import annotations

import os
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.getcwd(), "tensornetworks.jl_gb300"))

import tngpu as tn  # noqa: E402


# ---- the cases ------------------------------------------------------------------
def listed():
    return [
        # observables of a small chain: what an exact-diagonalisation-size
        # study calls most; launches and host work are everything here
        {"name": "measure-n10-chi8", "kind": "measure", "N": 10, "chi": 8},
        # energy and observables of an entangled state of the quench's chain length
        {"name": "measure-n64-chi128", "kind": "measure", "N": 64, "chi": 128},
        # canonicalising and truncating an unnormalised MPS
        {"name": "canonical-n64-chi64", "kind": "canonical", "N": 64, "chi": 64, "maxdim": 48},
        # the first steps of a quench from the Neel state, small chain
        {"name": "tebd-n16-neel", "kind": "tebd", "N": 16, "chi": 1, "maxdim": 32, "steps": 5,
         "precision": "fp64"},
        # one step of the quench in its entangled stage
        {"name": "tebd-n24-chi128", "kind": "tebd", "N": 24, "chi": 128, "maxdim": 128, "steps": 1,
         "precision": "fp64"},
        # the TFIM ground-state configuration: N=20, chi <= 64, Lanczos 8 x 2
        {"name": "dmrg-tfim-n20-chi64", "kind": "dmrg", "model": "tfim", "N": 20, "chi": 4,
         "maxdim": 64, "cutoff": 1e-10, "krylovdim": 8, "sweeps": 2, "precision": "fp64"},
        # a sweep of the XXZ chain at the ramp's middle bond dimension, FP64
        {"name": "dmrg-xxz-n28-chi256", "kind": "dmrg", "model": "xxz", "N": 28, "chi": 256,
         "maxdim": 256, "cutoff": 1e-10, "krylovdim": 3, "sweeps": 1, "precision": "fp64"},
        # bonds at the benchmark's chi=1024 in its precision mode
        {"name": "dmrg-xxz-n21-chi1024-mixed-env64", "kind": "dmrg", "model": "xxz", "N": 21,
         "chi": 1024, "maxdim": 1024, "cutoff": 1e-12, "krylovdim": 3, "sweeps": 1,
         "precision": "mixed-env64"},
        # H|psi> and the fit of |psi> - 0.1 H|psi>, as projector TEBD does
        {"name": "fit-n24-chi40", "kind": "fit", "N": 24, "chi": 40, "maxdim": 64},
        # one quantum-jump trajectory, small chain
        {"name": "trajectory-n10", "kind": "trajectory", "N": 10, "maxdim": 16, "steps": 10},
        # the trajectory ensemble configuration (N=32, 1024 trajectories),
        # some steps from an entangled state
        {"name": "ensemble-n32-1024", "kind": "ensemble", "N": 32, "chi": 16, "maxdim": 64,
         "ntraj": 1024, "steps": 2},
        # gradient of a driven TFIM evolution: forward, tape and backward
        {"name": "grad-n16-chi32", "kind": "grad", "N": 16, "chi": 32, "maxdim": 32, "segments": 2,
         "nsub": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["measure", "canonical", "tebd", "tebd", "dmrg", "dmrg", "fit", "trajectory",
                       "ensemble", "grad"])
    if kind == "measure":
        chi = _log_int(rng, 5, 128)
        return {"kind": kind, "N": rng.randint(8, 100 if chi <= 64 else 64), "chi": chi}
    if kind == "canonical":
        chi = _log_int(rng, 8, 128)
        return {"kind": kind, "N": rng.randint(10, 60), "chi": chi,
                "maxdim": max(4, int(chi * rng.uniform(0.5, 1.0)))}
    if kind == "tebd":
        chi = _log_int(rng, 6, 200)
        hi = 64 if chi <= 64 else 24
        return {"kind": kind, "N": rng.randint(9, hi), "chi": chi, "maxdim": chi, "steps": 1,
                "precision": rng.choice(["fp64", "fp64", "mixed"])}
    if kind == "dmrg":
        chi = _log_int(rng, 8, 320)
        N = rng.randint(10, 40 if chi <= 128 else 20)
        return {"kind": kind, "model": rng.choice(["tfim", "xxz"]), "N": N, "chi": chi,
                "maxdim": int(chi * rng.uniform(0.75, 1.25)), "cutoff": 1e-10, "krylovdim": 3,
                "sweeps": rng.randint(1, 2) if chi <= 64 else 1,
                "precision": rng.choice(["fp64", "fp64", "mixed-env64"])}
    if kind == "fit":
        chi = _log_int(rng, 6, 40)
        return {"kind": kind, "N": rng.randint(8, 32), "chi": chi, "maxdim": chi + rng.randint(1, chi)}
    if kind == "trajectory":
        return {"kind": kind, "N": rng.randint(5, 16), "maxdim": _log_int(rng, 4, 32),
                "steps": rng.randint(3, 10)}
    if kind == "ensemble":
        chi = _log_int(rng, 2, 16)
        return {"kind": kind, "N": rng.randint(8, 32), "chi": chi, "maxdim": 64,
                "ntraj": _log_int(rng, 16, 1024), "steps": 2}
    chi = _log_int(rng, 4, 40)
    return {"kind": "grad", "N": rng.randint(6, 16), "chi": chi, "maxdim": chi,
            "segments": rng.randint(1, 3), "nsub": 2}


# ---- inputs -----------------------------------------------------------------------
def _dims(N, chi, d=2):
    return [int(min(chi, d ** min(i, N - i, 40))) for i in range(N + 1)]


def _mps_arrays(seed, N, chi, real=False, decades=1.5):
    """Random site tensors whose bond weights fall geometrically over
    ``decades`` decades on each side of a bond, so that the Schmidt values
    fall over about twice as many, as those of ground and evolved states do;
    scaled to a norm near one."""
    r = np.random.default_rng([seed, N, chi])
    dims, out = _dims(N, chi), []
    for i in range(N):
        a = r.standard_normal((dims[i], 2, dims[i + 1]))
        if not real:
            a = a + 1j * r.standard_normal(a.shape)
        lam = 10.0 ** (-decades * np.arange(dims[i + 1]) / max(dims[i + 1], 2))
        a = a * (lam / np.linalg.norm(lam) / np.sqrt(2.0 if real else 4.0))
        out.append(np.asfortranarray(a, dtype=np.complex128))
    return out


def _state(seed, N, chi, real=False, decades=1.5):
    psi = tn.GMPS.from_tensors(_mps_arrays(seed, N, chi, real, decades))
    psi.movecenter(1)
    psi.normalize()
    return psi


def _xxz(N, delta=1.0, field=0.0):
    H = tn.OpList(N)
    for i in range(1, N):
        for o, c in (("x", 1.0), ("y", 1.0), ("z", delta)):
            H.add([o, o], [i, i + 1], c)
    if field:
        for i in range(1, N + 1):
            H.add("z", i, field * (-1) ** i)
    return H


def _tfim(N, zz, x):
    H = tn.OpList(N)
    for i in range(1, N):
        H.add(["z", "z"], [i, i + 1], zz)
    for i in range(1, N + 1):
        H.add("x", i, x)
    return H


def _local(N, names="xz"):
    Z = tn.OpList(N)
    for i in range(1, N + 1):
        for o in names:
            Z.add(o, i, 1.0)
    return Z


def _jumps(N):
    J = tn.OpList(N)
    for i in range(1, N + 1):
        J.add("s-", i, np.sqrt(0.1))
    return J


TEBD_DT, TEBD_DELTA, TEBD_FIELD = 0.05, 0.5, 0.2
QJMC_DT = 0.01


def prepare(case, seed):
    k, N = case["kind"], case["N"]
    st = tn.spinhalf()
    s = {"case": case, "st": st}
    if k == "measure":
        s["psi"] = _state(seed, N, case["chi"])
        s["terms"] = _xxz(N) + _local(N)
    elif k == "canonical":
        s["psi"] = tn.GMPS.from_tensors(_mps_arrays(seed, N, case["chi"]))
    elif k == "tebd":
        if case["chi"] == 1:  # a product state; the seed picks its up spins
            up = np.random.default_rng([seed, N]).permutation(N) < N // 2
            s["psi"] = tn.productMPS(st, ["up" if u else "dn" for u in up])
        else:
            s["psi"] = _state(seed, N, case["chi"])
        s["H"] = _xxz(N, TEBD_DELTA, TEBD_FIELD)
        s["obs"] = _local(N) + _xxz(N)
    elif k == "dmrg":
        s["H"] = _xxz(N) if case["model"] == "xxz" else _tfim(N, -1.0, -0.5)
        s["W"] = tn.MPO(st, s["H"])
        s["psi"] = _state(seed, N, case["chi"], real=True, decades=0.75)
        s["obs"] = _tfim(N, 1.0, 1.0)
    elif k == "fit":
        s["psi"] = _state(seed, N, case["chi"])
        s["W"] = tn.MPO(st, _xxz(N))
        s["obs"] = _local(N)
    elif k in ("trajectory", "ensemble"):
        s["H"], s["J"] = _tfim(N, 1.0, 0.8), _jumps(N)
        s["obs"] = _local(N)
        r = np.random.default_rng([seed, N])
        if k == "ensemble":
            s["psi"] = _state(seed, N, case["chi"])
            s["seed"] = int(r.integers(1 << 40))
        else:
            th = r.uniform(0.0, 0.5 * np.pi, N)  # a tilted product state
            s["psi"] = tn.GMPS.from_tensors(
                [np.reshape([np.cos(t), np.sin(t)], (1, 2, 1)) for t in th])
            s["draws"] = r.random(3 * case["steps"] + 3)
    else:
        s["psi"] = _state(seed, N, case["chi"])
        s["h"] = np.random.default_rng([seed, N]).uniform(0.0, 1.0, case["segments"])
        s["prob"] = tn.TEBDGradProblem(st, lambda h: _tfim(N, 1.0, float(h)), 0.02, case["nsub"],
                                       "z", (N + 1) // 2, cutoff=1e-10, maxdim=case["maxdim"])
    return s


# ---- one pass ---------------------------------------------------------------------
def run(s):
    c, st = s["case"], s["st"]
    k, N = c["kind"], c["N"]
    if k == "measure":
        return {"terms": tn.inner(st, s["psi"], s["terms"], s["psi"])}
    psi = s["psi"].copy()
    if k == "canonical":
        psi.movecenter(N)
        psi.movecenter(1, cutoff=1e-12, maxdim=c["maxdim"])
        norm = abs(psi.norm())
        psi.normalize()
        return {"norm": norm, "dims": np.asarray(psi.bonddims()),
                "spectrum": _pad(psi.singular_values(N // 2), c["maxdim"])}
    if k == "tebd":
        ob = tn.TEBDOperators(st, s["obs"])
        T = c["steps"] * TEBD_DT
        psi, energy = tn.tebd(st, psi, s["H"], TEBD_DT, T, T, observers=[ob], cutoff=1e-10,
                              maxdim=c["maxdim"], evol="real", precision=c["precision"])
        out = {"energy": np.asarray(energy), "obs": np.asarray(ob.measurements),
               "dims": np.asarray(psi.bonddims())}
        return _single(out) if c["precision"] != "fp64" else out
    if k == "dmrg":
        stats = {}
        psi, energy = tn.dmrg(psi, s["W"], krylovdim=c["krylovdim"], maxsweeps=c["sweeps"],
                              cutoff=c["cutoff"], maxdim=c["maxdim"], verbose=False,
                              precision=c["precision"], stats=stats)
        out = {"energy": np.asarray(energy), "energy64": np.asarray(stats["energy_fp64"]),
               "obs": tn.inner(st, psi, s["obs"], psi), "dims": np.asarray(psi.bonddims())}
        return _single(out) if c["precision"] != "fp64" else out
    if k == "fit":
        hpsi = tn.applyMPO(s["W"], psi, cutoff=1e-12, maxdim=c["maxdim"])
        stats = {}
        fit = tn.vmps(psi, hpsi, coeffs=[1.0, -0.1], cutoff=1e-12, maxdim=c["maxdim"], maxsweeps=2,
                      stats=stats)
        return {"cost": np.asarray(stats["cost"]), "hpsi": np.asarray(hpsi.norm()),
                "fit_psi": np.asarray(tn.overlap(fit, psi)),
                "fit_hpsi": np.asarray(tn.overlap(fit, hpsi)),
                "obs": tn.inner(st, fit, s["obs"], fit), "dims": np.asarray(fit.bonddims())}
    if k == "trajectory":
        ob = tn.QJMCOperators(s["obs"], st)
        jumps, times = tn.qjmc_simulation(st, psi, s["H"], s["J"], c["steps"] * QJMC_DT, QJMC_DT,
                                          observers=[ob], cutoff=1e-10, maxdim=c["maxdim"],
                                          draws=s["draws"])
        return {"jumps": _pad(np.asarray(jumps, dtype=np.int64), c["steps"]),
                "times": _pad(np.asarray(times), c["steps"]),
                "obs": np.asarray(ob.measurements), "dims": np.asarray(psi.bonddims())}
    if k == "ensemble":
        times, obs, nj = tn.qjmc_ensemble(st, psi, s["H"], s["J"], c["steps"] * QJMC_DT, QJMC_DT,
                                          s["obs"], c["ntraj"], seed=s["seed"], cutoff=1e-10,
                                          maxdim=c["maxdim"], engine="device")
        return {"obs": obs, "jumps": np.asarray(nj, dtype=np.int64)}
    f, back = s["prob"].rrule(psi, s["h"])
    return {"f": np.asarray(f), "grad": np.asarray(back())}


def _pad(v, n):
    """v with zeros up to n entries: how many are kept depends on the inputs."""
    return np.concatenate([v[:n], np.zeros(max(0, n - len(v)), v.dtype)])


def _single(out):
    to = {"float64": np.float32, "complex128": np.complex64}
    return {k: np.asarray(v).astype(to.get(np.asarray(v).dtype.name, np.asarray(v).dtype))
            for k, v in out.items()}


# ---- what a pass cannot do without --------------------------------------------------
def _mps_bytes(dims):
    return 16.0 * sum(2 * dims[i] * dims[i + 1] for i in range(len(dims) - 1))


def _split_flops(m, n, k, g):
    """Gram (half), top-k Hermitian eigenpairs (LAPACK count), projection."""
    return 4.0 * g * g * max(m, n) * min(m, n) / min(g, max(m, n)) + 16.0 / 3.0 * g ** 3 \
        + 8.0 * g * g * k + 8.0 * m * n * k


def _gate_layer_flops(dims):
    """One gate per bond: two-site tensor, gate leg, split, and a gauge move."""
    f = 0.0
    for i in range(1, len(dims) - 1):
        l, m, r = dims[i - 1], dims[i], dims[i + 1]
        f += 8.0 * 4 * l * m * r + 8.0 * 16 * l * r + _split_flops(2 * l, 2 * r, m, 2 * l)
        f += _split_flops(2 * l, m, m, 2 * l) + 8.0 * 2 * m * m * r
    return f


def _measure_flops(dims, two):
    """Overlap blocks both ways and one contraction per local term."""
    f = 0.0
    for i in range(1, len(dims)):
        l, r = dims[i - 1], dims[i]
        f += 8.0 * 4 * (l * l * r + l * r * r) * (1 + two)
    return f


def work(case):
    k, N = case["kind"], case["N"]
    dims = _dims(N, max(case.get("chi", 1), 1))
    if k == "measure":
        return {"bytes": _mps_bytes(dims), "flops": _measure_flops(dims, 1)}
    if k == "canonical":
        f = sum(2 * (_split_flops(2 * dims[i - 1], dims[i], dims[i], 2 * dims[i - 1])
                     + 16.0 * dims[i] ** 2 * dims[min(i + 1, N)]) for i in range(1, N))
        return {"bytes": 2 * _mps_bytes(dims), "flops": f}
    if k == "tebd":
        cap = _dims(N, case["maxdim"] if case["chi"] > 1 else min(case["maxdim"], 12))
        return {"bytes": 2 * _mps_bytes(cap),
                "flops": case["steps"] * 1.5 * _gate_layer_flops(cap) + 2 * _measure_flops(cap, 1)}
    if k == "dmrg":
        dims = _dims(N, min(case["maxdim"], 4 * case["chi"]))
        w, d = (5, 2) if case["model"] == "xxz" else (3, 2)
        mv = 5 if case["krylovdim"] == 3 else 12
        f = 0.0
        for i in range(1, N):
            l, r, m = dims[i - 1], dims[i + 1], dims[i]
            h = 8.0 * (w * d * d * (l * l * r + l * r * r) + w * w * d ** 4 * l * r)
            env = 8.0 * w * d * 2 * (l * l * m + l * m * m)
            f += mv * h + 2 * env + _split_flops(2 * l, 2 * r, m, 2 * l)
        return {"bytes": 2 * _mps_bytes(dims), "flops": case["sweeps"] * f}
    if k == "fit":
        big, fit = _dims(N, 5 * case["chi"]), _dims(N, case["maxdim"])
        f = sum(2 * _split_flops(2 * big[i - 1], big[i], big[i], 2 * big[i - 1]) for i in range(1, N))
        f += 2 * sum(_split_flops(2 * fit[i - 1], 2 * fit[i + 1], fit[i], 2 * fit[i - 1])
                     for i in range(1, N))
        return {"bytes": 3 * _mps_bytes(dims), "flops": f}
    if k in ("trajectory", "ensemble"):
        cap = _dims(N, min(case["maxdim"], 2 * case.get("chi", 2)))
        f = case.get("ntraj", 1) * case["steps"] * (1.5 * _gate_layer_flops(cap)
                                                    + 2 * _measure_flops(cap, 0))
        return {"bytes": case.get("ntraj", 1) * 2 * _mps_bytes(dims), "flops": f}
    steps = case["segments"] * case["nsub"]
    return {"bytes": 2 * _mps_bytes(dims), "flops": 4 * steps * 1.5 * _gate_layer_flops(dims)}


# ---- the same values in plain numpy, 64 bits ------------------------------------------
OPS = {"x": np.array([[0, 1], [1, 0]], complex), "y": np.array([[0, -1j], [1j, 0]]),
       "z": np.diag([1.0 + 0j, -1.0])}


class _Plain:
    """A numpy MPS with a truncating SVD gauge centre (sites from 0)."""

    def __init__(self, ts, cutoff=0.0, maxdim=0):
        self.A = [np.asarray(t, complex) for t in ts]
        self.c, self.N = None, len(ts)
        self.cutoff, self.maxdim = cutoff, maxdim

    def svd(self, M, trunc):
        U, S, V = np.linalg.svd(M, full_matrices=False)
        k = len(S)
        if trunc:
            w = np.cumsum(S[::-1] ** 2)[::-1] / np.sum(S ** 2)
            if self.cutoff:
                k = max(1, int(np.sum(w > self.cutoff)))
            k = min(k, self.maxdim) if self.maxdim else k
        return U[:, :k], S[:k], V[:k]

    def right(self, i, trunc=False):
        l, d, r = self.A[i].shape
        U, S, V = self.svd(self.A[i].reshape(l * d, r), trunc)
        self.A[i] = U.reshape(l, d, -1)
        self.A[i + 1] = np.tensordot(S[:, None] * V, self.A[i + 1], 1)

    def left(self, i, trunc=False):
        l, d, r = self.A[i].shape
        U, S, V = self.svd(self.A[i].reshape(l, d * r), trunc)
        self.A[i] = V.reshape(-1, d, r)
        self.A[i - 1] = np.tensordot(self.A[i - 1], U * S, 1)

    def move(self, to, trunc=False):
        if self.c is None:
            for i in range(to):
                self.right(i, trunc)
            for i in range(self.N - 1, to, -1):
                self.left(i, trunc)
        else:
            for i in range(self.c, to):
                self.right(i, trunc)
            for i in range(self.c, to, -1):
                self.left(i, trunc)
        self.c = to

    def norm(self):
        return float(np.linalg.norm(self.A[self.c]))

    def normalize(self):
        self.A[self.c] = self.A[self.c] / self.norm()

    def gate(self, i, g, leftward):
        """g[(o1 o2), (i1 i2)] on sites i, i+1, or g[o, i] on site i."""
        if g.shape[0] == 2:
            self.A[i] = np.einsum("oi,aib->aob", g, self.A[i])
            nxt = i - 1 if leftward else i + 1
            if 0 <= nxt < self.N:
                self.move(nxt)
            return
        l, r = self.A[i].shape[0], self.A[i + 1].shape[2]
        th = np.tensordot(self.A[i], self.A[i + 1], 1)
        th = np.einsum("opij,aijb->aopb", g.reshape(2, 2, 2, 2), th).reshape(2 * l, 2 * r)
        U, S, V = self.svd(th, True)
        if leftward:
            U = U * S
        else:
            V = S[:, None] * V
        self.A[i], self.A[i + 1] = U.reshape(l, 2, -1), V.reshape(-1, 2, r)
        self.c = i if leftward else i + 1


def _plain_inner(ts, terms):
    """<psi|term|psi> of every term of an OpList."""
    N = len(ts)
    step = lambda L, A, B: np.tensordot(np.tensordot(L, B, 1).transpose(1, 0, 2).reshape(  # noqa: E731
        -1, B.shape[2]).T, A.transpose(1, 0, 2).reshape(-1, A.shape[2]).conj(), 1).T
    Ls, Rs = [np.ones((1, 1), complex)], [None] * N + [np.ones((1, 1), complex)]
    for A in ts:
        Ls.append(step(Ls[-1], A, A))
    for i in range(N - 1, -1, -1):
        Rs[i] = step(Rs[i + 1], ts[i].transpose(2, 1, 0), ts[i].transpose(2, 1, 0))
    out = []
    for ops, sites, c in zip(terms.ops, terms.sites, terms.coeffs):
        L = Ls[sites[0] - 1]
        for o, s in zip(ops, sites):
            L = step(L, ts[s - 1], np.einsum("oi,aib->aob", OPS[o], ts[s - 1]))
        out.append(c * np.sum(L * Rs[sites[-1]]))
    return np.asarray(out)


def _plain_gates(N):
    """Second-order rows of the quench: [(first site, gate)], even, odd, even."""
    rows = []
    for i0, tau in ((0, 0.5), (1, 1.0)):
        row = []
        for i in range(i0, N, 2):
            h = TEBD_FIELD * (-1) ** (i + 1) * OPS["z"]
            if i + 1 < N:
                h = np.kron(h, np.eye(2)) + sum(c * np.kron(OPS[o], OPS[o]) for o, c in (
                    ("x", 1.0), ("y", 1.0), ("z", TEBD_DELTA)))
            e, v = np.linalg.eigh(h)
            row.append((i, (v * np.exp(-1j * tau * TEBD_DT * e)) @ v.conj().T))
        rows.append(row)
    return rows + rows[:1]


def _plain_tebd(psi, N, steps):
    rows = _plain_gates(N)
    for _ in range(steps):
        for row in rows:
            a, b = row[0][0], row[-1][0] + (2 if row[-1][1].shape[0] == 4 else 1) - 1
            leftward = not abs(psi.c - a) < abs(psi.c - b)
            for i, g in (row[::-1] if leftward else row):
                psi.move(i + (1 if leftward and g.shape[0] == 4 else 0), True)
                psi.gate(i, g, leftward)
        psi.normalize()


def exact(case, seed):
    k, N = case["kind"], case["N"]
    if k == "measure":
        p = _Plain(_mps_arrays(seed, N, case["chi"]))
        p.move(0)
        p.normalize()
        return {"terms": _plain_inner(p.A, _xxz(N) + _local(N))}
    if k == "canonical":
        p = _Plain(_mps_arrays(seed, N, case["chi"]), 1e-12, case["maxdim"])
        p.move(N - 1)
        p.move(0, True)
        norm = p.norm()
        p.normalize()
        dims = np.asarray([1] + [A.shape[2] for A in p.A])
        p.move(N // 2 - 1)
        a = p.A[p.c]
        S = np.linalg.svd(a.reshape(-1, a.shape[2]), compute_uv=False)
        return {"norm": norm, "dims": dims, "spectrum": _pad(S, case["maxdim"])}
    if k == "tebd" and case["precision"] == "fp64" and case["steps"] * N * case["chi"] ** 3 < 2e8:
        if case["chi"] == 1:
            up = np.random.default_rng([seed, N]).permutation(N) < N // 2
            ts = [np.reshape([1.0, 0.0] if u else [0.0, 1.0], (1, 2, 1)) for u in up]
        else:
            ts = _mps_arrays(seed, N, case["chi"])
        p = _Plain(ts, 1e-10, case["maxdim"])
        p.move(0)
        p.normalize()
        obs, H = _local(N) + _xxz(N), _xxz(N, TEBD_DELTA, TEBD_FIELD)
        first = _plain_inner(p.A, obs)
        _plain_tebd(p, N, case["steps"])
        return {"energy": np.asarray(np.sum(_plain_inner(p.A, H)).real),
                "obs": np.stack([first, _plain_inner(p.A, obs)]),
                "dims": np.asarray([1] + [A.shape[2] for A in p.A])}
    return None  # an iterative solver or a stochastic average: no closed 64-bit value in 20 s
