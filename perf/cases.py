"""Performance cases: the calls a user of the exact-diagonalisation library
makes, each through a public entry point, over the range of sizes it serves.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges,
``prepare`` makes what a program holds before the call (handles, start
states, device panels), ``run`` is one pass, ``work`` counts what the pass
cannot do without and ``exact`` gives the same outputs in plain FP64 torch.

Kinds of case:

* ``gs``      ground states and their observables of K coupling points on one
  basis (lgt_ground_state_observe with a device panel);
* ``batch``   ground states of several lattices in one call;
* ``solve``   find_ground_state into host arrays;
* ``hpsi``    one H*psi on device panels;
* ``quench``  exp(-iHt) steps with observables, device panel;
* ``evolve``  evolve_ED from host arrays;
* ``basis``   build_basis and a key lookup;
* ``measure`` measure_ED of host states.

Results of "fp32_mixed" calls other than the energies carry the accuracy of
FP32 Krylov vectors (unrefined), so they are kept as float32.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import lgt_gb300 as lgt
from lgt_gb300 import _capi as C

STEPS_GUESS = 25  # Lanczos steps a ground state takes at the least (work())

# sector dimension, off-diagonal entries (reference model, plaquette model)
SIZES = {
    (3, 2, "stag"): (90, 344, 520), (2, 3, "stag"): (90, 344, 520),
    (4, 2, "stag"): (645, 3372, 5198), (2, 4, "stag"): (645, 3372, 5198),
    (3, 3, "stag"): (2443, 14584, 23304),
    (4, 3, "stag"): (72211, 597404, 970292), (3, 4, "stag"): (72211, 597404, 970292),
    (4, 4, "stag"): (8563545, 97480968, 161709772),
    (3, 4, "string"): (1020, 2538, 7478), (3, 3, "string"): (134, 306, 742),
}


def listed():
    return [
        # the smallest call: one FP64 point of the 3x2 lattice at a tight
        # tolerance (latency of one solve, launches and copies)
        dict(name="gs_3x2_fp64", kind="solve", nx=3, ny=2, K=1, model="ref", precision="fp64",
             tol=1e-12, refine=0),
        # the headline sweep: 64 couplings of the 4x2 lattice, mixed precision
        dict(name="gs_4x2_mixed_k64", kind="gs", nx=4, ny=2, K=64, model="ref",
             precision="fp32_mixed", tol=1e-10),
        # the same sweep in FP64 under the plaquette + Jordan-Wigner model
        dict(name="gs_4x2_pjw_fp64_k64", kind="gs", nx=4, ny=2, K=64, model="pjw",
             precision="fp64", tol=1e-10),
        # lattices of uneven size in one call, 16 (g, m) points each
        dict(name="gs_uneven_mixed_k16", kind="batch", lattices="3x2,4x2,3x3,4x3", K=16,
             model="ref", precision="fp32_mixed", tol=1e-10),
        # the 5 x 5 (m, g) ground-state grid on 3x4 (an odd panel width)
        dict(name="gs_grid_3x4_fp64_k25", kind="solve", nx=3, ny=4, K=25, model="ref",
             precision="fp64", tol=1e-10, refine=0),
        # one 4x3 point, mixed precision finished in FP64
        dict(name="gs_4x3_mixed_refined", kind="solve", nx=4, ny=3, K=1, model="ref",
             precision="fp32_mixed", tol=1e-10, refine=12),
        # one product on the largest panel (the inner kernel of a quench)
        dict(name="hpsi_4x4_fp32_k8", kind="hpsi", nx=4, ny=4, K=8, ncomp=2, model="ref",
             precision="fp32"),
        # a small ragged FP64 product: five real columns
        dict(name="hpsi_4x3_pjw_fp64_k5", kind="hpsi", nx=4, ny=3, K=5, ncomp=1, model="pjw",
             precision="fp64"),
        # the 4x4 quench panel in mixed precision, two steps of dt = 0.05
        dict(name="quench_4x4_mixed_k8", kind="quench", nx=4, ny=4, K=8, model="ref",
             precision="fp32_mixed", dt=0.05, steps=2),
        # the same lattice in FP64 with plaquettes, fewer points, one step
        dict(name="quench_4x4_pjw_fp64_k3", kind="quench", nx=4, ny=4, K=3, model="pjw",
             precision="fp64", dt=0.05, steps=1),
        # the 3x4 quench protocols: one point, FP64, dt = 0.02, from host arrays
        dict(name="evolve_3x4_fp64", kind="evolve", nx=3, ny=4, sector="stag", K=1,
             model="ref", precision="fp64", dt=0.02, steps=10),
        # the largest basis and a block of key lookups
        dict(name="basis_4x4_lookup", kind="basis", nx=4, ny=4, n=100000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gs", "solve", "batch", "hpsi", "quench", "evolve", "basis", "measure"])
    model = rng.choice(["ref", "pjw"])
    prec = rng.choice(["fp64", "fp32_mixed"])
    small = [(3, 2), (2, 3), (4, 2), (2, 4), (3, 3)]
    mid = [(4, 3), (3, 4)]
    if kind == "gs":
        nx, ny = rng.choice(small)
        return dict(kind=kind, nx=nx, ny=ny, K=_log_int(rng, 1, 100), model=model, precision=prec,
                    tol=1e-10)
    if kind == "solve":
        nx, ny = rng.choice(small + mid)
        big = nx * ny == 12
        return dict(kind=kind, nx=nx, ny=ny, K=_log_int(rng, 1, 24 if big else 100), model=model,
                    precision=prec, tol=1e-10,
                    refine=rng.choice([0, 12]) if prec == "fp32_mixed" else 0)
    if kind == "batch":
        names = ["3x2", "4x2", "3x3", "2x4"] + (["4x3"] if rng.random() < 0.5 else [])
        k = rng.randint(2, len(names))
        return dict(kind=kind, lattices=",".join(rng.sample(names, k)), K=_log_int(rng, 1, 16),
                    model=model, precision=prec, tol=1e-10)
    if kind == "hpsi":
        nx, ny = rng.choice([(3, 3), (4, 3), (3, 4), (4, 4)])
        return dict(kind=kind, nx=nx, ny=ny, K=_log_int(rng, 1, 8 if nx * ny == 16 else 33),
                    ncomp=rng.choice([1, 2]), model=model, precision=rng.choice(["fp64", "fp32"]))
    if kind == "quench":
        nx, ny = rng.choice([(3, 3), (4, 3), (3, 4), (4, 4)])
        if nx * ny == 16:
            return dict(kind=kind, nx=nx, ny=ny, K=rng.randint(1, 8 if prec != "fp64" else 3),
                        model=model, precision=prec, dt=round(rng.uniform(0.02, 0.05), 4), steps=1)
        return dict(kind=kind, nx=nx, ny=ny, K=_log_int(rng, 1, 16), model=model, precision=prec,
                    dt=round(rng.uniform(0.01, 0.1), 4), steps=rng.randint(1, 6))
    if kind == "evolve":
        return dict(kind=kind, nx=3, ny=rng.choice([3, 4]), sector=rng.choice(["string", "stag"]),
                    K=rng.randint(1, 5), model=model, precision=prec,
                    dt=round(rng.uniform(0.01, 0.05), 4), steps=rng.randint(1, 10))
    if kind == "basis":
        nx, ny = rng.choice(small + mid + [(4, 4)])
        return dict(kind=kind, nx=nx, ny=ny, n=_log_int(rng, 1, 100000))
    nx, ny = rng.choice([(4, 2), (3, 3), (4, 3), (3, 4)])
    return dict(kind=kind, nx=nx, ny=ny, K=_log_int(rng, 1, 33), cplx=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _charges(case, nx, ny):
    if case.get("sector", "stag") == "string":
        return lgt.string_charges(nx, ny)
    return lgt.staggered_charges(nx, ny)


def _couplings(case, seed):
    """K coupling points (g, m) from the seed, the distributions of the
    framework's own sweeps; hopping 1."""
    rng = np.random.default_rng(seed)
    K = case.get("K", 1)
    kind = case["kind"]
    if kind == "batch":
        return [(np.exp(rng.uniform(np.log(0.3), np.log(3.0), K)), rng.uniform(0.0, 1.0, K))
                for _ in case["lattices"].split(",")]
    if kind in ("quench", "evolve"):
        return rng.uniform(0.5, 1.5, K), np.full(K, 0.5 if kind == "quench" else 2.0)
    if K == 25:  # the (m, g) grid, each value moved by up to 5 %
        vals = np.array([0.25, 0.5, 1.0, 2.0, 4.0])
        g, m = np.repeat(vals, 5), np.tile(vals, 5)
        return g * rng.uniform(0.95, 1.05, K), m * rng.uniform(0.95, 1.05, K)
    return rng.uniform(0.5, 2.0, K), np.full(K, 0.5)


def _split(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["lattices"].split(",")]


def _product_index(case, nx, ny):
    """1-based basis index of the quench's start state is looked up by the
    library; the same configuration as (n_f, e_R, e_U) for exact()."""
    nf = np.zeros((nx, ny), np.int8)
    eR = np.zeros((nx - 1, ny), np.int8)
    eU = np.zeros((nx, ny - 1), np.int8)
    if case.get("sector", "stag") == "string":
        nf[1, ny // 2 - 1] = 1
        eR[0, ny // 2 - 1] = 1
    else:
        for ix in range(nx):
            for iy in range(ny):
                nf[ix, iy] = (ix + iy) % 2
    return nf, eR, eU


def _panel_input(case, seed, N, cols):
    """Random normal columns of unit norm (FP64, on the GPU)."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    x = torch.randn((N, cols), generator=gen, device="cuda", dtype=torch.float64)
    return x / x.norm(dim=0, keepdim=True)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "seed": int(seed)}
    if kind == "batch":
        s["H"], s["psi"] = [], []
        for (nx, ny), (g, m) in zip(_split(case), _couplings(case, seed)):
            b, _ = lgt.build_basis(nx, ny, 1, lgt.staggered_charges(nx, ny))
            s["H"].append(lgt.build_hamiltonian(b, g=g, t=1.0, m=m, model=case["model"]))
            s["psi"].append(torch.zeros((len(b), case["K"]), dtype=torch.float64, device="cuda"))
        torch.cuda.synchronize()
        return s
    nx, ny = case["nx"], case["ny"]
    if kind == "basis":
        b, _ = lgt.build_basis(nx, ny, 1, lgt.staggered_charges(nx, ny))
        rng = np.random.default_rng(seed)
        if len(b) <= case["n"]:
            keys = b.ref_keys()[rng.integers(0, len(b), case["n"])]
        else:
            at = int(rng.integers(0, len(b) - case["n"] + 1))
            keys = rng.permutation(b.ref_keys(at, case["n"]))
        # every eighth key is of a configuration that need not be in the basis
        flip = np.zeros(case["n"], np.int64)
        flip[::8] = np.int64(1) << rng.integers(0, nx * ny, flip[::8].size)
        b.close()
        s["charges"], s["keys"] = lgt.staggered_charges(nx, ny), keys ^ flip
        return s
    b, kd = lgt.build_basis(nx, ny, 1, _charges(case, nx, ny))
    s["b"], s["kd"] = b, kd
    N = len(b)
    if kind == "measure":
        x = _panel_input(case, seed, N, case["K"] * (2 if case["cplx"] else 1)).cpu().numpy()
        if case["cplx"]:
            x = (x[:, ::2] + 1j * x[:, 1::2]) / math.sqrt(2.0)
        s["psi"] = np.ascontiguousarray(x)
        return s
    g, m = _couplings(case, seed)
    K = case["K"]
    s["H"] = lgt.build_hamiltonian(b, g=g, t=1.0, m=m, model=case["model"])
    if kind == "gs":
        ns, npl = nx * ny, (nx - 1) * (ny - 1)
        s["psi"] = torch.zeros((N, K), dtype=torch.float64, device="cuda")
        o = C.defaults(False)
        o.tol = case["tol"]
        o.precision = C.LGT_FP64 if case["precision"] == "fp64" else C.LGT_FP32_MIXED
        o.seed = s["seed"]
        s["opts"], s["E0"], s["obs"] = o, np.zeros(K), (C.Obs * K)()
        s["nf"], s["e2"], s["pl"] = np.zeros((K, ns)), np.zeros((K, ns)), np.zeros((K, npl))
    elif kind == "hpsi":
        dt = torch.float64 if case["precision"] == "fp64" else torch.float32
        s["x"] = _panel_input(case, seed, N, K * case["ncomp"]).to(dt)
        s["y"] = torch.zeros_like(s["x"])
    elif kind in ("quench", "evolve"):
        v = lgt.string_state(b) if case.get("sector") == "string" else lgt.staggered_product_state(b)
        if kind == "evolve":
            s["psi0"] = v if K == 1 else np.repeat(v[:, None], K, axis=1)
        else:
            R, ns = (case["steps"] + 1) * K, nx * ny
            s["at"] = int(np.argmax(np.abs(v)))
            s["psi"] = torch.zeros((N, K, 2), dtype=torch.float64, device="cuda")
            o = C.defaults(True)
            o.precision = C.LGT_FP64 if case["precision"] == "fp64" else C.LGT_FP32_MIXED
            s["opts"], s["obs"] = o, (C.Obs * R)()
            s["nf"], s["e2"] = np.zeros((R, ns)), np.zeros((R, ns))
            s["pl"], s["drift"] = np.zeros((R, (nx - 1) * (ny - 1))), np.zeros(K)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _vec(a):
    return a.ctypes.data


def _by_precision(case, v):
    """Amplitudes and observables at the accuracy of the solve."""
    if case["precision"] == "fp64" or case.get("refine"):
        return v
    if isinstance(v, np.ndarray):
        return v.astype(np.float32)
    return v.to(torch.float32)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solve":
        E0, psi = lgt.find_ground_state(s["H"], tol=case["tol"], precision=case["precision"],
                                        refine_steps=case["refine"], seed=s["seed"],
                                        as_complex=False)
        return {"E0": E0, "psi": _by_precision(case, psi)}
    if kind == "gs":
        info = C.Info()
        C.check(C.load().lgt_ground_state_observe(
            s["H"].handle, ctypes.byref(s["opts"]), _vec(s["E0"]), s["psi"].data_ptr(), None,
            C.LGT_DEVICE_PTRS, ctypes.byref(info), _vec(s["nf"]), _vec(s["e2"]), _vec(s["pl"]),
            s["obs"]))
        return {"E0": s["E0"].copy(), "psi": _by_precision(case, s["psi"]),
                "obs": _by_precision(case, np.hstack((s["nf"], s["e2"], s["pl"])))}
    if kind == "batch":
        out = lgt.find_ground_states(s["H"], tol=case["tol"], precision=case["precision"],
                                     seed=s["seed"], device_psi=[p.data_ptr() for p in s["psi"]])
        return {"E0": [e for e, _ in out], "psi": [_by_precision(case, p) for p in s["psi"]]}
    if kind == "hpsi":
        s["H"].matvec_device(s["x"].data_ptr(), s["y"].data_ptr(), ncomp=case["ncomp"],
                             precision=case["precision"])
        return s["y"]
    if kind == "quench":
        psi = s["psi"]
        psi.zero_()
        psi[s["at"], :, 0] = 1.0
        torch.cuda.current_stream().synchronize()  # the library runs on the basis' stream
        info = C.Info()
        C.check(C.load().lgt_expm_steps_grids(
            s["H"].handle, ctypes.byref(s["opts"]), case["dt"], case["steps"], psi.data_ptr(),
            s["obs"], _vec(s["nf"]), _vec(s["e2"]), _vec(s["pl"]), _vec(s["drift"]),
            C.LGT_DEVICE_PTRS, ctypes.byref(info)))
        return {"psi": _by_precision(case, psi),
                "obs": _by_precision(case, np.hstack((s["nf"], s["e2"], s["pl"])))}
    if kind == "evolve":
        data, psi, _ = lgt.evolve_ED(s["psi0"], s["H"], dt=case["dt"], n_steps=case["steps"],
                                     precision=case["precision"], return_state=True)
        flat = data if case["K"] == 1 else [d for step in data for d in step]
        e2 = np.array([d["E2_mean"] for d in flat])
        nf = np.array([d["nf_mean"] for d in flat])
        grid = np.stack([d["nf_grid"] for d in flat])
        if case["precision"] != "fp64":
            psi = psi.astype(np.complex64)
        return {"psi": psi, "e2": _by_precision(case, e2), "nf": _by_precision(case, nf),
                "grid": _by_precision(case, grid)}
    if kind == "basis":
        b, _ = lgt.build_basis(case["nx"], case["ny"], 1, s["charges"])
        out = {"dim": len(b), "index": b.lookup(s["keys"])}
        b.close()
        return out
    obs = lgt.measure_ED(s["psi"], s["b"])
    return {"e2": np.array([d["E2_mean"] for d in obs]),
            "nf": np.stack([d["nf_grid"] for d in obs]),
            "plaq": np.stack([d["plaq_grid"] for d in obs])}  # one record per state


def work(case):
    """Compulsory bytes and floating-point operations of one pass: inputs and
    outputs once, the products a solver cannot do without."""
    kind = case["kind"]
    if kind == "batch":
        parts = [work(dict(case, kind="gs", nx=nx, ny=ny)) for nx, ny in _split(case)]
        return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}
    nx, ny = case["nx"], case["ny"]
    N, ref, pjw = SIZES[(nx, ny, case.get("sector", "stag"))]
    if kind == "basis":
        return {"bytes": 8.0 * N + 16.0 * case["n"], "flops": 0.0}
    K = case["K"]
    nnz = ref if case.get("model") == "ref" else pjw
    ns, npl = nx * ny, (nx - 1) * (ny - 1)
    if kind == "measure":
        C_ = K * (2 if case["cplx"] else 1)
        return {"bytes": 8.0 * N + 8.0 * N * C_, "flops": 2.0 * N * C_ * (2 * ns + npl + 1)}
    if kind in ("solve", "gs"):
        # products, and the orthogonalisation of each new vector against the
        # two before it
        return {"bytes": 8.0 * N * (1 + K),
                "flops": STEPS_GUESS * K * (2.0 * (nnz + N) + 10.0 * N)}
    if kind == "hpsi":
        e = 8.0 if case["precision"] == "fp64" else 4.0
        C_ = K * case["ncomp"]
        return {"bytes": 8.0 * N + 2 * e * N * C_, "flops": 2.0 * C_ * (nnz + N)}
    # time steps: about ten products each, the state read and written once
    return {"bytes": 8.0 * N + case["steps"] * 32.0 * N * K,
            "flops": case["steps"] * 10 * 4.0 * K * (nnz + N)}


# ---------------------------------------------------------------------------
# the same outputs in plain FP64
# ---------------------------------------------------------------------------

class _Sector:
    """Basis and moves of one sector, from the Gauss law alone.

    States are (mask, e_U digits) in ascending order of mask, then of the e_U
    values link by link; e_R follows from the Gauss law
    e_R(ix) = e_R(ix-1) + n + g - e_U(iy) + e_U(iy-1)."""

    def __init__(self, nx, ny, charges, dev):
        self.nx, self.ny, self.dev = nx, ny, dev
        ns, nu = nx * ny, nx * (ny - 1)
        self.ns, self.nu = ns, nu
        q = torch.tensor(np.asarray(charges).T.ravel().copy(), dtype=torch.int64, device=dev)
        masks = torch.arange(1 << ns, dtype=torch.int64, device=dev)
        pop = torch.zeros_like(masks)
        for b in range(ns):
            pop += (masks >> b) & 1
        mask = masks[pop == int(-q.sum())]
        dig = torch.zeros_like(mask)           # base-4 digits e_U + 1, first link on top
        eu = torch.zeros((mask.numel(), nx), dtype=torch.int8, device=dev)  # the row below
        er = torch.zeros_like(mask)
        for iy in range(ny):
            er.zero_()
            for ix in range(nx):
                c = iy * nx + ix
                inc = ((mask >> c) & 1) + q[c] + eu[:, ix].to(torch.int64)
                if iy < ny - 1:
                    parts = mask.numel()
                    u = torch.tensor([-1, 0, 1], dtype=torch.int64, device=dev).repeat(parts)
                    r = (er + inc).repeat_interleave(3) - u
                    ok = (r.abs() <= 1) if ix < nx - 1 else (r == 0)
                    keep = ok.nonzero().squeeze(1)
                    src = keep // 3
                    u, er = u[keep], r[keep]
                    mask, dig, eu = mask[src], dig[src] * 4 + (u + 1), eu[src]
                    eu[:, ix] = u.to(torch.int8)
                else:
                    r = er + inc
                    ok = (r.abs() <= 1) if ix < nx - 1 else (r == 0)
                    keep = ok.nonzero().squeeze(1)
                    mask, dig, eu, er = mask[keep], dig[keep], eu[keep], r[keep]
        self.mask, self.dig = mask, dig
        self.key = (mask << (2 * nu)) | dig
        self.N = mask.numel()
        # link values, int8
        self.eU = [[((dig >> (2 * (nu - 1 - (iy * nx + ix)))) & 3).to(torch.int8) - 1
                    for ix in range(nx)] for iy in range(ny - 1)]
        self.eR = []
        for iy in range(ny):
            row, acc = [], torch.zeros_like(mask)
            for ix in range(nx - 1):
                c = iy * nx + ix
                acc = acc + ((mask >> c) & 1) + q[c]
                if iy < ny - 1:
                    acc = acc - self.eU[iy][ix]
                if iy > 0:
                    acc = acc + self.eU[iy - 1][ix]
                row.append(acc.to(torch.int8))
            self.eR.append(row)
        self.e2 = sum((e.to(torch.int64) ** 2 for rows in (self.eR, self.eU) for r in rows
                       for e in r), torch.zeros_like(mask))
        self.stag = sum(((mask >> (iy * nx + ix)) & 1) * (1 if (ix + iy) % 2 == 0 else -1)
                        for iy in range(ny) for ix in range(nx))
        self._moves = {}

    def n(self, c):
        return (self.mask >> c) & 1

    def unit(self, j):
        return 1 << (2 * (self.nu - 1 - j))

    def index(self, key):
        return torch.searchsorted(self.key, key)

    def moves(self, model):
        """[(rows, columns, sign or None, "hop" or "plaq")]; for every listed
        entry (i, j) H also holds (j, i)."""
        if model in self._moves:
            return self._moves[model]
        nx, ny = self.nx, self.ny
        out = []

        def add(ok, dmask, ddig, sign, kind):
            rows = ok.nonzero().squeeze(1)
            key = self.key[rows] + (dmask << (2 * self.nu)) + ddig
            out.append((rows, self.index(key), None if sign is None else sign[rows], kind))

        def pos(ix, iy):  # column snake
            return ix * ny + (iy if ix % 2 == 0 else ny - 1 - iy)

        for iy in range(ny):
            for ix in range(nx - 1):
                c = iy * nx + ix
                ok = (self.n(c) == 0) & (self.n(c + 1) == 1) & (self.eR[iy][ix] < 1)
                sign = None
                if model == "pjw":
                    lo, hi = sorted((pos(ix, iy), pos(ix + 1, iy)))
                    par = torch.zeros_like(self.mask)
                    for jy in range(ny):
                        for jx in range(nx):
                            if lo < pos(jx, jy) < hi:
                                par ^= self.n(jy * nx + jx)
                    sign = 1.0 - 2.0 * par.to(torch.float64)
                add(ok, (1 << c) - (1 << (c + 1)), 0, sign, "hop")
        for iy in range(ny - 1):
            for ix in range(nx):
                c = iy * nx + ix
                ok = (self.n(c) == 0) & (self.n(c + nx) == 1) & (self.eU[iy][ix] < 1)
                add(ok, (1 << c) - (1 << (c + nx)), self.unit(c), None, "hop")
        if model == "pjw":
            for iy in range(ny - 1):
                for ix in range(nx - 1):
                    add(*self.plaq_args(ix, iy), None, "plaq")
        self._moves[model] = out
        return out

    def plaq_args(self, ix, iy):
        ok = ((self.eR[iy][ix] > -1) & (self.eU[iy][ix] < 1) & (self.eU[iy][ix + 1] > -1) &
              (self.eR[iy + 1][ix] < 1))
        j = iy * self.nx + ix
        return ok, 0, self.unit(j) - self.unit(j + 1)

    def apply(self, x, g, m, model):
        """H x for x [N, K, comp] (hopping 1)."""
        d = self.e2[:, None] * (0.5 * g * g)[None, :] + self.stag[:, None] * m[None, :]
        y = d.to(torch.float64)[:, :, None] * x
        cp = (-1.0 / (2.0 * g * g))[None, :, None]
        for rows, cols, sign, kind in self.moves(model):
            if kind == "plaq":
                y.index_add_(0, rows, cp * x[cols])
                y.index_add_(0, cols, cp * x[rows])
            elif sign is None:
                y.index_add_(0, rows, -x[cols])
                y.index_add_(0, cols, -x[rows])
            else:
                w = -sign[:, None, None]
                y.index_add_(0, rows, w * x[cols])
                y.index_add_(0, cols, w * x[rows])
        return y

    def observe(self, x):
        """(n_f [K, ns], E^2 [K, ns], plaquettes [K, np]) of x [N, K, comp]."""
        nx, ny = self.nx, self.ny
        p = (x * x).sum(2)
        nf, e2, pl = [], [], []
        for iy in range(ny):
            for ix in range(nx):
                nf.append(self.n(iy * nx + ix).to(torch.float64) @ p)
                e = torch.zeros(self.N, dtype=torch.float64, device=self.dev)
                if ix < nx - 1:
                    e += self.eR[iy][ix].to(torch.float64) ** 2
                if iy < ny - 1:
                    e += self.eU[iy][ix].to(torch.float64) ** 2
                e2.append(e @ p)
        for iy in range(ny - 1):
            for ix in range(nx - 1):
                ok, _, dd = self.plaq_args(ix, iy)
                rows = ok.nonzero().squeeze(1)
                cols = self.index(self.key[rows] + dd)
                pl.append(2.0 * (x[rows] * x[cols]).sum((0, 2)))
        empty = torch.zeros((x.shape[1], 0), dtype=torch.float64, device=self.dev)
        return (torch.stack(nf, 1), torch.stack(e2, 1), torch.stack(pl, 1) if pl else empty)


_sectors = {}


def _sector(case, nx, ny):
    key = (nx, ny, case.get("sector", "stag"))
    if key not in _sectors:
        for k in [k for k in _sectors if k[0] * k[1] == 16]:
            del _sectors[k]  # one sector of this size at a time
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        _sectors[key] = _Sector(nx, ny, _charges(case, nx, ny), dev)
    return _sectors[key]


def _mix(x):
    with np.errstate(over="ignore"):
        x = x + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return x ^ (x >> np.uint64(31))


def _start(seed, N, K):
    """The documented start vectors normal(seed, k): they fix the sign of the
    returned state (a positive overlap with its start)."""
    with np.errstate(over="ignore"):
        k = np.arange(K, dtype=np.uint64)[None, :]
        r = np.arange(N, dtype=np.uint64)[:, None]
        h = _mix(_mix(np.full((1, 1), seed, np.uint64)) ^ _mix(k + np.uint64(0x5851F42D4C957F2D)))
        h = _mix(h ^ r)
        h2 = _mix(h)
    u1 = ((h >> np.uint64(11)).astype(np.float64) + 1.0) * 2.0 ** -53
    u2 = (h2 >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
    return np.sqrt(-2.0 * np.log(u1)) * np.cos(2.0 * np.pi * u2)


def _ground(S, g, m, model, seed):
    """Lowest eigenpairs (E [K], x [N, K]) in FP64."""
    N, K, dev = S.N, g.numel(), S.dev
    v0 = torch.tensor(_start(seed, N, K), device=dev)
    if N <= 128:
        E, X = [], []
        for k in range(K):
            one = torch.eye(N, dtype=torch.float64, device=dev)[:, :, None]
            A = S.apply(one, g[k].expand(N), m[k].expand(N), model)[:, :, 0]
            w, z = torch.linalg.eigh(A.cpu())
            E.append(w[0])
            X.append(z[:, 0].to(dev))
        E, x = torch.stack(E).to(dev), torch.stack(X, 1)
    else:
        x = v0 / v0.norm(dim=0)
        for _ in range(12):  # Lanczos with full reorthogonalisation, restarted
            M = min(N, 100)
            V = torch.zeros((M, N, K), dtype=torch.float64, device=dev)
            T = torch.zeros((K, M, M), dtype=torch.float64, device=dev)
            V[0] = x
            for j in range(M):
                w = S.apply(V[j][:, :, None], g, m, model)[:, :, 0]
                T[:, j, j] = (w * V[j]).sum(0)
                for _ in range(2):
                    h = torch.einsum("jnk,nk->jk", V[:j + 1], w)
                    w = w - torch.einsum("jnk,jk->nk", V[:j + 1], h)
                if j + 1 < M:
                    b = w.norm(dim=0)
                    T[:, j, j + 1] = T[:, j + 1, j] = b
                    V[j + 1] = w / b.clamp_min(1e-290)
            _, z = torch.linalg.eigh(T.cpu())
            x = torch.einsum("jnk,kj->nk", V, z[:, :, 0].to(dev))
            x = x / x.norm(dim=0)
            hx = S.apply(x[:, :, None], g, m, model)[:, :, 0]
            E = (x * hx).sum(0)
            if float((hx - E * x).norm(dim=0).max()) < 1e-12:
                break
    return E, x * torch.sign((x * v0).sum(0))


def _evolve(S, x, g, m, model, dt, steps, t_end_only=False):
    """Normalised exp(-iH dt) steps of x [N, K, 2]; yields x after each."""
    bound = float((S.e2.max() * 0.5 * g.max() ** 2 + S.stag.abs().max() * m.abs().max() +
                   2 * S.ns + S.ns / g.min() ** 2))
    parts = max(1, math.ceil(bound * dt / 4.0))
    h = dt / parts
    for _ in range(steps):
        for _ in range(parts):
            term, out = x, x.clone()
            for n in range(1, 60):
                y = S.apply(term, g, m, model)
                term = torch.stack((y[..., 1], -y[..., 0]), 2) * (h / n)
                out += term
                if float(term.abs().max()) < 1e-19:
                    break
            x = out
        x = x / (x * x).sum((0, 2), keepdim=True).sqrt()
        yield x


def exact(case, seed):
    kind = case["kind"]
    if kind == "basis":
        return None  # whole numbers only
    if kind == "batch":
        out = {"E0": [], "psi": []}
        for (nx, ny), (g, m) in zip(_split(case), _couplings(case, seed)):
            S = _sector(case, nx, ny)
            E, x = _ground(S, torch.tensor(g, device=S.dev), torch.tensor(m, device=S.dev),
                           case["model"], seed)
            out["E0"].append(E.cpu().numpy())
            out["psi"].append(x)
        return out
    nx, ny = case["nx"], case["ny"]
    S = _sector(case, nx, ny)
    if kind == "measure":
        K = case["K"]
        x = _panel_input(case, seed, S.N, K * (2 if case["cplx"] else 1))
        x = x.reshape(S.N, K, 2) / math.sqrt(2.0) if case["cplx"] else x[:, :, None]
        nf, e2, pl = S.observe(x)

        def grid(a, a1, a2):
            return a.reshape(K, a2, a1).transpose(1, 2).cpu().numpy()
        # E2_mean averages over the sites
        return {"e2": e2.mean(1).cpu().numpy(), "nf": grid(nf, nx, ny),
                "plaq": grid(pl, nx - 1, ny - 1)}
    g, m = (torch.tensor(v, device=S.dev) for v in _couplings(case, seed))
    K = case["K"]
    if kind == "solve":
        E, x = _ground(S, g, m, case["model"], seed)
        return {"E0": float(E[0]) if K == 1 else E.cpu().numpy(),
                "psi": (x[:, 0] if K == 1 else x).cpu().numpy()}
    if kind == "gs":
        E, x = _ground(S, g, m, case["model"], seed)
        return {"E0": E.cpu().numpy(), "psi": x,
                "obs": torch.cat(S.observe(x[:, :, None]), 1).cpu().numpy()}
    if kind == "hpsi":
        x = _panel_input(case, seed, S.N, K * case["ncomp"])
        if case["precision"] != "fp64":
            x = x.to(torch.float32).to(torch.float64)
        y = S.apply(x.reshape(S.N, K, case["ncomp"]), g, m, case["model"])
        return y.reshape(S.N, K * case["ncomp"])
    # time evolution from the product state
    nf0, _, eU0 = _product_index(case, nx, ny)
    key = sum(int(nf0[ix, iy]) << (iy * nx + ix) for ix in range(nx) for iy in range(ny))
    for iy in range(ny - 1):
        for ix in range(nx):
            key = key * 4 + int(eU0[ix, iy]) + 1
    x = torch.zeros((S.N, K, 2), dtype=torch.float64, device=S.dev)
    x[int(S.index(torch.tensor([key], device=S.dev))[0]), :, 0] = 1.0
    obs = [S.observe(x)]
    for x in _evolve(S, x, g, m, case["model"], case["dt"], case["steps"]):
        obs.append(S.observe(x))
    nf, e2, pl = (torch.cat([o[i] for o in obs]).cpu().numpy() for i in range(3))
    if kind == "quench":
        return {"psi": x, "obs": np.hstack((nf, e2, pl))}
    z = torch.view_as_complex(x.contiguous()).cpu().numpy()
    return {"psi": z[:, 0] if K == 1 else z, "e2": e2.mean(1), "nf": nf.mean(1),
            "grid": nf.reshape(-1, ny, nx).transpose(0, 2, 1)}
