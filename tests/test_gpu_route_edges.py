"""The default routes at the edges that their own tests leave out: expansion
panels of more than eight points, one-launch cycles whose neighbour lists stay
in global memory and those on either side of the widest panel that fits, the
plaquette role of the 4x4 observables, and two solvers at once.

Bars: exponentials as in the expansion's own test (1e-12 FP64, 2e-6 mixed, four
steps); ground states 1e-10 in energy, states 1e-8 (FP64) and 1e-3
(FP32-mixed); observables 1e-12 of the norm."""
import threading

import numpy as np
import pytest

import lgt_gb300 as lgt
from lgt_gb300 import _capi as C
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,bar", [("fp64", 1e-12), ("fp32_mixed", 2e-6)])
@pytest.mark.parametrize("model", ["ref", "pjw"])
@pytest.mark.parametrize("K", [12, 33, 85, 128])
def test_wide_expansion_panels(K, model, precision, bar):
    ch = lgt.staggered_charges(3, 2)
    b, _ = lgt.build_basis(3, 2, 1, ch)
    ob = O.build_basis(3, 2, 1, ch)
    g = np.linspace(0.6, 1.6, K)
    H = lgt.build_hamiltonian(b, g=g, t=0.9, m=0.4, model=model)
    rng = np.random.default_rng(K)
    psi = rng.normal(size=(len(b), K)) + 1j * rng.normal(size=(len(b), K))
    psi /= np.linalg.norm(psi, axis=0)
    _, out, drift = lgt.evolve_ED(psi, H, dt=0.07, n_steps=4, precision=precision,
                                  return_state=True)
    for k in range(K):
        w, z = np.linalg.eigh(O.build_hamiltonian(ob, g=g[k], t=0.9, m=0.4,
                                                  model=model).toarray())
        ref = z @ (np.exp(-1j * w * 0.28) * (z.T @ psi[:, k]))
        assert np.linalg.norm(out[:, k] - ref) <= bar
    assert np.max(drift) <= bar
    H.close()
    b.close()


# 72,211 states, krylovdim 50: lists in shared memory up to 33 (mixed) and 35
# columns (FP64), a block's rows up to 41 and 43
@pytest.mark.parametrize("precision,K,cycle", [
    ("fp32_mixed", 33, True), ("fp32_mixed", 34, True), ("fp32_mixed", 41, True),
    ("fp32_mixed", 42, False), ("fp64", 36, True), ("fp64", 43, True), ("fp64", 44, False)])
def test_widest_cycles(monkeypatch, precision, K, cycle):
    b, _ = lgt.build_basis(4, 3, 1, lgt.staggered_charges(4, 3))
    got, n = {}, {}
    for env in ("0", "1"):
        monkeypatch.setenv("LGT_PANEL_GRID", env)
        H = lgt.build_hamiltonian(b, g=np.geomspace(0.5, 2.5, K), t=1.0, m=0.5)
        if env == "0":  # (tunes the single launches)
            lgt.find_ground_state(H, precision=precision, as_complex=False)
        n0 = C.launch_count()
        got[env] = lgt.find_ground_state(H, precision=precision, seed=3, as_complex=False)
        n[env] = C.launch_count() - n0
        H.close()
    assert (n["1"] < n["0"] / 2) == cycle
    assert np.max(np.abs(got["1"][0] - got["0"][0]) / np.abs(got["0"][0])) <= 1e-10
    bar = 1e-8 if precision == "fp64" else 1e-3
    assert np.max(np.linalg.norm(got["1"][1] - got["0"][1], axis=0)) <= bar
    b.close()


@pytest.mark.parametrize("ncomp,K", [(2, 3), (1, 2)])
def test_4x4_plaquette_role(monkeypatch, ncomp, K):
    """Against the one-role FP64 sums (LGT_DF_REDUCTIONS=0)."""
    import torch
    b, _ = lgt.build_basis(4, 4, 1, lgt.staggered_charges(4, 4))
    H = lgt.build_hamiltonian(b, g=np.ones(K), t=1.0, m=0.5, model="pjw")
    N = len(b)
    gen = torch.Generator(device="cuda").manual_seed(K)
    x = torch.randn((N, K, ncomp), generator=gen, dtype=torch.float64, device="cuda")
    x += 0.5  # (plaquettes that do not cancel)
    x /= (x * x).sum((0, 2), keepdim=True).sqrt()
    torch.cuda.synchronize()
    out = {}
    for flag in ("1", "0"):
        monkeypatch.setenv("LGT_DF_REDUCTIONS", flag)
        nf, e2, pl = np.zeros((K, 16)), np.zeros((K, 16)), np.zeros((K, 9))
        C.check(C.load().lgt_observe(H.handle, x.data_ptr(), ncomp, C.LGT_FP64,
                                     C.LGT_DEVICE_PTRS, 0.0, nf.ctypes.data, e2.ctypes.data,
                                     pl.ctypes.data, (C.Obs * K)()))
        out[flag] = (nf, e2, pl)
    assert np.all(np.abs(out["0"][2]) > 1e-3)
    for a, r in zip(out["1"], out["0"]):
        assert np.max(np.abs(a - r)) <= 1e-12
    H.close()
    b.close()


def test_two_solvers_at_once():
    """One-launch cycles and expansions of two Hamiltonians on two bases, from
    two threads, give what they give one after the other."""
    def work(k):
        nx, ny = ((4, 3), (3, 4))[k]
        b, _ = lgt.build_basis(nx, ny, 1, lgt.staggered_charges(nx, ny))
        H = lgt.build_hamiltonian(b, g=[0.7, 1.1 + k], t=1.0, m=0.4)
        v = lgt.staggered_product_state(b)
        out = []
        for seed in range(4):
            out.append(lgt.find_ground_state(H, seed=seed, as_complex=False)[0])
            out.append(lgt.evolve_ED(np.stack([v, v], axis=1), H, dt=0.05, n_steps=2,
                                     return_state=True)[1])
        H.close()
        b.close()
        return out

    ref = [work(0), work(1)]
    got = [None, None]

    def run(k):
        got[k] = work(k)

    threads = [threading.Thread(target=run, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r, g in zip(ref, got):
        assert g is not None
        for a, c in zip(r, g):
            assert np.max(np.abs(a - c)) <= 1e-10
