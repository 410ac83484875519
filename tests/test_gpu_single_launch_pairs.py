"""The single-launch kernels of the panel drivers compared with each other where
the default routes (the expansion of cheb.cu, the one-launch cycle) would run
in both arms: LGT_EXPM=krylov and LGT_PANEL_GRID=0 hold the drivers to them.

Bars: streamed and register-load kernels add the same rows in the same order,
so FP32-mixed results are equal bit for bit.  Double-float and FP64 reductions
of FP32 panels, and both against exact propagation: panels rounded to 2^-24 at
each of some ten vectors and three steps, 1e-6."""
import numpy as np
import pytest

import lgt_gb300 as lgt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _single_launches(monkeypatch):
    monkeypatch.setenv("LGT_EXPM", "krylov")
    monkeypatch.setenv("LGT_PANEL_GRID", "0")


@pytest.fixture(scope="module")
def b43():
    b, _ = lgt.build_basis(4, 3, 1, lgt.staggered_charges(4, 3))
    yield b
    b.close()


def _stream(monkeypatch, on):
    monkeypatch.setenv("LGT_BULK_STREAM", on)
    monkeypatch.setenv("LGT_BULK_DOTS", on)


@pytest.mark.parametrize("K", [1, 2, 8])
def test_streamed_exponential_bitwise(monkeypatch, b43, K):
    v0 = lgt.staggered_product_state(b43)
    out = {}
    for on in ("1", "0"):
        _stream(monkeypatch, on)
        H = lgt.build_hamiltonian(b43, g=np.linspace(0.7, 1.3, K), t=1.0, m=0.5)
        out[on] = lgt.evolve_ED(np.repeat(v0[:, None], K, axis=1), H, dt=0.05, n_steps=3,
                                tol=1e-12, precision="fp32_mixed", return_state=True)
        H.close()
    assert np.array_equal(out["1"][1], out["0"][1])
    assert np.array_equal(out["1"][2], out["0"][2])


@pytest.mark.parametrize("K", [4, 16])
def test_streamed_ground_state_bitwise(monkeypatch, b43, K):
    out = {}
    for on in ("1", "0"):
        _stream(monkeypatch, on)
        H = lgt.build_hamiltonian(b43, g=np.linspace(0.6, 1.8, K), t=1.0, m=0.5, model="pjw")
        out[on] = lgt.find_ground_state(H, tol=1e-12, precision="fp32_mixed", solver="panel",
                                        as_complex=False)
        H.close()
    assert np.array_equal(out["1"][0], out["0"][0])
    assert np.array_equal(out["1"][1], out["0"][1])


def test_double_float_and_fp64_reductions(monkeypatch, b43):
    v0 = lgt.staggered_product_state(b43)
    gs = [0.7, 1.3]
    psi, gst = {}, {}
    for flag in ("1", "0"):
        monkeypatch.setenv("LGT_DF_REDUCTIONS", flag)
        H = lgt.build_hamiltonian(b43, g=gs, t=1.0, m=0.5)
        psi[flag] = lgt.evolve_ED(np.stack([v0, v0], axis=1), H, dt=0.05, n_steps=3, tol=1e-12,
                                  precision="fp32_mixed", return_state=True)[1]
        gst[flag] = lgt.find_ground_state(H, tol=1e-12, precision="fp32_mixed", solver="panel",
                                          as_complex=False)
        H.close()
    assert np.max(np.linalg.norm(psi["1"] - psi["0"], axis=0)) <= 1e-6
    assert np.max(np.abs(gst["1"][0] - gst["0"][0]) / np.abs(gst["0"][0])) <= 1e-11


@pytest.mark.parametrize("precision,bar", [("fp64", 1e-10), ("fp32_mixed", 1e-6)])
@pytest.mark.parametrize("model", ["ref", "pjw"])
def test_krylov_exponential_against_exact(precision, bar, model):
    ch = lgt.staggered_charges(4, 2)
    b, _ = lgt.build_basis(4, 2, 1, ch)
    ob = O.build_basis(4, 2, 1, ch)
    g = np.linspace(0.6, 1.4, 5)
    H = lgt.build_hamiltonian(b, g=g, t=1.0, m=0.4, model=model)
    rng = np.random.default_rng(11)
    psi = rng.normal(size=(len(b), 5)) + 1j * rng.normal(size=(len(b), 5))
    psi /= np.linalg.norm(psi, axis=0)
    out = lgt.evolve_ED(psi, H, dt=0.07, n_steps=3, tol=1e-12, precision=precision,
                        return_state=True)[1]
    for k in range(5):
        w, z = np.linalg.eigh(O.build_hamiltonian(ob, g=g[k], t=1.0, m=0.4,
                                                  model=model).toarray())
        ref = z @ (np.exp(-1j * w * 0.21) * (z.T @ psi[:, k]))
        assert np.linalg.norm(out[:, k] - ref) <= bar
    H.close()
    b.close()
