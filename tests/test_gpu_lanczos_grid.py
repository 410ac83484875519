"""The one-launch Lanczos cycles of the panel solver (lanczos_grid.cu) against
the FP64 oracle and the multi-launch steps (LGT_PANEL_GRID=0): panel widths
that leave threads over, fill them and exceed a warp, sectors with a partial
last block, restarts in which only some columns go on, and spaces that are
exhausted.

Bars: energies as for every solver, 1e-10 relative.  States: FP64 residuals
below 1e-10 over gaps above 0.1 give 1e-8; FP32-mixed residuals 2e-5 give
1e-3 in the worst case, both paths the same side of it."""
import numpy as np
import pytest

import lgt_gb300 as lgt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _energies(nx, ny, g, m, model):
    ob = O.build_basis(nx, ny, 1, lgt.staggered_charges(nx, ny))
    return np.array([O.ground_state(O.build_hamiltonian(ob, g=a, t=1.0, m=b, model=model))[0]
                     for a, b in zip(g, m)])


@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
@pytest.mark.parametrize("nx,ny,K,model,kd", [
    (3, 2, 1, "ref", 50), (4, 2, 1, "pjw", 50), (4, 2, 3, "ref", 14), (4, 2, 25, "pjw", 20),
    (4, 2, 70, "ref", 50), (3, 3, 16, "pjw", 16), (3, 3, 33, "ref", 50), (2, 2, 5, "ref", 50),
])
def test_against_oracle_and_multi_launch(monkeypatch, precision, nx, ny, K, model, kd):
    g, m = np.geomspace(0.5, 2.5, K), np.linspace(0.2, 0.9, K)
    b, _ = lgt.build_basis(nx, ny, 1, lgt.staggered_charges(nx, ny))
    got = {}
    for env in ("1", "0"):
        monkeypatch.setenv("LGT_PANEL_GRID", env)
        H = lgt.build_hamiltonian(b, g=g, t=1.0, m=m, model=model)
        E, psi, info = lgt.find_ground_state(H, precision=precision, solver="panel",
                                             krylovdim=kd, seed=4, as_complex=False,
                                             return_info=True)
        got[env] = (np.atleast_1d(E), psi.reshape(len(b), K), info)
        H.close()
    ref = _energies(nx, ny, g, m, model)
    for env in got:
        assert np.max(np.abs(got[env][0] - ref) / np.abs(ref)) <= 1e-10
        assert got[env][2]["converged"] == K
    bar = 1e-8 if precision == "fp64" else 1e-3
    assert np.max(np.linalg.norm(got["1"][1] - got["0"][1], axis=0)) <= bar
    b.close()


def test_4x3_wide_odd_panel_and_refinement():
    g = np.geomspace(0.4, 2.0, 17)
    b, _ = lgt.build_basis(4, 3, 1, lgt.staggered_charges(4, 3))
    H = lgt.build_hamiltonian(b, g=g, t=1.0, m=0.3, model="pjw")
    E64, p64 = lgt.find_ground_state(H, solver="panel", as_complex=False)
    E32, p32 = lgt.find_ground_state(H, solver="panel", precision="fp32_mixed",
                                     refine_steps=12, as_complex=False)
    assert np.max(np.abs(E64 - E32) / np.abs(E64)) <= 1e-12
    assert np.max(np.linalg.norm(p64 - p32, axis=0)) <= 1e-8
    H.close()
    b.close()


def test_not_converged_is_reported():
    b, _ = lgt.build_basis(3, 3, 1, lgt.staggered_charges(3, 3))
    H = lgt.build_hamiltonian(b, g=[0.5, 1.0], t=1.0, m=0.3)
    with pytest.raises(lgt.NotConverged):
        lgt.find_ground_state(H, solver="panel", krylovdim=5, maxiter=1, tol=1e-14)
    E, _ = lgt.find_ground_state(H, solver="panel")
    assert E.shape == (2,)
    H.close()
    b.close()
