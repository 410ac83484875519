"""How the panel solver chooses between its one-launch cycle and the single
launches: a cycle whose barrier wait runs out is done again by single launches,
and panels that the cycle cannot take cost no table.

Bars as for every solver: energies 1e-10 relative, states 1e-8 (FP64) and 1e-3
(FP32-mixed, residual 2e-5)."""
import numpy as np
import pytest

import lgt_gb300 as lgt
from lgt_gb300 import _capi as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
@pytest.mark.parametrize("nx,ny,K,kd", [(3, 3, 4, 50), (3, 3, 3, 14), (4, 3, 5, 50)])
def test_expired_wait_falls_back(monkeypatch, precision, nx, ny, K, kd):
    b, _ = lgt.build_basis(nx, ny, 1, lgt.staggered_charges(nx, ny))
    g = np.geomspace(0.5, 2.0, K)

    def solve(**env):
        for name in ("LGT_PANEL_GRID", "LGT_PANEL_GRID_SPIN"):
            monkeypatch.delenv(name, raising=False)
        for name, v in env.items():
            monkeypatch.setenv(name, v)
        H = lgt.build_hamiltonian(b, g=g, t=1.0, m=0.4)
        n0 = C.launch_count()
        E, psi = lgt.find_ground_state(H, precision=precision, solver="panel", krylovdim=kd,
                                       seed=7, as_complex=False)
        n1 = C.launch_count()
        y = H.matvec(psi)  # the basis' error word is clear
        H.close()
        return E, psi, n1 - n0, y

    solve(LGT_PANEL_GRID="0")  # (tunes the single launches once)
    single = solve(LGT_PANEL_GRID="0")
    cycle = solve()
    expired = solve(LGT_PANEL_GRID_SPIN="0")
    assert cycle[2] < single[2] <= expired[2]
    bar = 1e-8 if precision == "fp64" else 1e-3
    for got in (cycle, expired):
        assert np.max(np.abs(got[0] - single[0]) / np.abs(single[0])) <= 1e-10
        assert np.max(np.linalg.norm(got[1] - single[1], axis=0)) <= bar
        assert np.all(np.isfinite(got[3]))
    b.close()


def test_no_table_for_panels_the_cycle_cannot_take(monkeypatch):
    """4x3, K = 64 in FP64: a block's rows do not fit, and with the tuner off
    the single launches need no table."""
    monkeypatch.setenv("LGT_AUTOTUNE", "0")
    b, _ = lgt.build_basis(4, 3, 1, lgt.staggered_charges(4, 3))
    n = {}
    for env in ("0", "1"):
        monkeypatch.setenv("LGT_PANEL_GRID", env)
        H = lgt.build_hamiltonian(b, g=np.geomspace(0.5, 2.0, 64), t=1.0, m=0.4)
        n0 = C.launch_count()
        with pytest.raises(lgt.NotConverged):
            lgt.find_ground_state(H, solver="panel", krylovdim=10, maxiter=0, as_complex=False)
        n[env] = C.launch_count() - n0
        H.close()
    assert n["1"] == n["0"]
    b.close()
