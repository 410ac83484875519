"""FP32-mixed exponential steps: the Chebyshev expansion is no further from
FP64 than the Krylov steps it stands in for (LGT_EXPM=krylov), for product
states and general ones, short and long times, both models.

The two differ by independent roundings, so errors are compared as the root
mean square over points and starts, with a tenth for the spread of that mean."""
import numpy as np
import pytest

import lgt_gb300 as lgt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,model,dt,steps,K", [
    (3, 3, "ref", 0.03, 1, 4), (3, 3, "pjw", 0.01, 1, 4), (3, 3, "ref", 0.1, 4, 5),
    (4, 3, "ref", 0.05, 2, 3), (4, 3, "pjw", 0.05, 2, 2), (3, 4, "pjw", 0.01, 6, 5),
    (4, 4, "ref", 0.05, 2, 8),
])
@pytest.mark.parametrize("start", ["product", "random"])
def test_no_further_than_krylov(monkeypatch, nx, ny, model, dt, steps, K, start):
    if nx * ny == 16 and start == "random":
        pytest.skip("the 4x4 quench starts from a product state")
    b, _ = lgt.build_basis(nx, ny, 1, lgt.staggered_charges(nx, ny))
    v = lgt.staggered_product_state(b)
    e2 = {"default": 0.0, "krylov": 0.0}
    for seed in (1, 2, 3):
        rng = np.random.default_rng(seed)
        H = lgt.build_hamiltonian(b, g=rng.uniform(0.5, 1.5, K), t=1.0, m=0.5, model=model)
        if start == "product":
            psi = np.repeat(v[:, None], K, axis=1).astype(complex)
        else:
            psi = rng.normal(size=(len(b), K)) + 1j * rng.normal(size=(len(b), K))
            psi /= np.linalg.norm(psi, axis=0)
        monkeypatch.delenv("LGT_EXPM", raising=False)
        ref = lgt.evolve_ED(psi, H, dt=dt, n_steps=steps, tol=1e-13, return_state=True)[1]
        for path in e2:
            if path == "krylov":
                monkeypatch.setenv("LGT_EXPM", "krylov")
            out = lgt.evolve_ED(psi, H, dt=dt, n_steps=steps, precision="fp32_mixed",
                                return_state=True)[1]
            e2[path] += np.sum(np.abs(out - ref) ** 2)
        H.close()
    b.close()
    assert e2["default"] ** 0.5 <= 1.1 * e2["krylov"] ** 0.5
