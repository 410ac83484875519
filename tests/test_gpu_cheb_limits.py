"""Exponential steps at Krylov dimensions above the solver's limit of 63: the
expansion is held to that limit as the Krylov space is, so a long step is
split and a short one runs as at 63.

Bars: FP64, tol = 1e-12 a step: 1e-9 against exact propagation (the split
step adds at most tol per sub-step, a few dozen of them)."""
import numpy as np
import pytest

import lgt_gb300 as lgt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kd,dt,K", [(200, 0.05, 3), (200, 30.0, 128), (64, 8.0, 2),
                                     (10 ** 6, 0.05, 2), (10 ** 6, 30.0, 128)])
def test_krylovdim_above_the_limit(kd, dt, K):
    ch = lgt.staggered_charges(3, 2)
    b, _ = lgt.build_basis(3, 2, 1, ch)
    ob = O.build_basis(3, 2, 1, ch)
    g = np.linspace(0.6, 1.4, K)
    H = lgt.build_hamiltonian(b, g=g, t=1.0, m=0.3)
    rng = np.random.default_rng(K)
    psi = rng.normal(size=(len(b), K)) + 1j * rng.normal(size=(len(b), K))
    psi /= np.linalg.norm(psi, axis=0)
    _, out, _ = lgt.evolve_ED(psi, H, dt=dt, n_steps=1, krylovdim=kd, tol=1e-12,
                              return_state=True)
    for k in range(K):
        w, z = np.linalg.eigh(O.build_hamiltonian(ob, g=g[k], t=1.0, m=0.3).toarray())
        ref = z @ (np.exp(-1j * w * dt) * (z.T @ psi[:, k]))
        assert np.linalg.norm(out[:, k] - ref) <= 1e-9
    H.close()
    b.close()
