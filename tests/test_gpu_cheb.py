"""exp(-iHt) steps by Chebyshev expansion (cheb.cu) against exact propagation
and against the Krylov path, at panel widths that take every slice of the
table product, and the calls that must stay with the Krylov path.

Bars: FP64 -- the truncation is below 2e-16 a step and the recurrence of n
products adds about n^2 rounding errors of 1.1e-16 in norm: 1e-12 covers
n <= 30 and 4 steps.  FP32-mixed -- panels rounded to 2^-24 = 6e-8, weighted
by 2 |J_n| (sum below 3) and n: 2e-6.
"""
import numpy as np
import pytest

import lgt_gb300 as lgt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _start(N, K, seed):
    rng = np.random.default_rng(seed)
    p = rng.normal(size=(N, K)) + 1j * rng.normal(size=(N, K))
    return p / np.linalg.norm(p, axis=0)


def _exact(ob, psi, g, m, model, dt, steps):
    out = []
    for k in range(psi.shape[1]):
        A = O.build_hamiltonian(ob, g=g[k], t=1.0, m=m, model=model).toarray()
        w, z = np.linalg.eigh(A)
        v = z @ (np.exp(-1j * w * dt * steps) * (z.T @ psi[:, k]))
        out.append(v / np.linalg.norm(v))
    return np.stack(out, axis=1)


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("model", ["ref", "pjw"])
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_steps_against_exact(K, model, precision):
    nx, ny = 4, 2
    ch = lgt.staggered_charges(nx, ny)
    b, _ = lgt.build_basis(nx, ny, 1, ch)
    ob = O.build_basis(nx, ny, 1, ch)
    g = np.linspace(0.6, 1.4, K)
    H = lgt.build_hamiltonian(b, g=g, t=1.0, m=0.4, model=model)
    psi = _start(len(b), K, K)
    arg = psi[:, 0] if K == 1 else psi
    data, out, drift = lgt.evolve_ED(arg, H, dt=0.07, n_steps=4, precision=precision,
                                     return_state=True)
    bar = 1e-12 if precision == "fp64" else 2e-6
    ref = _exact(ob, psi, g, 0.4, model, 0.07, 4)
    assert np.max(np.linalg.norm(out.reshape(len(b), K) - ref, axis=0)) <= bar
    assert np.max(drift) <= bar
    assert len(data) == 5
    H.close()
    b.close()


def test_agrees_with_krylov_path(monkeypatch):
    b, _ = lgt.build_basis(3, 3, 1, lgt.staggered_charges(3, 3))
    H = lgt.build_hamiltonian(b, g=[0.7, 1.2], t=1.0, m=0.5, model="pjw")
    psi = _start(len(b), 2, 3)
    psi[:, 1] *= 3.0  # the first step's norm counts the start's
    got = lgt.evolve_ED(psi, H, dt=0.05, n_steps=3, tol=1e-13, return_state=True)
    monkeypatch.setenv("LGT_EXPM", "krylov")
    ref = lgt.evolve_ED(psi, H, dt=0.05, n_steps=3, tol=1e-13, return_state=True)
    assert np.max(np.abs(got[1] - ref[1])) <= 1e-12
    assert np.max(np.abs(got[2] - ref[2])) <= 1e-11 and abs(got[2][1] - 2.0) <= 1e-11
    for a, r in zip(got[0], ref[0]):
        for k in range(2):
            assert abs(a[k]["E2_mean"] - r[k]["E2_mean"]) <= 1e-12
    H.close()
    b.close()


def test_short_krylovdim_and_long_steps():
    """A step that needs more products than krylovdim is split by the Krylov
    path; both agree with exact propagation."""
    ch = lgt.staggered_charges(3, 2)
    b, _ = lgt.build_basis(3, 2, 1, ch)
    ob = O.build_basis(3, 2, 1, ch)
    H = lgt.build_hamiltonian(b, g=1.1, t=1.0, m=0.3)
    psi = _start(len(b), 1, 9)
    for dt, kd in ((0.05, 6), (2.0, 30)):
        _, out, _ = lgt.evolve_ED(psi[:, 0], H, dt=dt, n_steps=2, krylovdim=kd, tol=1e-12,
                                  return_state=True)
        ref = _exact(ob, psi, [1.1], 0.3, "ref", dt, 2)[:, 0]
        assert np.linalg.norm(out - ref) <= 1e-9
    H.close()
    b.close()


def test_zero_and_non_finite_states():
    b, _ = lgt.build_basis(3, 2, 1, lgt.staggered_charges(3, 2))
    H = lgt.build_hamiltonian(b, g=[0.9, 1.1], t=1.0, m=0.3)
    psi = _start(len(b), 2, 4)
    psi[:, 1] = 0.0
    _, out, drift = lgt.evolve_ED(psi, H, dt=0.05, n_steps=2, return_state=True)
    assert np.all(out[:, 1] == 0.0) and drift[1] == 1.0 and drift[0] <= 1e-12
    psi[3, 1] = np.nan
    with pytest.raises(lgt.NotConverged):
        lgt.evolve_ED(psi, H, dt=0.05, n_steps=2)
    # dt <= 0 leaves the state as it is (renormalised)
    psi[:, 1] = psi[:, 0]
    _, out, _ = lgt.evolve_ED(psi, H, dt=-0.05, n_steps=1, return_state=True)
    assert np.max(np.abs(out - psi)) <= 1e-14
    H.close()
    b.close()
