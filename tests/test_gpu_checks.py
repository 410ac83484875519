"""Convergence checks of the Lanczos tridiagonal for start vectors with little
of the ground state (small pivots at the top of T, late convergence) and for
nearly degenerate lowest states, against the FP64 oracle.

Bars: FP64 residuals of 1e-11 leave the energy within 1e-10 of its size; mixed
residuals of 3e-6 |E| over gaps above 0.1 leave (3e-6 |E|)^2 / 0.1, below 1e-8
|E| for |E| up to 100.  Start shares stay well above the residual a precision
resolves: below it no solver can tell the ground state is missing."""
import numpy as np
import pytest

import lgt_gb300 as lgt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["cta", "panel"])
@pytest.mark.parametrize("precision,share", [
    ("fp64", 1e-2), ("fp64", 1e-3), ("fp64", 1e-4), ("fp64", 1e-5), ("fp64", 1e-6),
    ("fp64", 1e-8), ("fp32_mixed", 1e-2), ("fp32_mixed", 2e-3)])
def test_small_share_of_the_ground_state(solver, precision, share):
    ob = O.build_basis(3, 2, 1, lgt.staggered_charges(3, 2))
    oh = O.build_hamiltonian(ob, g=1.1, t=1.0, m=0.4, model="pjw")
    w, v = np.linalg.eigh(oh.toarray().real)
    x = np.random.default_rng(3).standard_normal(len(w))
    x -= v[:, 0] * (v[:, 0] @ x)
    x = x / np.linalg.norm(x) + share * v[:, 0]
    b, _ = lgt.build_basis(3, 2, 1, lgt.staggered_charges(3, 2))
    H = lgt.build_hamiltonian(b, g=1.1, t=1.0, m=0.4, model="pjw")
    E, psi = lgt.find_ground_state(H, tol=1e-11, precision=precision, solver=solver, v0=x,
                                   as_complex=False)
    assert abs(float(E) - w[0]) <= (1e-10 if precision == "fp64" else 1e-8) * abs(w[0])
    H.close()
    b.close()


@pytest.mark.parametrize("solver", ["cta", "panel"])
@pytest.mark.parametrize("t", [1e-3, 1e-5])
def test_nearly_degenerate(solver, t):
    b, _ = lgt.build_basis(3, 2, 1, lgt.staggered_charges(3, 2))
    ob = O.build_basis(3, 2, 1, lgt.staggered_charges(3, 2))
    oh = O.build_hamiltonian(ob, g=1e-3, t=t, m=0.5, model="ref")
    w = np.linalg.eigvalsh(oh.toarray().real)
    H = lgt.build_hamiltonian(b, g=1e-3, t=t, m=0.5, model="ref")
    E, _ = lgt.find_ground_state(H, tol=1e-11, solver=solver, as_complex=False)
    assert abs(float(E) - w[0]) <= 1e-10 * abs(w[0])
    H.close()
    b.close()
