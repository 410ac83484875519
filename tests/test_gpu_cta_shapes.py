"""The per-point solver's launch shape is timed for what it depends on: another
Krylov dimension or model of the same batch size is timed again (both decide
what fits the shared memory), the same one is not."""
import numpy as np
import pytest

import lgt_gb300 as lgt
from lgt_gb300 import _capi as C

pytestmark = pytest.mark.gpu


def test_shape_is_timed_per_model_and_krylovdim():
    b, _ = lgt.build_basis(3, 3, 1, lgt.staggered_charges(3, 3))
    g = np.geomspace(0.5, 2.0, 13)  # a number of points no other test uses here

    def launches(model, kd):
        H = lgt.build_hamiltonian(b, g=g, t=1.0, m=0.4, model=model)
        lgt.find_ground_state(H, solver="cta", krylovdim=40, as_complex=False)
        n = []
        for _ in range(2):
            n0 = C.launch_count()
            lgt.find_ground_state(H, solver="cta", krylovdim=kd, as_complex=False)
            n.append(C.launch_count() - n0)
        H.close()
        return n

    for model, kd in (("ref", 24), ("pjw", 30), ("ref", 31)):
        first, second = launches(model, kd)
        assert first > second
    first, second = launches("ref", 24)
    assert first == second
    b.close()
