"""FP64 products of the smallest numbers: with no diagonal (g = m = 0, t = 1)
a row of H psi is a sum of neighbours, so integers times 2^-1074 stay exact, in
every kernel, alone in a row or beside zeros, and where rows of ordinary
numbers lie next to them."""
import numpy as np
import pytest

import lgt_gb300 as lgt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["", "2", "3", "5", "6"])
@pytest.mark.parametrize("nx,ny,K", [(4, 3, 1), (4, 3, 2), (3, 4, 4), (3, 3, 3)])
def test_smallest_numbers(monkeypatch, nx, ny, K, variant):
    if variant:
        monkeypatch.setenv("LGT_HPSI_VARIANT", variant)
    ch = lgt.staggered_charges(nx, ny)
    b, _ = lgt.build_basis(nx, ny, 1, ch)
    A = O.build_hamiltonian(O.build_basis(nx, ny, 1, ch), g=0.0, t=1.0, m=0.0).tocsr()
    H = lgt.build_hamiltonian(b, g=np.zeros(K), t=1.0, m=0.0)
    rng = np.random.default_rng(K)
    m = rng.integers(-2 ** 32, 2 ** 32, (len(b), K))  # high words zero, or not
    m[rng.random(m.shape) < 0.3] = 0
    for scale in (1, 2 ** 20):
        q = m // 2 ** 20 * scale
        x = np.ldexp(q.astype(float), -1074)
        y = H.matvec(x[:, 0] if K == 1 else x).reshape(len(b), K)
        np.testing.assert_array_equal(y, np.ldexp((A @ q.astype(float)), -1074))
    # one ordinary column beside tiny ones
    if K > 1:
        x = np.ldexp((m // 2 ** 20).astype(float), -1074)
        x[:, 1] = rng.integers(-9, 10, len(b))
        y = H.matvec(x)
        np.testing.assert_array_equal(y[:, 1], A @ x[:, 1])
        np.testing.assert_array_equal(y[:, 0], np.ldexp(A @ (m[:, 0] // 2 ** 20).astype(float), -1074))
    H.close()
    b.close()
