"""FP64 products whose neighbour sums run in integers (lgt_intsum.cuh), and
panels of any width and alignment through the fixed-shape kernel, against the
oracle's CSR matrix.

Bar, per entry: the integer sum drops at most 2^-57 of the largest neighbour
per term (31 terms at most: 2^-52) and the four coupling operations round at
2^-53 of terms no larger than B = |offdiag H| |x| + (g^2/2 e^2 + |m stag|) |x|
(the two diagonal parts can cancel, and plain FP64 rounds them differently
from the oracle's site-by-site sum): 16 * 2^-53 B covers both and the oracle's
own summation."""
import numpy as np
import pytest

import lgt_gb300 as lgt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _inputs(rng, N, C, kind):
    x = rng.standard_normal((N, C))
    if kind == "wide":
        x *= 10.0 ** rng.uniform(-18, 18, (N, C))
        x[rng.random((N, C)) < 0.2] = 0.0
    elif kind == "tiny":
        x *= 1e-306
    elif kind == "huge":
        x *= 1e300
    elif kind == "sparse":
        x[rng.random((N, C)) < 0.999] = 0.0
    return x


def _size(ob, A, g, m):
    """|offdiag A| + diag(g^2/2 e^2 + |m stag|), the matrix of the bar."""
    import scipy.sparse as sp
    nx, ny = ob.nx, ob.ny
    sign = np.array([[(-1) ** (ix + iy) for iy in range(ny)] for ix in range(nx)])
    e2 = (ob.eR.astype(int) ** 2).sum((1, 2)) + (ob.eU.astype(int) ** 2).sum((1, 2))
    stag = (ob.nf * sign).sum((1, 2))
    return abs(A - sp.diags(A.diagonal())) + sp.diags(g * g / 2 * e2 + m * np.abs(stag))


@pytest.mark.parametrize("nx,ny", [(4, 3), (3, 4)])
@pytest.mark.parametrize("model", ["ref", "pjw"])
@pytest.mark.parametrize("K", [1, 2, 3, 5, 8])
def test_products(nx, ny, model, K):
    ch = lgt.staggered_charges(nx, ny)
    b, _ = lgt.build_basis(nx, ny, 1, ch)
    ob = O.build_basis(nx, ny, 1, ch)
    g = np.linspace(0.5, 1.5, K)
    H = lgt.build_hamiltonian(b, g=g, t=0.9, m=0.4, model=model)
    rng = np.random.default_rng(K)
    mats = [O.build_hamiltonian(ob, g=v, t=0.9, m=0.4, model=model) for v in g[[0, -1]]]
    size = [_size(ob, A, v, 0.4) for A, v in zip(mats, g[[0, -1]])]
    for kind in ("normal", "wide", "tiny", "huge", "sparse"):
        x = _inputs(rng, len(b), K, kind)
        y = np.asarray(H.matvec(x)).reshape(len(b), K)
        for k, A, B in zip((0, K - 1), mats, size):
            bar = 16 * 2.0 ** -53 * (B @ np.abs(x[:, k])) + 1e-318
            assert np.all(np.abs(y[:, k] - A @ x[:, k]) <= bar), kind
    x = rng.standard_normal((len(b), K)) + 1j * rng.standard_normal((len(b), K))
    y = H.matvec(x)
    A = mats[1]
    bar = 16 * 2.0 ** -53 * (size[1] @ (np.abs(x[:, -1].real) + np.abs(x[:, -1].imag)))
    assert np.all(np.abs(y[:, -1] - A @ x[:, -1]) <= bar)
    H.close()
    b.close()


def test_non_finite_entries_stay_where_they_belong():
    ch = lgt.staggered_charges(4, 3)
    b, _ = lgt.build_basis(4, 3, 1, ch)
    ob = O.build_basis(4, 3, 1, ch)
    H = lgt.build_hamiltonian(b, g=1.1, t=0.9, m=0.4)
    A = O.build_hamiltonian(ob, g=1.1, t=0.9, m=0.4)
    x = np.random.default_rng(0).standard_normal(len(b))
    x[123], x[4567], x[50000] = np.inf, -np.inf, np.nan
    y, ref = H.matvec(x), A @ x
    np.testing.assert_array_equal(np.isnan(y), np.isnan(ref))
    np.testing.assert_array_equal(np.isposinf(y), np.isposinf(ref))
    np.testing.assert_array_equal(np.isneginf(y), np.isneginf(ref))
    H.close()
    b.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_unaligned_device_panels(precision):
    import torch
    b, _ = lgt.build_basis(4, 3, 1, lgt.staggered_charges(4, 3))
    H = lgt.build_hamiltonian(b, g=np.linspace(0.5, 1.5, 4), t=1.0, m=0.4)
    dt = torch.float64 if precision == "fp64" else torch.float32
    N, C = len(b), 8
    buf = torch.randn(N * C + 1, dtype=dt, device="cuda")
    out = torch.zeros(N * C + 1, dtype=dt, device="cuda")
    x, y = buf[1:].clone(), torch.zeros(N * C, dtype=dt, device="cuda")
    torch.cuda.synchronize()
    H.matvec_device(buf[1:].data_ptr(), out[1:].data_ptr(), ncomp=2, precision=precision)
    H.matvec_device(x.data_ptr(), y.data_ptr(), ncomp=2, precision=precision)
    tol = 1e-13 if precision == "fp64" else 1e-4
    assert float((out[1:] - y).abs().max()) <= tol
    H.close()
    b.close()
