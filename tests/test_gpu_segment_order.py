"""The order of the fermion-mask segments (order.cu): levels of the masks'
dipole sum(x + y), alternately forwards and backwards, and products that visit
their tiles in it.  The order changes no sum, so products are compared bit for
bit."""
import numpy as np
import pytest

import lgt_gb300 as lgt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 2), (2, 4), (4, 3)])
def test_levels(nx, ny):
    b, _ = lgt.build_basis(nx, ny, 1, lgt.staggered_charges(nx, ny))
    H = lgt.build_hamiltonian(b, g=1.0, t=1.0, m=0.5)
    perm = np.asarray(H.row_order())
    assert np.array_equal(np.sort(perm), np.arange(len(b)))
    nf = b.states()[0][perm].astype(np.int64)  # [n, nx, ny]
    Y = np.einsum("nxy,y->n", nf, np.arange(ny))
    P = Y + np.einsum("nxy,x->n", nf, np.arange(nx))
    assert np.all(np.diff(P) >= 0)
    for p in np.unique(P):
        d = np.diff(Y[P == p])
        assert np.all(d <= 0) if p % 2 else np.all(d >= 0)
    H.close()
    b.close()


@pytest.mark.parametrize("model,prec,K,ncomp", [
    ("ref", "fp32", 8, 2), ("pjw", "fp32", 4, 1), ("ref", "fp64", 2, 1)])
def test_tile_order_keeps_the_product(monkeypatch, model, prec, K, ncomp):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("LGT_HPSI_VARIANT", "5")
    b, _ = lgt.build_basis(4, 4, 1, lgt.staggered_charges(4, 4))
    dt = torch.float64 if prec == "fp64" else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn((len(b), K * ncomp), dtype=dt, device="cuda", generator=gen)
    y = {}
    for order in ("mask", "0"):
        monkeypatch.setenv("LGT_TABLE_ORDER", order)
        H = lgt.build_hamiltonian(b, g=np.linspace(0.5, 1.5, K), t=1.0, m=0.5, model=model)
        y[order] = torch.full_like(x, float("nan"))
        torch.cuda.synchronize()
        H.matvec_device(x.data_ptr(), y[order].data_ptr(), ncomp, prec)
        torch.cuda.synchronize()
        H.close()
    assert torch.equal(y["mask"], y["0"])
    b.close()
