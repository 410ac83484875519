"""The two block roles of the observables kernel (k_observe_roles) against the
one-role FP64 sums (LGT_DF_REDUCTIONS=0) and against features formed on the
host, for point counts that leave threads over, real and complex states, both
precisions and panels that start off a 16-byte boundary.

Bar: double-float sums keep 2^-47 relative per term and all features are
sums of at most one sign of |psi|^2 (or bounded by it): 1e-12 of the norm."""
import numpy as np
import pytest

import lgt_gb300 as lgt
from lgt_gb300 import _capi as C

pytestmark = pytest.mark.gpu


def _observe(H, ptr, ncomp, prec, K, ns, npl):
    nf, e2, pl = np.zeros((K, ns)), np.zeros((K, ns)), np.zeros((K, max(npl, 1)))
    summ = (C.Obs * K)()
    C.check(C.load().lgt_observe(H.handle, ptr, ncomp, prec, C.LGT_DEVICE_PTRS, 0.0,
                                 nf.ctypes.data, e2.ctypes.data, pl.ctypes.data, summ))
    norm = np.frombuffer(summ, np.float64).reshape(K, 8)[:, 7].copy()
    return nf, e2, pl[:, :npl], norm


@pytest.mark.parametrize("nx,ny,sector", [(4, 2, "stag"), (2, 2, "stag"), (3, 3, "stag"),
                                          (3, 4, "string"), (2, 6, "stag"), (4, 3, "stag")])
@pytest.mark.parametrize("K", [1, 3, 8, 70])
def test_roles(monkeypatch, nx, ny, sector, K):
    import torch
    ch = lgt.string_charges(nx, ny) if sector == "string" else lgt.staggered_charges(nx, ny)
    b, _ = lgt.build_basis(nx, ny, 1, ch)
    H = lgt.build_hamiltonian(b, g=np.ones(K), t=1.0, m=0.5, model="pjw")
    N, ns, npl = len(b), nx * ny, (nx - 1) * (ny - 1)
    n_f, e_R, e_U = (a.astype(float) for a in b.states())
    eg = np.zeros((N, nx, ny))
    eg[:, :nx - 1, :] += e_R ** 2
    eg[:, :, :ny - 1] += e_U ** 2
    gen = torch.Generator(device="cuda").manual_seed(K)
    for ncomp in (1, 2):
        for dt, prec in ((torch.float64, C.LGT_FP64), (torch.float32, C.LGT_FP32)):
            n = N * K * ncomp
            buf = torch.randn(n + 1, generator=gen, dtype=dt, device="cuda") / N ** 0.5
            for off in (0, 1):
                v = buf[off:off + n]
                torch.cuda.synchronize()
                monkeypatch.delenv("LGT_DF_REDUCTIONS", raising=False)
                got = _observe(H, v.data_ptr(), ncomp, prec, K, ns, npl)
                monkeypatch.setenv("LGT_DF_REDUCTIONS", "0")
                ref = _observe(H, v.data_ptr(), ncomp, prec, K, ns, npl)
                x = v.double().cpu().numpy().reshape(N, K, ncomp)
                p = (x ** 2).sum(2)
                bar = 1e-12 * p.sum(0).max()
                for a, r in zip(got, ref):
                    assert np.max(np.abs(a - r), initial=0.0) <= bar
                nf = np.einsum("nk,nxy->kyx", p, n_f).reshape(K, ns)
                e2 = np.einsum("nk,nxy->kyx", p, eg).reshape(K, ns)
                assert np.max(np.abs(got[0] - nf)) <= bar and np.max(np.abs(got[1] - e2)) <= 8 * bar
                assert np.max(np.abs(got[3] - p.sum(0))) <= bar
    H.close()
    b.close()
