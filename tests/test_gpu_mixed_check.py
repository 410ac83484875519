"""The FP32 convergence check of the mixed per-point solver against FP64:
Lanczos tridiagonals of 300 levels whose start vectors hold from a third down
to 2e-5 of the lowest one.

Bars: theta to 2e-6 of the spread (the bracket's width and FP32 rounding).  The
residual |beta_n z_n| comes from a vector after one inverse iteration: its
shift lies at most 1e-6 of the spread below theta and the next level 1/38 of it
above, so what is left of the other levels is 4e-5 of itself, and n products
add n 6e-8: 1e-3 has room for both."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = str(tmp_path_factory.mktemp("tri") / "tri_check.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-shared", "-Xcompiler", "-fPIC", os.path.join(HERE, "tri_check.cu"),
                    "-o", so], check=True)
    f = ctypes.CDLL(so).tri_check
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    return f


def _lanczos(share, n, rng):
    """(a, b) of n steps, b[n-1] the last residual norm, in long double."""
    levels = -7 + 30 * rng.uniform(size=300) * rng.uniform(size=300)
    levels[0] = -8
    v = rng.normal(size=300)
    v[0] = 0
    v /= np.linalg.norm(v)
    v[0] = share
    levels, v = levels.astype(np.longdouble), (v / np.linalg.norm(v)).astype(np.longdouble)
    V, a, b = [], np.zeros(n), np.zeros(n)
    for j in range(n):
        V.append(v)
        w = levels * v
        al = np.longdouble(0)
        for _ in range(2):
            for c in range(j, -1, -1):
                d = (V[c] * w).sum()
                w = w - d * V[c]
                if c == j:
                    al += d
        be = np.sqrt((w * w).sum())
        a[j], b[j] = al, be
        v = w / be
    return a, b


def _tail(a, b):
    """theta and |z_{n-1}| by the ratios of the bottom-up pivots in FP64."""
    n = len(a)
    th = np.linalg.eigvalsh(np.diag(a) + np.diag(b[:-1], 1) + np.diag(b[:-1], -1))[0]
    u = np.zeros(n)
    u[n - 1] = a[n - 1] - th
    for i in range(n - 2, 0, -1):
        u[i] = a[i] - th - b[i] ** 2 / u[i + 1]
    z = np.ones(n)
    for i in range(1, n):
        z[i] = -z[i - 1] * b[i - 1] / u[i]
    return th, abs(z[-1]) / np.linalg.norm(z)


@pytest.mark.parametrize("n", [10, 20, 33, 50, 63])
def test_residual_of_the_iterated_vector(check, n):
    import torch
    rng = np.random.default_rng(n)
    mats = [_lanczos(s, n, rng) for s in (0.3, 0.04, 1e-2, 1e-3, 1e-4, 4e-5, 2e-5) for _ in "ab"]
    a = torch.tensor(np.stack([m[0] for m in mats]), device="cuda")
    b = torch.tensor(np.stack([m[1] for m in mats]), device="cuda")
    out = torch.zeros((len(mats), 3), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert check(a.data_ptr(), b.data_ptr(), n, len(mats), out.data_ptr()) == 0
    got = out.cpu().numpy()
    for (am, bm), (th, r, zn) in zip(mats, got):
        ref, tail = _tail(am, bm)
        spread = am.max() - am.min() + 2 * bm.max()
        assert abs(th - ref) <= 2e-6 * spread
        assert abs(r - bm[-1] * tail) <= 1e-3 * bm[-1] * tail
        assert r == abs(bm[-1] * zn)
