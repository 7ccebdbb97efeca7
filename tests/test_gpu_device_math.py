"""The device's own elementary functions (eu3d_device.cuh) against CUDA's exp, 1/x
and x/sqrt(x d), over the ranges that they state. The probe is compiled here,
against the library's headers."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "eu3d-gpu_b200", "csrc")
SOURCE = """
#include "eu3d_device.cuh"
using namespace eu3d;
__global__ void k(const double *x, const double *d, double *out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    out[i] = exp_fast(x[i]);
    out[n + i] = exp_paired(x[i]);
    out[2 * n + i] = exp(x[i]);
    out[3 * n + i] = rcp_nr(d[i]);
    out[4 * n + i] = 1.0 / d[i];
    out[5 * n + i] = sound_speed(d[i], d[n - 1 - i]);
    out[6 * n + i] = sqrt(d[i] / d[n - 1 - i]);
}
extern "C" int run(const double *x, const double *d, double *out, int n)
{
    k<<<(n + 255) / 256, 256>>>(x, d, out, n);
    return cudaDeviceSynchronize();
}
"""


def test_elementary_functions(gpu, tmp_path):
    """exp_fast and exp_paired within one unit in the last place of CUDA's exp
    (itself within one of the exact value, so two apart at most) on all of
    [-708, 708], NaN for NaN; rcp_nr within one unit of the quotient rounded to
    nearest; sound_speed within 4 (the argument's product, its root and the last
    product each round; the quotient and root it is compared with do too)."""
    import torch
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    (tmp_path / "probe.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-shared", "-Xcompiler", "-fPIC",
                    "-I", CSRC, str(tmp_path / "probe.cu"), "-o", str(tmp_path / "probe.so")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "probe.so"))
    rng = np.random.default_rng(0)
    n = 1 << 20
    x = rng.uniform(-708.0, 708.0, n)
    x[: n // 4] = rng.uniform(-1.0, 1.0, n // 4)
    x[:8] = [-708.0, 708.0, 0.0, -0.0, np.log(2) / 2, -np.log(2) / 2, 1e-300, np.nan]
    d = 2.0 ** rng.uniform(-500, 500, n) * rng.choice([1.0], n)
    xs, ds, out = (torch.tensor(v, device="cuda") for v in (x, d, np.zeros(7 * n)))
    torch.cuda.synchronize()
    assert lib.run(*(ctypes.c_void_p(t.data_ptr()) for t in (xs, ds, out)), n) == 0
    fast, paired, exact, rcp, quotient, speed, root = out.cpu().numpy().reshape(7, n)

    def ulps(a, b):
        return np.abs(a - b) / np.spacing(np.abs(b))

    assert np.isnan(fast[7]) and np.isnan(paired[7])
    for got in (fast, paired):
        keep = np.isfinite(x)
        assert ulps(got[keep], exact[keep]).max() <= 2
        assert ulps(got[keep], np.exp(x[keep])).max() <= 1  # the host's, nearly always rounded to nearest
    assert ulps(rcp, quotient).max() <= 1
    assert ulps(speed, root).max() <= 4
