"""The quotient of the beta = 3/5 solve's last step (kinematic_wave_ff.cuh) against CUDA's division: within 0.51 units in the
last place of the exact quotient, the bound that its derivation gives, and so at most one from the rounded one."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "kinematic_wave_ff.cuh"
__global__ void k(const float* a, const float* b, float* q, float* d, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    q[i] = lue_gb300::refined_quotient(a[i], b[i], lue_gb300::rcp_approx(b[i]));
    d[i] = __fdiv_rn(a[i], b[i]);
}
extern "C" int run(const float* a, const float* b, float* q, float* d, int n)
{
    k<<<(n + 255) / 256, 256>>>(a, b, q, d, n);
    return (int)cudaDeviceSynchronize();
}
"""


def test_refined_quotient(tmp_path):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import _build
    source, library = tmp_path / "quotient.cu", tmp_path / "libquotient.so"
    source.write_text(SOURCE)
    r = subprocess.run([_build.nvcc(), *_build.NVCC_FLAGS, "-shared", str(source), "-o", str(library)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rng = np.random.default_rng(3)
    n = 1 << 20
    b = np.exp(rng.uniform(np.log(1e-20), np.log(1e35), n)).astype(np.float32)
    a = (b * np.exp(rng.uniform(np.log(1e-12), np.log(1e2), n)) * rng.choice([-1.0, 1.0], n)).astype(np.float32)
    a[:16] = 0.0
    x, y = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    q, d = torch.empty_like(x), torch.empty_like(x)
    torch.cuda.synchronize()
    p = ctypes.c_void_p
    assert ctypes.CDLL(str(library)).run(p(x.data_ptr()), p(y.data_ptr()), p(q.data_ptr()), p(d.data_ptr()), n) == 0
    q, d = q.cpu().numpy(), d.cpu().numpy()
    ulp = np.spacing(np.abs(d)).astype(np.float64)
    assert np.all(np.abs(q.astype(np.float64) - a.astype(np.float64) / b.astype(np.float64)) <= 0.51 * ulp)
    assert np.all(np.abs(q - d) <= ulp)
