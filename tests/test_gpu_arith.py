"""The refined reciprocal and square root of the step's kernels (castro_device.cuh, CASTRO_NR_ARITH), compiled
into a small library of their own and compared with IEEE division and square root.

Tolerance: 2^-52 relative.  Both end in one rounding (2^-53); the truncated term of the refinement is below 2^-54
for a seed error below 2^-18, and root's rounded product x * y enters with half its rounding error (2^-54)."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR

pytestmark = pytest.mark.gpu

SOURCE = """
#define CASTRO_NR_ARITH
#include "castro_device.cuh"
__global__ void k(const double* x, double* r, double* s, int n)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) { r[t] = castro::rcp(x[t]); s[t] = castro::root(x[t]); }
}
extern "C" int eval(const double* x, double* r, double* s, int n)
{
    k<<<(n + 255) / 256, 256>>>(x, r, s, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("arith")
    (d / "a.cu").write_text(SOURCE)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I", os.path.join(PKG_DIR, "csrc"), "-o", str(d / "a.so"), str(d / "a.cu")], check=True)
    L = C.CDLL(str(d / "a.so"))
    L.eval.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int]
    return L


# every leading 20 bits of the mantissa (what the seeds read), at exponents over the range of the step's values
@pytest.mark.parametrize("exponent", [-900, -301, -52, -1, 0, 1, 52, 300, 901])
def test_refined_reciprocal_and_root(lib, exponent):
    import torch

    rng = np.random.default_rng(exponent + 1000)
    lead = np.arange(1 << 20, dtype=np.uint64) << np.uint64(32)
    low = rng.integers(0, 1 << 32, 1 << 20, dtype=np.uint64)
    x = np.concatenate([lead | low, lead, lead | np.uint64(0xffffffff)]) | (np.uint64(1023 + exponent) << np.uint64(52))
    x = x.view(np.float64)
    t = torch.from_numpy(x).cuda()
    r, s = torch.empty_like(t), torch.empty_like(t)
    assert lib.eval(t.data_ptr(), r.data_ptr(), s.data_ptr(), t.numel()) == 0
    assert np.abs(r.cpu().numpy() * x - 1.0).max() <= 2.0 ** -52 + 2.0 ** -53   # the product here rounds once more
    ref = np.sqrt(x)
    assert (np.abs(s.cpu().numpy() - ref) / ref).max() <= 2.0 ** -52
