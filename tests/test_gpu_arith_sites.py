"""What the refined reciprocal and square root are used for (castro_device.cuh): the seeds their error bound rests on,
quot, root_floor, and the two transverse corrections with a corrected density below zero, where they fall back to the
uncorrected state after the reciprocal of the negative density has been formed.

Bounds, with u = 2^-53.  Premise, checked on every leading 20 bits of the argument: the seeds leave e = 1 - x y (rcp)
and e = 1 - x y y (root) below 2^-18 in magnitude.
  rcp   truncated e^3 (u/2) and the last rounding (u): 1.5 u
  quot  rcp and the product's rounding: 2.5 u
  root  truncated 5/16 e^3 (under u/4), half the rounding of x y (u/2) and the last rounding (u): under 2 u
  root_floor  root of max(lo * lo, |x|); half the rounding of lo * lo (u/2) on top: 2.5 u
each plus terms of order u 2^-18.  The corrections are compared with the same source compiled with IEEE / : a product
with the reciprocal moves by 1.5 u + u (the two reciprocals) + 2 u (the two products), a quotient by less, and the
internal energy (total less kinetic) by 4.5 u of the kinetic energy (5.5 u with the rounding of the kinetic energy formed
here) and two roundings of the difference."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
ROOM = 1.0 + 2.0 ** -10   # the terms of order u 2^-18, and the long double reference's own rounding

SOURCE = """
#include "castro_device.cuh"
using namespace castro;
__global__ void k_scalar(const double* a, const double* b, double* er, double* es, double* q, double* f, int n)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    double y, z;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b[t]));
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(z) : "d"(b[t]));
    er[t] = fma(-b[t], y, 1.0);
    es[t] = fma(-(b[t] * z), z, 1.0);
    q[t] = quot(a[t], b[t], rcp(b[t]));
    f[t] = root_floor(b[t], a[t]);
}
template <int NS>
__global__ void k_trans(const double* lq, const double* f, const double* g, double* out, int* reset, int n)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    constexpr int NQS = Dims<NS>::NQS, N = TF<NS>::N;
    double o[NQS];
    reset[t] = trans1_state<NS>(lq + t * NQS, f + t * 2 * N, f + t * 2 * N + N, 1.6, 0.3, o);
    for (int c = 0; c < NQS; ++c) out[t * 2 * NQS + c] = o[c];
    reset[n + t] = trans2_state<NS>(lq + t * NQS, f + t * 2 * N, f + t * 2 * N + N, g + t * 2 * N, g + t * 2 * N + N, 1.6,
                                    0.2, 0.2, o);
    for (int c = 0; c < NQS; ++c) out[t * 2 * NQS + NQS + c] = o[c];
}
extern "C" int scalar(const double* a, const double* b, double* er, double* es, double* q, double* f, int n)
{
    k_scalar<<<(n + 255) / 256, 256>>>(a, b, er, es, q, f, n);
    return (int)cudaDeviceSynchronize();
}
extern "C" int trans(int ns, const double* lq, const double* f, const double* g, double* out, int* reset, int n)
{
    if (ns == 2) k_trans<2><<<(n + 127) / 128, 128>>>(lq, f, g, out, reset, n);
    else k_trans<13><<<(n + 127) / 128, 128>>>(lq, f, g, out, reset, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    d = tmp_path_factory.mktemp("sites")
    (d / "s.cu").write_text(SOURCE)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    out = []
    for name, flags in (("refined", ["-DCASTRO_NR_ARITH"]), ("ieee", [])):
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                        "-fPIC", *flags, "-I", os.path.join(PKG_DIR, "csrc"), "-o", str(d / f"{name}.so"),
                        str(d / "s.cu")], check=True)
        L = C.CDLL(str(d / f"{name}.so"))
        L.scalar.argtypes = [C.c_void_p] * 6 + [C.c_int]
        L.trans.argtypes = [C.c_int] + [C.c_void_p] * 5 + [C.c_int]
        out.append(L)
    return out


@pytest.mark.parametrize("exponent", [-120, -40, -1, 0, 1, 40, 120])
def test_seeds_quotient_and_floored_root(libs, exponent):
    import torch

    rng = np.random.default_rng(exponent + 500)
    lead = np.arange(1 << 20, dtype=np.uint64) << np.uint64(32)
    low = rng.integers(0, 1 << 32, 1 << 20, dtype=np.uint64)
    bits = np.concatenate([lead, lead | low, lead | np.uint64(0xffffffff)]) | (np.uint64(1023 + exponent) << np.uint64(52))
    b = bits.view(np.float64)
    a = b * b * 10.0 ** rng.uniform(-3, 3, b.size) * rng.choice([-1.0, 1.0], b.size)   # on either side of the floor's square
    a[::1000] = 0.0
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    er, es, q, f = (torch.empty_like(tb) for _ in range(4))
    assert libs[0].scalar(*(t.data_ptr() for t in (ta, tb, er, es, q, f)), b.size) == 0
    assert float(er.abs().max()) < 2.0 ** -18 and float(es.abs().max()) < 2.0 ** -18
    al, bl = a.astype(np.longdouble), b.astype(np.longdouble)
    assert (np.abs(q.cpu().numpy() - al / bl) <= 2.5 * U * ROOM * np.abs(al / bl)).all()
    ref = np.sqrt(np.maximum(bl * bl, np.abs(al)))
    assert (np.abs(f.cpu().numpy() - ref) <= 2.5 * U * ROOM * ref).all()


@pytest.mark.parametrize("ns", [2, 13])
def test_transverse_density_reset(libs, ns):
    import torch

    rng = np.random.default_rng(ns)
    n, nqs, ntf = 1 << 16, 6 + ns, 7 + ns
    lq = rng.uniform(0.5, 2.0, (n, nqs))
    f, g = rng.uniform(-4.0, 4.0, (n, 2, ntf)), rng.uniform(-4.0, 4.0, (n, 2, ntf))
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (lq, f, g)]
    got, flag = [], []
    for L in libs:
        out = torch.empty((n, 2, nqs), dtype=torch.float64, device="cuda")
        reset = torch.empty((2, n), dtype=torch.int32, device="cuda")
        assert L.trans(ns, *(t.data_ptr() for t in dev), out.data_ptr(), reset.data_ptr(), n) == 0
        got.append(out.cpu().numpy())
        flag.append(reset.cpu().numpy())
    np.testing.assert_array_equal(flag[0], flag[1])
    assert (0.05 < flag[0].mean(axis=1)).all() and (flag[0].mean(axis=1) < 0.95).all()
    a, b = got
    rho, vel, pres, rei = 0, slice(1, 4), 4, 5   # SRHO, SU..SW, SPRES, SREI
    np.testing.assert_array_equal(a[..., rho], b[..., rho])
    np.testing.assert_array_equal(a[..., pres], b[..., pres])
    assert (a[..., rho] > 0).all()
    quotients = [1, 2, 3] + list(range(6, nqs))
    assert (np.abs(a - b)[..., quotients] <= 4.5 * U * ROOM * np.abs(b[..., quotients])).all()
    # the corrected state's kinetic energy, 0.5 rho v^2, and the energy left after it
    ke = 0.5 * b[..., rho] * (b[..., vel] ** 2).sum(-1)
    assert (np.abs(a - b)[..., rei] <= (5.5 * ke + 2.0 * np.abs(b[..., rei])) * U * ROOM).all()
