"""The box entry points captured in a caller's CUDA graph (they launch each kernel but the first behind its predecessor,
so the graph holds programmatic edges): two calls in a row over the same scratch, replayed on inputs that were not there
when they were captured, must give what direct calls give, bit for bit.  A box on either side of the line where the two
trace passes go from one launch to two."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gpu_harness import to_dev
from test_gpu_box_flow import flow

pytestmark = pytest.mark.gpu


def _inputs(pkg, L, dims, nspec, e0, seed):
    glo, ghi = [-4] * 3, [n + 3 for n in dims]
    sb = to_dev(flow(np.random.default_rng(seed), glo, ghi, nspec, e0))
    for _ in range(2):
        pkg.castro.call(L, "castro_clean_state", glo, ghi, sb, glo, ghi)
    return sb


@pytest.mark.parametrize("entry", ["castro_construct_hydro_source_box", "castro_construct_hydro_source_box_noalloc"])
@pytest.mark.parametrize("nspec", [2, 13])
@pytest.mark.parametrize("dims", [(7, 5, 9), (16, 16, 16), (34, 34, 34)], ids=str)
def test_captured_box_calls(pkg, table, dims, nspec, entry):
    import torch

    if entry.endswith("noalloc") and dims[0] > 16:
        pytest.skip("beyond the static scratch")
    net = pkg.configs.NET2 if nspec == 2 else pkg.configs.NET13
    L = pkg.castro.init(*net, table)
    nv = 7 + nspec
    lo, hi = [0, 0, 0], [n - 1 for n in dims]
    glo, ghi = [-4] * 3, [n + 3 for n in dims]
    e0 = 1.0e14
    first, second = (_inputs(pkg, L, dims, nspec, e0, s) for s in (1, 2))
    n = max(dims)
    dx, dt = [1.0 / n] * 3, 0.05 / n / np.sqrt(e0)
    shape = (nv,) + tuple(dims[::-1])
    src = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(2)]
    flux = [[torch.zeros((nv,) + tuple(dims[2 - a] + (2 - a == d) for a in range(3)), dtype=torch.float64, device="cuda")
             for d in range(3)] for _ in range(2)]
    flo = (C.c_int * 9)(*([0] * 9))
    fhi = (C.c_int * 9)(*[hi[k] + (k == d) for d in range(3) for k in range(3)])
    sb = [torch.empty_like(first) for _ in range(2)]

    def calls():
        for m in range(2):
            src[m].zero_()
            ptr = (C.c_void_p * 3)(*[f.data_ptr() for f in flux[m]])
            pkg.castro.call(L, entry, lo, hi, sb[m], glo, ghi, src[m], lo, hi, ptr, flo, fhi, lo, hi, dx, dt)

    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    try:
        with torch.cuda.stream(stream):
            L.castro_set_stream(C.c_void_p(stream.cuda_stream))
            want = []
            for a, b in ((first, second), (second, first)):
                sb[0].copy_(a)
                sb[1].copy_(b)
                calls()
                stream.synchronize()
                want.append([t.clone() for m in range(2) for t in (src[m], *flux[m])])
            with torch.cuda.graph(graph, stream=stream):
                calls()
            for rep, (a, b) in enumerate(((first, second), (second, first), (first, second))):
                sb[0].copy_(a)
                sb[1].copy_(b)
                for m in range(2):
                    for t in (src[m], *flux[m]):
                        t.fill_(float("nan"))
                graph.replay()
                stream.synchronize()
                for got, ref in zip([t for m in range(2) for t in (src[m], *flux[m])], want[rep % 2]):
                    assert torch.isfinite(ref).all() and torch.equal(got, ref)
    finally:
        L.castro_set_stream(C.c_void_p(0))
        torch.cuda.synchronize()
    assert not torch.equal(want[0][0], want[1][0])
