"""Offsets of the FAB view (castro_common.cuh, Fab) against exact integer arithmetic, for planes of more than 2^32
points (34 GB a component: a one-component array of that size fits the GPU), rows and columns of them on either side of
2^31 and 2^32, and small ones.  The view's operator is host code as well as device code; this compiles the host side."""
from __future__ import annotations

import os
import random
import subprocess

from conftest import PKG_DIR

SOURCE = """
#include "castro_common.cuh"
#include <stdio.h>
int main()
{
    int lo[3], hi[3], i, j, k, n;
    double* const base = (double*)(1ull << 60);   // (an address only; nothing is read)
    while (scanf("%d %d %d %d %d %d %d %d %d %d", lo, lo + 1, lo + 2, hi, hi + 1, hi + 2, &i, &j, &k, &n) == 10) {
        const castro::Fab f = castro::make_fab(base, lo, hi);
        printf("%lld\\n", ((long long)&f(i, j, k, n) - (long long)base) / 8);
    }
    return 0;
}
"""

# extents of arrays: small, ragged, planes around 2^31 and 2^32 points, thin ones of as many rows
EXTENTS = [(1, 1, 1), (5, 3, 2), (1290, 1290, 1290), (1625, 1625, 1625), (1626, 1626, 1626), (2048, 2048, 1040),
           (1, 70000, 70000), (70000, 1, 70000), (70000, 70000, 1), (3, 40000, 40000), (100000, 100000, 2)]


def test_fab_offsets(tmp_path):
    (tmp_path / "fab.cu").write_text(SOURCE)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-I",
                    os.path.join(PKG_DIR, "csrc"), "-o", str(tmp_path / "fab"), str(tmp_path / "fab.cu")], check=True)
    rng = random.Random(0)
    lines, want = [], []
    for ext in EXTENTS:
        lo = [rng.randint(-9, 9) for _ in range(3)]
        hi = [l + n - 1 for l, n in zip(lo, ext)]
        corners = [lo, hi] + [[rng.randint(l, h) for l, h in zip(lo, hi)] for _ in range(20)]
        for p in corners:
            for n in (0, 1, 12):
                lines.append(" ".join(map(str, [*lo, *hi, *p, n])))
                x, y, z = (a - l for a, l in zip(p, lo))
                want.append(x + ext[0] * (y + ext[1] * (z + ext[2] * n)))
    out = subprocess.run([str(tmp_path / "fab")], input="\n".join(lines), capture_output=True, text=True, check=True)
    assert [int(v) for v in out.stdout.split()] == want
