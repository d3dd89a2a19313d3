"""Domains whose extents are the edge cases of the work items' point numbering (castro_sim.cu, item_point): extents of
one zone, rows shorter and longer than a block, a row longer than 2^15 zones (whose quotient has its own branch).  One
coarse step of the batched and the persistent path, and the box entry point's device-built items, exact build bit for
bit against the oracle, production build within 1e-12 of each component's magnitude."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from gpu_harness import RTOL_STEP, assert_match, from_dev, nan_dev, sborder_from_domain, to_dev

pytestmark = pytest.mark.gpu


def level(oracle, pkg, table, dims, bc):
    dx = 1.0 / max(dims)
    prob = pkg.configs.problem(r_init=4.0 * dx)
    inst = dict(dom_lo=(0, 0, 0), dom_hi=tuple(n - 1 for n in dims), problo=(0.0, 0.0, 0.0),
                probhi=tuple(n * dx for n in dims), bc=bc, boxes=[((0, 0, 0), tuple(n - 1 for n in dims))], problem=prob,
                n=dims[0])
    oracle.network_init(*pkg.configs.NET2)
    oracle.eos_init(table)
    lev, _ = oracle.level_from_instance(inst, 9)
    return inst, lev


@pytest.mark.parametrize("exact", [True, False], ids=["exact", "production"])
@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 5, 2), (3, 1, 130), (127, 2, 1), (129, 3, 2), (33000, 1, 1)], ids=str)
def test_extents(pkg, oracle, table, dims, exact):
    bc = 1 if dims[0] % 2 else 0
    inst, lev = level(oracle, pkg, table, dims, bc)
    start = oracle.assemble(lev, inst)
    lev.coarse_step(-1.0)
    ref = oracle.assemble(lev, inst)
    L = pkg.castro.init(*pkg.configs.NET2, table, exact=exact)
    for mode in (pkg.castro.MODE_BATCHED, pkg.castro.MODE_PERSISTENT):
        sim = pkg.make_sim(L, dict(instances=[inst]), mode)
        sim.init_data()
        sim.step(1)
        got = pkg.castro.assemble(inst, sim.box_states()[0])
        sim.close()
        assert_match(got, ref, exact, rtol=RTOL_STEP, what=f"mode {mode}")
    # the box entry point on the same state: its source from Sborder
    lo, hi = inst["dom_lo"], inst["dom_hi"]
    glo, ghi = [l - 4 for l in lo], [h + 4 for h in hi]
    sb = to_dev(sborder_from_domain(start, lo, lo, hi, bc))
    for _ in range(2):   # clean_state(S_old), pointwise, and clean_state(Sborder)
        pkg.castro.call(L, "castro_clean_state", glo, ghi, sb, glo, ghi)
    src = nan_dev(lo, hi, 9).zero_()
    dx = [(h - l) / n for l, h, n in zip(inst["problo"], inst["probhi"], dims)]   # the level's, which may differ by an ulp
    pkg.castro.call(L, "castro_construct_hydro_source_box", lo, hi, sb, glo, ghi, src, lo, hi, None, None, None, lo, hi,
                    dx, lev.dt)
    s = from_dev(src)
    assert np.isfinite(s).all()
    # Castro::advance by hand: S_old cleaned + dt * source, the two cleans of S_new
    u = to_dev(start)
    pkg.castro.call(L, "castro_clean_state", lo, hi, u, lo, hi)
    pkg.castro.call(L, "castro_saxpy", u, src, ctypes.c_longlong(u.numel()), float(lev.dt))
    for _ in range(2):
        pkg.castro.call(L, "castro_clean_state", lo, hi, u, lo, hi)
    assert_match(from_dev(u), ref, exact, rtol=RTOL_STEP, what="box entry point")
