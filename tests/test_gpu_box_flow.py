"""The box entry point on flow that is supersonic towards every face (Mach -3 to 3, density and energy varying by a
tenth from zone to zone): the traces' characteristic terms then take every combination of signs, not only those of
subsonic flow.  Boxes of one zone, of ragged extents, and of the two extents beside the line where the two trace passes
go from one launch to two (2 x 201 and 2 x 243 blocks against 444).

The exact build must equal the oracle bit for bit.  The production build rounds differently by some 1e-15 a zone, and a
limiter that then falls on its other side moves one zone of the box by at most its slope, so its relative L1 distance is
held to RTOL_L1."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gpu_harness import RTOL_L1, assert_match, from_dev, rel_l1, to_dev

pytestmark = pytest.mark.gpu


def flow(rng, lo, hi, nspec, e0):
    """A state on [lo, hi]: density 1, energy e0 per mass, velocities up to 3 sqrt(e0), each with noise."""
    shape = tuple(h - l + 1 for l, h in zip(lo, hi))
    u = np.zeros(shape + (7 + nspec,), order="F")
    rho = 1.0 + 0.1 * rng.uniform(-1, 1, shape)
    e = e0 * (1.0 + 0.1 * rng.uniform(-1, 1, shape))
    x = np.meshgrid(*[np.arange(n) / 7.0 for n in shape], indexing="ij")
    ke = 0.0
    for d in range(3):
        v = np.sqrt(e0) * (2.7 * np.sin(x[d] + 2.0 * x[(d + 1) % 3] + d) + 0.3 * rng.uniform(-1, 1, shape))
        u[..., 1 + d] = rho * v
        ke = ke + 0.5 * rho * v * v
    u[..., 0] = rho
    u[..., 4] = rho * e + ke
    u[..., 5] = rho * e
    u[..., 6] = 1e6
    X = rng.uniform(0.5, 1.5, shape + (nspec,))
    u[..., 7:] = rho[..., None] * X / X.sum(-1, keepdims=True)
    return u


@pytest.mark.parametrize("exact", [True, False], ids=["exact", "production"])
@pytest.mark.parametrize("nspec", [2, 13])
@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 3, 2), (33, 33, 33), (34, 34, 34)], ids=str)
def test_box_supersonic(pkg, oracle, table, dims, nspec, exact):
    net = pkg.configs.NET2 if nspec == 2 else pkg.configs.NET13
    oracle.network_init(*net)
    oracle.eos_init(table)
    one = dict(dom_lo=(0, 0, 0), dom_hi=(0, 0, 0), problo=(0.0,) * 3, probhi=(1.0,) * 3, bc=1,
               boxes=[((0, 0, 0), (0, 0, 0))], n=1,
               problem=pkg.configs.problem(r_init=1e-3, T_ambient=1e6, X=[1.0 / nspec] * nspec))
    lev, _ = oracle.level_from_instance(one, 7 + nspec)
    s0 = oracle.assemble(lev, one)[0, 0, 0]
    e0 = s0[5] / s0[0]
    lo, hi = [0, 0, 0], [n - 1 for n in dims]
    glo, ghi = [-4] * 3, [h + 4 for h in hi]
    sb = flow(np.random.default_rng(sum(dims) + nspec), glo, ghi, nspec, e0)
    for name in ("enforce_minimum_density", "normalize_species", "reset_internal_e", "compute_temp"):
        oracle.call(name, glo, ghi, sb, glo, ghi)
    n = max(dims)
    dx = [1.0 / n] * 3
    dt = 0.05 * dx[0] / np.sqrt(e0)
    ref = np.zeros(dims + (7 + nspec,), order="F")
    oracle.lib().oracle_construct_hydro_source_tile(
        oracle.ivec(lo), oracle.ivec(hi), sb.ctypes.data_as(C.POINTER(C.c_double)), oracle.ivec(glo), oracle.ivec(ghi),
        ref.ctypes.data_as(C.POINTER(C.c_double)), oracle.ivec(lo), oracle.ivec(hi), oracle.ivec(lo), oracle.ivec(hi),
        oracle.dvec(dx), C.c_double(dt))
    assert np.isfinite(ref).all() and (np.abs(ref[..., 0]) > 0).all()
    L = pkg.castro.init(*net, table, exact=exact)
    src = to_dev(np.zeros_like(ref))
    state = to_dev(sb)
    pkg.castro.call(L, "castro_construct_hydro_source_box", lo, hi, state, glo, ghi, src, lo, hi, None, None, None, lo, hi,
                    dx, dt)
    got = from_dev(src)
    if exact:
        assert_match(got, ref, True, what="source")
    else:
        live = [c for c in range(ref.shape[-1]) if c != 6]   # no source of temperature
        assert (rel_l1(got, ref)[live] <= RTOL_L1).all()
