"""Single-component calls on an array of more than 2^32 points (2048 x 2048 x 1040, 35 GB), in zones whose point number
is beyond 2^32: density tags, average_down from and into such an array, and the flux register's crse_init.  2^32 points
are 1024 planes of this array, so a number that wrapped would fall 1024 planes lower, which hold zeros here and must
stay so.  The results are compared with the same rules in numpy; a mean of eight values takes seven additions on either
side (and an exact product), so the two differ by at most 14 * 2^-53 of the mean magnitude."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NY, NZ = 2048, 2048, 1040
LO, HI = (0, 0, 0), (NX - 1, NY - 1, NZ - 1)
X0, Z0 = NX - 6, NZ - 6          # the corner region: 6 zones to each upper end
MEAN_TOL = 14 * 2.0 ** -53


@pytest.fixture(scope="module")
def big():
    import torch

    if torch.cuda.mem_get_info()[0] < 44 << 30:
        pytest.skip("needs 44 GB of free device memory")
    t = torch.empty((NZ, NY, NX), dtype=torch.float64, device="cuda")
    yield t
    del t
    torch.cuda.empty_cache()


@pytest.fixture
def corner(big):
    """(array, the corner region's values as [x, y, z]); the planes a wrapped number would reach are zero."""
    import torch

    v = np.random.default_rng(3).uniform(0.5, 2.0, (6, 6, 6))
    big[Z0 - 1024:Z0 - 1018].zero_()
    big[Z0:, X0:, X0:] = torch.from_numpy(np.ascontiguousarray(v.transpose(2, 1, 0))).cuda()
    yield big, v
    assert float(big[Z0 - 1024:Z0 - 1018].abs().max()) == 0.0


def _call(pkg, L, name, *args):
    import torch

    K = pkg.castro
    conv = [K.ivec(a) if isinstance(a, tuple) else C.c_void_p(a.data_ptr()) if hasattr(a, "data_ptr") else a for a in args]
    getattr(L, name)(*conv)
    torch.cuda.synchronize()
    K.check(L, name)


def test_density_tags(pkg, table, corner):
    import torch

    t, v = corner
    L = pkg.castro.init(*pkg.configs.NET2, table)
    lo, hi = (X0 + 1, X0 + 1, Z0 + 1), (X0 + 4, X0 + 4, Z0 + 4)
    tag = torch.zeros((4, 4, 4), dtype=torch.int8, device="cuda")
    pkg.castro.call(L, "denerror", lo, hi, C.c_void_p(tag.data_ptr()), lo, hi, t, LO, HI, 1, 0)
    torch.cuda.synchronize()
    c = v[1:5, 1:5, 1:5]
    step = [np.abs(v[1 + a:5 + a, 1 + b:5 + b, 1 + d:5 + d] - c)
            for a, b, d in ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1))]
    want = (np.max(step, axis=0) >= np.abs(0.25 * c)).astype(np.int8)
    assert 0 < want.sum() < want.size
    np.testing.assert_array_equal(tag.cpu().numpy().transpose(2, 1, 0), want)


def test_average_down_from_it(pkg, table, corner):
    import torch

    t, v = corner
    L = pkg.castro.init(*pkg.configs.NET2, table)
    clo = (X0 // 2, X0 // 2, Z0 // 2)
    chi = tuple(c + 2 for c in clo)
    out = torch.zeros((3, 3, 3), dtype=torch.float64, device="cuda")
    _call(pkg, L, "castro_average_down", clo, chi, out, clo, chi, t, LO, HI, 1, 2)
    ref = v.reshape(3, 2, 3, 2, 3, 2).mean(axis=(1, 3, 5))
    np.testing.assert_allclose(out.cpu().numpy().transpose(2, 1, 0), ref, rtol=MEAN_TOL)


def test_average_down_into_it(pkg, table, corner):
    import torch

    t, _ = corner
    L = pkg.castro.init(*pkg.configs.NET2, table)
    lo, hi = (X0, X0, Z0), (X0 + 5, X0 + 5, Z0 + 5)
    flo, fhi = tuple(2 * c for c in lo), tuple(2 * c + 1 for c in hi)
    f = np.random.default_rng(4).standard_normal((12, 12, 12))
    _call(pkg, L, "castro_average_down", lo, hi, t, LO, HI, torch.from_numpy(f).cuda(), flo, fhi, 1, 2)
    ref = f.reshape(6, 2, 6, 2, 6, 2).mean(axis=(1, 3, 5))
    np.testing.assert_allclose(t[Z0:, X0:, X0:].cpu().numpy(), ref, rtol=0, atol=MEAN_TOL * np.abs(f).max())


def test_flux_register_on_it(pkg, table, corner):
    import torch

    t, v = corner
    L = pkg.castro.init(*pkg.configs.NET2, table)
    lo, hi = (X0, X0, Z0), (X0 + 5, X0 + 5, Z0 + 5)
    reg = torch.zeros((6, 6, 6), dtype=torch.float64, device="cuda")
    _call(pkg, L, "castro_flux_register_crse_init", lo, hi, reg, lo, hi, t, LO, HI, 1)
    np.testing.assert_array_equal(reg.cpu().numpy().transpose(2, 1, 0), -v)
