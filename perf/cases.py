"""Work that programs have this framework do, as cases that can be timed.

A case is a dict of plain values.  ``listed()`` names the standing ones,
``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes what a
program holds before the call (the simulation, the boxes of a host code, a
gradient handle) from a seed, ``run`` is one pass through the public entry
points, ``work`` what that pass cannot do without, and ``exact`` the same
outputs from plain float64 torch operations.

Kinds of work:

* ``sim``      -- a Sedov level advanced by coarse steps (``Sim.step``): one
                  domain cut into boxes, any aspect, odd sizes, 2 or 13 species,
                  outflow or periodic.
* ``ensemble`` -- many independent Sedov instances of mixed sizes in one sim.
* ``host``     -- upload, some steps and download in one call from pinned host
                  memory (``castro_sim_run_host``), as a coupled host code runs.
* ``box``      -- the hydro source and face fluxes of one box of a host code's
                  own BoxArray (``castro_construct_hydro_source_box``).
* ``adjoint``  -- the objective and its gradient (``SedovAdjoint``).
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

NET = {2: ([4.0, 16.0], [2.0, 8.0]),
       13: ([4., 12., 16., 20., 24., 28., 32., 36., 40., 44., 48., 52., 56.],
            [2., 6., 8., 10., 12., 14., 16., 18., 20., 22., 24., 26., 28.])}
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"   # (no GPU: only the plain torch part can run)
WARM_STEPS = 2   # steps a sim has taken before the timed ones: its blast has begun to move


def listed():
    return [
        # the smallest level: one 16^3 box, where launches and latency are the time
        dict(name="sim 16 one box", kind="sim", nx=16, ny=16, nz=16, cuts=1, ns=2, bc=1, steps=1),
        # the reference CPU case: one 64^3 box
        dict(name="sim 64 one box", kind="sim", nx=64, ny=64, nz=64, cuts=1, ns=2, bc=1, steps=1),
        # the headline workload: 128^3 in 64 boxes of 32^3
        dict(name="sim 128 64 boxes", kind="sim", nx=128, ny=128, nz=128, cuts=4, ns=2, bc=1, steps=1),
        # the largest level here: 256^3 in an uneven BoxArray
        dict(name="sim 256 uneven", kind="sim", nx=256, ny=256, nz=256, cuts=-6, ns=2, bc=1, steps=1),
        # a flat domain of odd extents in an uneven BoxArray, periodic
        dict(name="sim 97x61x45 periodic", kind="sim", nx=97, ny=61, nz=45, cuts=-3, ns=2, bc=0, steps=1),
        # the reference problem's 13 species, periodic, 8 boxes
        dict(name="sim 64 13 species", kind="sim", nx=64, ny=64, nz=64, cuts=2, ns=13, bc=0, steps=1),
        # 32 independent instances of 32^3 .. 96^3 in one batched sim
        dict(name="ensemble 32", kind="ensemble", ninst=32, nmin=32, nmax=96, sizes=7, steps=1),
        # a host code that keeps its state in host memory: upload, 10 steps, download
        dict(name="host 64 10 steps", kind="host", nx=64, ny=64, nz=64, cuts=2, ns=2, bc=1, steps=10),
        # one box of a host code's loop over its own boxes
        dict(name="box 32", kind="box", nx=32, ny=32, nz=32, ns=2),
        # a small box with the full network
        dict(name="box 16 13 species", kind="box", nx=16, ny=16, nz=16, ns=13),
        # gradients: the tests' size, and the 64^3, 20-step configuration
        dict(name="adjoint 32 10 steps", kind="adjoint", n=32, steps=10, checkpoint=5),
        dict(name="adjoint 64 20 steps", kind="adjoint", n=64, steps=20, checkpoint=5),
    ]


def draw(rng):
    kind = rng.choice(["sim", "sim", "sim", "box", "ensemble", "host", "adjoint"])

    def extent(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind in ("sim", "host"):
        top = 160 if kind == "sim" else 96
        return dict(kind=kind, nx=extent(10, top), ny=extent(10, top), nz=extent(10, top),
                    cuts=rng.choice([1, 1, 2, -2, -3]), ns=rng.choice([2, 2, 13]), bc=rng.choice([0, 1]),
                    steps=rng.randint(1, 3) if kind == "sim" else rng.randint(2, 10))
    if kind == "box":
        return dict(kind=kind, nx=extent(8, 64), ny=extent(8, 64), nz=extent(8, 64), ns=rng.choice([2, 13]))
    if kind == "ensemble":
        lo = extent(16, 40)
        return dict(kind=kind, ninst=rng.randint(4, 32), nmin=lo, nmax=lo + rng.randint(8, 40),
                    sizes=rng.randint(0, 10 ** 6), steps=1)
    return dict(kind=kind, n=extent(12, 56), steps=rng.randint(3, 10), checkpoint=rng.randint(2, 5))


# ---------------------------------------------------------------------------
# what a program holds
# ---------------------------------------------------------------------------
_lib = {}


def _package():
    if "mini_castro_b200" not in sys.modules:
        d = os.path.join(ROOT, "mini-castro_b200")
        spec = importlib.util.spec_from_file_location("mini_castro_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["mini_castro_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["mini_castro_b200"]


def _library(ns):
    """The library with its table loaded (once per process) and the species network set."""
    pkg = _package()
    if "L" not in _lib:
        _lib["L"] = pkg.castro.init(*NET[ns], pkg.helm_table.ensure_table())
        _lib["ns"] = ns
    if _lib["ns"] != ns:
        a, z = (np.asarray(v, dtype=np.float64) for v in NET[ns])
        p = ctypes.POINTER(ctypes.c_double)
        _lib["L"].castro_network_init(len(a), a.ctypes.data_as(p), z.ctypes.data_as(p))
        pkg.castro.check(_lib["L"], "castro_network_init")
        _lib["ns"] = ns
    return pkg, _lib["L"]


def _cut(n, cuts, rng):
    """Sizes of the pieces of n zones: |cuts| near-equal ones, uneven (seeded) ones for cuts < 0."""
    k = max(1, min(abs(cuts), n // 4))
    if cuts < 0:
        inner = rng.permutation(np.arange(1, n // 4))[:k - 1] * 4
        edges = np.concatenate([[0], np.sort(inner), [n]])
    else:
        edges = np.linspace(0, n, k + 1).round().astype(int)
    return [int(b - a) for a, b in zip(edges[:-1], edges[1:])]


def _smooth(shape, width, gen):
    """Unit-variance Gaussian field on the GPU, smoothed over `width` zones (periodic)."""
    f = torch.fft.rfftn(torch.randn(shape, dtype=torch.float64, device=DEVICE, generator=gen))
    for ax, n in enumerate(shape):
        k = (torch.fft.rfftfreq(n) if ax == len(shape) - 1 else torch.fft.fftfreq(n)).to(DEVICE, torch.float64)
        w = torch.exp(-2.0 * (math.pi * width * k) ** 2)
        f = f * w.reshape([-1 if a == ax else 1 for a in range(len(shape))])
    g = torch.fft.irfftn(f, s=shape)
    return (g - g.mean()) / g.std()


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _instance(dims, cuts, ns, bc, seed, energy=None, rho=None, pert=True):
    """One Sedov instance: domain, BoxArray, boundary condition, problem constants."""
    rng = np.random.default_rng(int(seed))
    shape = np.random.default_rng(abs(cuts) * 1000 + sum(dims))   # the BoxArray belongs to the case
    cfgs = _package().configs
    boxes = cfgs.boxes_from_sizes(*[_cut(n, cuts, shape) for n in dims])
    if ns == 2:
        dx = 1.0 / max(dims)
        p = cfgs.problem(exp_energy=energy or 10.0 ** rng.uniform(49.9, 50.1), dens_ambient=rho or 1.0)
    else:   # the Source/Prob.F90 problem
        dx = 1e9 / max(dims)
        X = rng.uniform(0.2, 1.0, ns)
        p = cfgs.problem(ambient_from_T=0, dens_ambient=1e4, p_ambient=1e21,
                         exp_energy=10.0 ** rng.uniform(51.9, 52.1), X=list(X / X.sum()), T_init=1e9)
    p["r_init"] = 4.0 * dx
    if pert:
        g = _smooth((dims[2], dims[1], dims[0]), 4.0, _generator(seed))
        p["pert"], p["pert_amp"] = np.asfortranarray(g.cpu().numpy().transpose(2, 1, 0)), 1e-3
    return dict(dom_lo=(0, 0, 0), dom_hi=tuple(n - 1 for n in dims), problo=(0.0, 0.0, 0.0),
                probhi=tuple(n * dx for n in dims), bc=bc, boxes=boxes, problem=p, n=dims[0])


def _instances(case, seed):
    if case["kind"] == "ensemble":
        sizes = np.random.default_rng(case["sizes"]).integers(case["nmin"], case["nmax"] + 1, case["ninst"])
        rng = np.random.default_rng(int(seed))
        return [_instance((int(n),) * 3, -(-int(n) // 64), 2, 1, seed, 10.0 ** rng.uniform(49.0, 51.0),
                          10.0 ** rng.uniform(-1.0, 1.0), pert=False) for n in sizes]
    if case["kind"] == "adjoint":
        return [_instance((case["n"],) * 3, 1, 2, 1, seed)]
    return [_instance((case["nx"], case["ny"], case["nz"]), case["cuts"], case["ns"], case["bc"], seed)]


class _Memory:
    """The n doubles of `owner` at a device address; a tensor made of it (no copy) keeps the owner alive."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}


def _box_inputs(case, seed):
    """A host code's cleaned Sborder of one box, (NVAR, nz+8, ny+8, nx+8): a smooth, moving
    13- or 2-species gas in the table's range, with its zone width and time step."""
    ns = case["ns"]
    shape = tuple(case[k] + 8 for k in ("nz", "ny", "nx"))
    gen = _generator(seed)
    field = lambda: _smooth(shape, 3.0, gen).clamp(-3.0, 3.0)  # noqa: E731
    rho = 1e4 * torch.exp(0.4 * field())
    T = 1e9 * torch.exp(0.3 * field())
    X = torch.stack([torch.exp(0.3 * field()) for _ in range(ns)])
    X = X / X.sum(0)
    A = torch.tensor(NET[ns][0], dtype=torch.float64, device=DEVICE)
    Z = torch.tensor(NET[ns][1], dtype=torch.float64, device=DEVICE)
    ions = (X / A[:, None, None, None]).sum(0)
    ye = (X * (Z / A)[:, None, None, None]).sum(0)
    e = 1.5 * 1.380650424e-16 * 6.0221417930e23 * T * (ions + ye) + 4.0 * 5.67051e-5 / 2.99792458e10 * T ** 4 / rho
    cs = torch.sqrt(0.5 * e)
    vel = [0.4 * cs * field() for _ in range(3)]
    ke = 0.5 * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2)
    U = torch.stack([rho, rho * vel[0], rho * vel[1], rho * vel[2], rho * (e + ke), rho * e, T] + list(rho * X))
    dx = 1e7
    dt = float(0.2 * dx / (cs * 3.0).max())
    return U.contiguous(), dx, dt


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    s.steps = case.get("steps")
    pkg, s.L = _library(case.get("ns", 2))
    s.pkg = pkg
    if s.kind == "box":
        n = [case[k] for k in ("nx", "ny", "nz")]
        s.sb, dx, s.dt = _box_inputs(case, seed)
        s.dx = [dx] * 3
        s.lo, s.hi = [0, 0, 0], [k - 1 for k in n]
        s.glo, s.ghi = [-4, -4, -4], [k + 3 for k in n]
        pkg.castro.call(s.L, "castro_clean_state", s.glo, s.ghi, s.sb, s.glo, s.ghi)
        nv = s.sb.shape[0]
        s.src = torch.empty((nv, n[2], n[1], n[0]), dtype=torch.float64, device=DEVICE)
        s.flux = [torch.empty((nv,) + tuple(n[2 - a] + (2 - a == d) for a in range(3)), dtype=torch.float64, device=DEVICE)
                  for d in range(3)]
        s.fptr = (ctypes.c_void_p * 3)(*[f.data_ptr() for f in s.flux])
        s.flo = (ctypes.c_int * 9)(*([0] * 9))
        s.fhi = (ctypes.c_int * 9)(*[s.hi[k] + (k == d) for d in range(3) for k in range(3)])
        torch.cuda.synchronize()
        return s
    insts = _instances(case, seed)
    if s.kind == "adjoint":
        s.inst = insts[0]
        s.run = pkg.adjoint.SedovAdjoint(s.L, s.inst, case["steps"], case["checkpoint"])
        return s
    s.sim = pkg.make_sim(s.L, dict(instances=insts))
    s.sim.init_data()
    n = s.sim.total_size
    if s.kind == "host":
        s.host_in = torch.empty(n, dtype=torch.float64, pin_memory=True)
        s.host_out = torch.empty(n, dtype=torch.float64, pin_memory=True)
        s.L.castro_sim_download(s.sim.h, s.host_in.data_ptr())
        s.sim.sync()
        s.L.castro_sim_run_host(s.sim.h, s.host_in.data_ptr(), 1, s.host_out.data_ptr())
        pkg.castro.check(s.L, "castro_sim_run_host")
        return s
    s.sim.step(WARM_STEPS)
    s.sim.sync()
    s.U = torch.as_tensor(_Memory(s.sim, s.L.castro_sim_box_state(s.sim.h, 0, 0), n), device=DEVICE)
    # one box: its components are planes of the state; more boxes: the state as it lies in memory
    s.out = list(s.U.reshape(7 + case.get("ns", 2), -1)) if len(insts) == 1 and len(insts[0]["boxes"]) == 1 else s.U
    return s


def run(s):
    if s.kind in ("sim", "ensemble"):
        s.sim.step(s.steps)
        return s.out
    if s.kind == "host":
        s.L.castro_sim_run_host(s.sim.h, s.host_in.data_ptr(), s.steps, s.host_out.data_ptr())
        s.pkg.castro.check(s.L, "castro_sim_run_host")
        return s.host_out
    if s.kind == "box":
        s.src.zero_()   # hydro_source.setVal(0)
        s.pkg.castro.call(s.L, "castro_construct_hydro_source_box", s.lo, s.hi, s.sb, s.glo, s.ghi, s.src, s.lo, s.hi,
                          s.fptr, s.flo, s.fhi, s.lo, s.hi, s.dx, s.dt)
        return dict(source=s.src, fluxes=s.flux)
    p = s.inst["problem"]
    J = s.run.forward(p["exp_energy"], p["dens_ambient"])
    dE, drho, dpert = s.run.backward()
    return dict(J=J, dE=dE, drho=drho, dpert=dpert, final=s.run.final_state())


def work(case):
    """State read and written once a step; FP64 operations of the algorithm's stages a zone and step (the transverse
    and Riemann stages carry each species)."""
    kind = case["kind"]
    if kind == "ensemble":
        sizes = np.random.default_rng(case["sizes"]).integers(case["nmin"], case["nmax"] + 1, case["ninst"])
        zones = int(sum(int(n) ** 3 for n in sizes))
    elif kind == "adjoint":
        zones = case["n"] ** 3
    else:
        zones = case["nx"] * case["ny"] * case["nz"]
    ns = case.get("ns", 2)
    nv, steps = 7 + ns, case.get("steps", 1)
    flops = (12.0e3 + 500.0 * ns) * zones * steps
    if kind == "box":
        grown = (case["nx"] + 8) * (case["ny"] + 8) * (case["nz"] + 8)
        return {"bytes": 8.0 * nv * (grown + 4 * zones), "flops": 0.7 * flops}
    if kind == "adjoint":   # forward, recompute and reverse (twice the forward's operations) of every step
        return {"bytes": 5 * 16.0 * nv * zones * steps, "flops": 4.0 * flops}
    return {"bytes": 16.0 * nv * zones * steps, "flops": flops}


# ---------------------------------------------------------------------------
# the same outputs from plain float64 torch operations.  Arrays are (z, y, x);
# _ax(d) is the axis of direction d.
# ---------------------------------------------------------------------------
SMALL_DENS, SMALL_PRES, SMALL, SMALLU, SMALL_TEMP = 1e-12, 1e-200, 1e-8, 1e-12, 1e3
IMAX, JMAX = 541, 201


def _ax(d):
    return 2 - d


def _cut_of(a, d, lo, n):
    return a.narrow(_ax(d), lo, n)


class _Gas:
    """Helmholtz EOS on the table file, for one network."""

    def __init__(self, ns):
        path = _package().helm_table.DEFAULT_PATH
        with open(path) as f:
            v = np.fromstring(f.read().replace("D", "E"), sep=" ")
        m = IMAX * JMAX
        a, b = v[:9 * m].reshape(m, 9), v[9 * m:13 * m].reshape(m, 4)
        # free energy by [density order][temperature order], then dp/dd and its derivatives likewise
        self.f = torch.from_numpy(np.ascontiguousarray(a[:, [0, 2, 4, 1, 5, 7, 3, 6, 8]])).to(DEVICE)
        self.dp = torch.from_numpy(np.ascontiguousarray(b[:, [0, 2, 1, 3]])).to(DEVICE)
        self.t = torch.tensor([10.0 ** (3.0 + j * (10.0 / 200.0)) for j in range(JMAX)], dtype=torch.float64, device=DEVICE)
        self.d = torch.tensor([10.0 ** (-12.0 + i * (27.0 / 540.0)) for i in range(IMAX)], dtype=torch.float64, device=DEVICE)
        self.A = torch.tensor(NET[ns][0], dtype=torch.float64, device=DEVICE)
        self.Z = torch.tensor(NET[ns][1], dtype=torch.float64, device=DEVICE)

    @staticmethod
    def _axis(nodes, x, n):
        i = (torch.bucketize(x, nodes, right=True) - 1).clamp(0, n - 2)
        return i, nodes[i], nodes[i + 1] - nodes[i]

    def eval(self, rho, T, ions, ye):
        din = ye * rho
        i, d0, dd = self._axis(self.d, din, IMAX)
        j, t0, dt = self._axis(self.t, T, JMAX)
        xd, xt = ((din - d0) / dd).clamp(min=0.0), ((T - t0) / dt).clamp(min=0.0)

        def basis(z, h):   # quintic Hermite value, first and second derivative weights, lower node
            p = [z ** 3 * (z * (-6 * z + 15) - 10) + 1, z * (z * z * (z * (-3 * z + 8) - 6) + 1) * h,
                 0.5 * z * z * (z * (z * (-z + 3) - 3) + 1) * h * h]
            q = [z * z * (z * (-30 * z + 60) - 30) / h, z * z * (z * (-15 * z + 32) - 18) + 1,
                 0.5 * z * (z * (z * (-5 * z + 12) - 9) + 2) * h]
            r = [z * (z * (-120 * z + 180) - 60) / (h * h), z * (z * (-60 * z + 96) - 36) / h,
                 0.5 * (z * (z * (-20 * z + 36) - 18) + 2)]
            return p, q, r

        def both(z, h):
            lo, up = basis(z, h), basis(1 - z, h)
            sign = ((1, -1, 1), (-1, 1, -1), (1, -1, 1))
            return [[(lo[k][o], sign[k][o] * up[k][o]) for o in range(3)] for k in range(3)]

        wd, wt = both(xd, dd), both(xt, dt)
        F = dict.fromkeys(("f", "fd", "ft", "ftt", "fdt"), 0.0)
        for a in range(3):
            for di in range(2):
                g = [0.0, 0.0, 0.0]
                for b in range(3):
                    for dj in range(2):
                        v = self.f[(j + dj) * IMAX + i + di, 3 * a + b]
                        for k in range(3):
                            g[k] = g[k] + v * wt[k][b][dj]
                s, ds = wd[0][a][di], wd[1][a][di]
                F["f"] = F["f"] + g[0] * s
                F["fd"] = F["fd"] + g[0] * ds
                F["ft"] = F["ft"] + g[1] * s
                F["ftt"] = F["ftt"] + g[2] * s
                F["fdt"] = F["fdt"] + g[1] * ds

        def cubic(z, h):
            lo = (z * z * (2 * z - 3) + 1, z * (z * (z - 2) + 1) * h)
            m = 1 - z
            return lo, (m * m * (2 * m - 3) + 1, -m * (m * (m - 2) + 1) * h)

        cd, ct = cubic(xd, dd), cubic(xt, dt)
        dpe = 0.0
        for di in range(2):
            for dj in range(2):
                for a in range(2):
                    for b in range(2):
                        dpe = dpe + self.dp[(j + dj) * IMAX + i + di, 2 * a + b] * cd[di][a] * ct[dj][b]
        asol3, kav = 4.0 * 5.67051e-5 / 2.99792458e10 / 3.0, 1.380650424e-16 * 6.0221417930e23
        prad, pion = asol3 * T ** 4, kav * ions * rho * T
        erad, eion = 3 * prad / rho, 1.5 * pion / rho
        sele, dsepdt = -F["ft"] * ye, -F["ftt"] * ye
        o = _State()
        o.p = prad + pion + din * din * F["fd"]
        o.e = erad + eion + ye * F["f"] + T * sele
        dpdr = kav * ions * T + (ye * dpe).clamp(min=0.0)
        o.dpdT = 4 * asol3 * T ** 3 + kav * ions * rho + din * din * F["fdt"]
        o.dedT = 12 * asol3 * T ** 3 / rho + 1.5 * kav * ions + T * dsepdt
        chit = T / o.p * o.dpdT
        o.gam1 = chit * (o.p / rho) * chit / (T * o.dedT) + dpdr * rho / o.p
        return o

    def composition(self, X):
        """sum(X/A) and sum(X Z/A) of fractions X (any scale)."""
        k = (slice(None),) + (None,) * (X.dim() - 1)
        return (X / self.A[k]).sum(0), (X * (self.Z / self.A)[k]).sum(0)

    def invert(self, rho, T, want, ions, ye, what="e"):
        """Newton inversion for T, each zone stopping at its own convergence."""
        T = T.clone()
        todo = torch.arange(T.numel(), device=T.device)
        rho, want, ions, ye, flat = (v.expand_as(T).reshape(-1) for v in (rho, want, ions, ye, T))
        flat = flat.clone()
        for _ in range(100):
            if not todo.numel():
                break
            left = []
            for t in todo.split(2_000_000):
                old = flat[t]
                o = self.eval(rho[t], old, ions[t], ye[t])
                v, dv = (o.e, o.dedT) if what == "e" else (o.p, o.dpdT)
                new = torch.maximum(0.5 * old, torch.minimum(old - (v - want[t]) / dv, 2.0 * old)).clamp(min=1e3)
                flat[t] = new
                left.append(t[((new - old) / old).abs() >= 1e-8])
            todo = torch.cat(left)
        return flat.reshape(T.shape)

    def state(self, rho, T, ions, ye):
        p, g = torch.empty_like(rho).reshape(-1), torch.empty_like(rho).reshape(-1)
        r, t, a, y = (v.reshape(-1) for v in (rho, T, ions, ye))
        for q in torch.arange(r.numel(), device=r.device).split(2_000_000):
            o = self.eval(r[q], t[q], a[q], y[q])
            p[q], g[q] = o.p, o.gam1
        return p.reshape(rho.shape), g.reshape(rho.shape)


def _clean(gas, U):
    """Castro::clean_state on (NVAR, z, y, x), densities above the floor."""
    U = U.clone()
    rho = U[0]
    X = torch.maximum(1e-30 * rho, torch.minimum(rho, U[7:]))
    U[7:] = X / X.sum(0)
    ke = 0.5 * rho * ((U[1] / rho) ** 2 + (U[2] / rho) ** 2 + (U[3] / rho) ** 2)
    re = U[4] - ke
    U[5] = torch.where((re > 0) & (re / U[4] > 1e-4), re, U[5])
    ions, ye = gas.composition(U[7:] / rho)
    U[6] = gas.invert(rho, U[6], U[5] / rho, ions, ye)
    return U


def _sound_dt(gas, U, dx):
    rho = U[0]
    ions, ye = gas.composition(U[7:] / rho)
    T = gas.invert(rho, U[6], U[5] / rho, ions, ye)
    p, g = gas.state(rho, T, ions, ye)
    c = torch.sqrt(g * p / rho)
    return min(float((dx / (c + (U[1 + d] / rho).abs())).min()) for d in range(3))


def _grow(U, bc, g=4):
    for d in range(3):
        n = U.shape[1 + _ax(d)]
        i = torch.arange(-g, n + g, device=U.device)
        U = U.index_select(1 + _ax(d), i % n if bc == 0 else i.clamp(0, n - 1))
    return U


def _prim(gas, U):
    rho = U[0]
    q = {"r": rho, 0: U[1] / rho, 1: U[2] / rho, 2: U[3] / rho}
    X = U[7:] / rho
    ions, ye = gas.composition(X)
    e = U[5] / rho
    T = gas.invert(rho, U[6], e, ions, ye)
    q["p"], q["g"] = gas.state(rho, T, ions, ye)
    q["re"] = e * rho
    q["c"] = torch.sqrt(q["g"] * q["p"] / rho)
    for k in range(X.shape[0]):
        q["X%d" % k] = X[k]
    return q


def _flatten(q):
    """uflatten on grow(box, 1) from q on grow(box, 4)."""
    p = q["p"]
    flat = None
    for d in range(3):
        at = lambda a, o: _inner(a, 3, d, o)  # noqa: E731
        dp = at(p, 1) - at(p, -1)
        s = torch.where(dp > 0, -1, 1)

        def term(o):
            pr, pl = at(p, 1 + o), at(p, o - 1)
            dp2 = at(p, 2 + o) - at(p, o - 2)
            du = at(q[d], 1 + o) - at(q[d], o - 1)
            delta = pr - pl
            zeta = delta.abs() / dp2.abs().clamp(min=SMALL_PRES)
            z = ((1.0 / (0.85 - 0.75)) * (zeta - 0.75)).clamp(0.0, 1.0)
            hit = (du <= 0) & (delta.abs() > 0.33 * torch.minimum(pr, pl))
            return torch.where(hit, z, torch.zeros_like(z))

        here = term(0)
        side = torch.where(s > 0, term(1), term(-1))
        f = 1.0 - torch.maximum(side, here)
        flat = f if flat is None else torch.minimum(flat, f)
    return flat


def _inner(a, cut, d, off):
    """a without `cut` zones on every side, displaced by `off` zones along d."""
    for e in range(3):
        a = _cut_of(a, e, cut + (off if e == d else 0), a.shape[_ax(e)] - 2 * cut)
    return a


def _parabola(s, d, flat):
    """PPM edges (sm, sp) on grow(box, 1) along d of s on grow(box, 4)."""
    v = [_inner(s, 3, d, o) for o in range(-2, 3)]

    def slope(a, b, c):
        l, r, m = 2.0 * (b - a), 2.0 * (c - b), 0.5 * (c - a)
        return torch.where(l * r > 0, torch.sign(m) * torch.minimum(torch.minimum(m.abs(), l.abs()), r.abs()),
                           torch.zeros_like(m))

    def edge(a, b, da, db):
        e = 0.5 * (b + a) - (1.0 / 6.0) * (db - da)
        return torch.minimum(torch.maximum(e, torch.minimum(a, b)), torch.maximum(a, b))

    sl, sc, sr = slope(*v[0:3]), slope(*v[1:4]), slope(*v[2:5])
    s0 = v[2]
    sm, sp = edge(v[1], s0, sl, sc), edge(s0, v[3], sc, sr)
    sm, sp = flat * sm + (1 - flat) * s0, flat * sp + (1 - flat) * s0
    ext = (sp - s0) * (s0 - sm) <= 0
    right = ~ext & ((sp - s0).abs() >= 2 * (sm - s0).abs())
    left = ~ext & ~right & ((sm - s0).abs() >= 2 * (sp - s0).abs())
    sp2 = torch.where(ext, s0, torch.where(right, 3 * s0 - 2 * sm, sp))
    sm2 = torch.where(ext, s0, torch.where(left, 3 * s0 - 2 * sp, sm))
    return s0, sm2, sp2


def _wave(par, speed, dtdx):
    s0, sm, sp = par
    s6 = 6 * s0 - 3 * (sm + sp)
    g = speed.abs() * dtdx
    up = speed > 0
    Ip = torch.where(up, sp - 0.5 * g * (sp - sm - (1 - 2.0 / 3.0 * g) * s6), sp)
    Im = torch.where(up, sm, sm + 0.5 * g * (sp - sm + (1 - 2.0 / 3.0 * g) * s6))
    return Ip, Im


def _trace(q, flat, d, dtdx, names):
    """Face states (left, right) on the d-faces, transverse directions grown by 1."""
    un, cc = _inner(q[d], 3, d, 0), _inner(q["c"], 3, d, 0)
    speeds = (un - cc, un, un + cc)
    I = {}
    for n in ("r", d, "p", "re"):
        par = _parabola(q[n], d, flat)
        I[n] = [_wave(par, s, dtdx) for s in speeds]
    par = _parabola(q["g"], d, flat)
    gam = [_wave(par, speeds[0], dtdx)[1], _wave(par, speeds[2], dtdx)[0]]
    out = []
    for plus in (True, False):
        k, ref = (1, 0) if plus else (0, 2)
        g = gam[0] if plus else gam[1]
        rr, pr = I["r"][ref][k].clamp(min=SMALL_DENS), I["p"][ref][k].clamp(min=SMALL_PRES)
        ur, er = I[d][ref][k], I["re"][ref][k]
        csq = g * pr / rr
        c = torch.sqrt(csq)
        h = (pr + er) / rr
        am = 0.5 * ((pr - I["p"][0][k]) / (rr * c) - (ur - I[d][0][k])) * rr / c
        ap = 0.5 * ((pr - I["p"][2][k]) / (rr * c) + (ur - I[d][2][k])) * rr / c
        dp0 = pr - I["p"][1][k]
        a0, ae = rr - I["r"][1][k] - dp0 / csq, er - I["re"][1][k] - dp0 * h / csq
        zero = torch.zeros_like(am)
        keep = [(s <= 0) if plus else (s > 0) for s in speeds]
        am, ap = torch.where(keep[0], -am, zero), torch.where(keep[2], -ap, zero)
        a0, ae = torch.where(keep[1], -a0, zero), torch.where(keep[1], -ae, zero)
        st = {"r": (rr + ap + am + a0).clamp(min=SMALL_DENS), d: ur + (ap - am) * c / rr,
              "re": er + (ap + am) * h + ae, "p": (pr + (ap + am) * csq).clamp(min=SMALL_PRES)}
        out.append(st)
    for n in [m for m in (0, 1, 2) if m != d] + names:
        Ip, Im = _wave(_parabola(q[n], d, flat), un, dtdx)
        out[0][n], out[1][n] = Im, Ip
    n = un.shape[_ax(d)] - 1   # faces: zones lo-1 .. hi give left states, lo .. hi+1 right states
    return ({k: _cut_of(v, d, 0, n) for k, v in out[1].items()}, {k: _cut_of(v, d, 1, n) for k, v in out[0].items()})


def _riemann(l, r, gl, gr, cl, cr, d, names):
    """The flux record of compute_flux on d-faces."""
    t1, t2 = [m for m in (0, 1, 2) if m != d]
    rl, rr = l["r"].clamp(min=SMALL_DENS), r["r"].clamp(min=SMALL_DENS)
    pl, pr = l["p"].clamp(min=SMALL_PRES), r["p"].clamp(min=SMALL_PRES)
    ul, ur = l[d], r[d]
    csmall = (SMALL * torch.maximum(cl, cr)).clamp(min=SMALL)
    ws = SMALL_DENS * csmall
    wl = torch.maximum(ws, torch.sqrt((gl * pl * rl).abs()))
    wr = torch.maximum(ws, torch.sqrt((gr * pr * rr).abs()))
    ps = (((wr * pl + wl * pr) + wl * wr * (ul - ur)) / (wl + wr)).clamp(min=SMALL_PRES)
    us = ((wl * ul + wr * ur) + (pl - pr)) / (wl + wr)
    us = torch.where(us.abs() < SMALLU * 0.5 * (ul.abs() + ur.abs()), torch.zeros_like(us), us)
    fp = 0.5 * (1 + torch.sign(us))
    pick = lambda a, b: fp * a + (1 - fp) * b  # noqa: E731
    ro, uo, po, reo, go = pick(rl, rr).clamp(min=SMALL_DENS), pick(ul, ur), pick(pl, pr), pick(l["re"], r["re"]), pick(gl, gr)
    co = torch.maximum(csmall, torch.sqrt((go * po / ro).abs()))
    rs = (ro + (ps - po) / (co * co)).clamp(min=SMALL_DENS)
    es = reo + (ps - po) * ((reo + po) / ro / (co * co))
    cs = torch.maximum(csmall, torch.sqrt((go * ps / rs).abs()))
    sg = torch.where(torch.signbit(us), -1.0, 1.0)
    spout, spin = co - sg * uo, cs - sg * us
    shock = ps > po
    mid = 0.5 * (spin + spout)
    spin, spout = torch.where(shock, mid, spin), torch.where(shock, mid, spout)
    scr = torch.where(spout == spin, SMALL * 0.5 * (cl + cr), spout - spin)
    frac = ((1 + (spout + spin) / scr) * 0.5).clamp(0.0, 1.0)
    take = lambda s, o: torch.where(spin >= 0, s, torch.where(spout < 0, o, frac * s + (1 - frac) * o))  # noqa: E731
    q, u, re = take(rs, ro), take(us, uo), take(es, reo)
    p = take(ps, po).clamp(min=SMALL_PRES)
    v1, v2 = pick(l[t1], r[t1]), pick(l[t2], r[t2])
    F = {"r": q * u, "P": p, "V": u, "re": u * re}
    F[d], F[t1], F[t2] = F["r"] * u, F["r"] * v1, F["r"] * v2
    F["E"] = u * (re + 0.5 * q * (u * u + v1 * v1 + v2 * v2) + p)
    for n in names:
        F[n] = F["r"] * pick(l[n], r[n])
    return F


def _transverse(l, corr, names):
    """A face state less the transverse flux differences `corr` (each times dt/dx)."""
    c = {k: sum(x[k] for x in corr) for k in corr[0]}
    o = {}
    rn = l["r"] - c["r"]
    bad = rn < 0
    keep = lambda new, old: torch.where(bad, old, new)  # noqa: E731
    ke = 0.5 * l["r"] * (l[0] ** 2 + l[1] ** 2 + l[2] ** 2)
    E = keep(l["re"] + ke - c["E"], l["re"] + ke)
    m = {d: keep(l["r"] * l[d] - c[d], l["r"] * l[d]) for d in range(3)}
    for n in names:
        o[n] = (l["r"] * l[n] - c[n]) / rn
    o["r"] = keep(rn, l["r"])
    for d in range(3):
        o[d] = m[d] / o["r"]
    o["re"] = E - 0.5 * (m[0] ** 2 + m[1] ** 2 + m[2] ** 2) / o["r"]
    o["p"] = torch.where(bad, l["p"], (l["p"] - c["p"]).clamp(min=SMALL_PRES))
    return o


def _difference(F, d, f, gam):
    """f times the difference of a flux record across each zone along d, with the pressure equation's term."""
    n = F["r"].shape[_ax(d)] - 1
    a, b = ({k: _cut_of(v, d, o, n) for k, v in F.items()} for o in (1, 0))
    out = {k: f * (a[k] - b[k]) for k in F if k not in ("P", "V", "re")}
    out["p"] = f * (a["P"] * a["V"] - b["P"] * b["V"] + 0.5 * (a["P"] + b["P"]) * (a["V"] - b["V"]) * (gam - 1.0))
    return out


def _trim(v, dirs):
    if isinstance(v, dict):
        return {k: _trim(x, dirs) for k, x in v.items()}
    for d in dirs:
        v = _cut_of(v, d, 1, v.shape[_ax(d)] - 2)
    return v


def _fluxes(gas, Sb, dx, dt):
    """The final face fluxes of a box from its Sborder (grow 4): per direction a record."""
    q = _prim(gas, Sb)
    names = ["X%d" % k for k in range(Sb.shape[0] - 7)]
    flat = _flatten(q)
    g1 = {k: _inner(q[k], 3, 0, 0) for k in ("g", "c")}
    sides = lambda a, d: (_cut_of(a, d, 0, a.shape[_ax(d)] - 1), _cut_of(a, d, 1, a.shape[_ax(d)] - 1))  # noqa: E731
    solve = lambda l, r, d, cut: _riemann(l, r, *sides(_trim(g1["g"], cut), d), *sides(_trim(g1["c"], cut), d), d, names)  # noqa: E731
    tr = [_trace(q, flat, d, dt / dx, names) for d in range(3)]
    F1 = [solve(*tr[d], d, []) for d in range(3)]
    cross = {}
    for b in range(3):
        # the flux differences along b of the zones inside along b
        diff = _difference(F1[b], b, dt / dx / 3.0, _trim(g1["g"], [b]))
        for a in (m for m in range(3) if m != b):
            n = diff["r"].shape[_ax(a)] - 1
            l, r = (_transverse(_trim(tr[a][s], [b]), [{k: _cut_of(v, a, s, n) for k, v in diff.items()}], names)
                    for s in (0, 1))
            cross[a, b] = solve(l, r, a, [b])
    # divu at the nodes
    div = 0.0
    for d in range(3):
        e, f = [m for m in range(3) if m != d]
        for oe in (0, -1):
            for of in (0, -1):
                div = div + 0.25 * (_displaced(q[d], {d: 0, e: oe, f: of}) - _displaced(q[d], {d: -1, e: oe, f: of})) / dx
    Ub = _inner_all(Sb, 3)
    node = {0: ((0, 0, 0), (0, 1, 0), (0, 0, 1), (0, 1, 0)), 1: ((0, 0, 0), (1, 0, 0), (0, 0, 1), (1, 0, 0)),
            2: ((0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0))}
    out = []
    for d in range(3):
        t1, t2 = [m for m in range(3) if m != d]
        gam = _trim(g1["g"], [t1, t2])
        corr = [_difference(cross[t1, t2], t1, 0.5 * dt / dx, gam), _difference(cross[t2, t1], t2, 0.5 * dt / dx, gam)]
        n = gam.shape[_ax(d)] - 1
        l, r = (_transverse(_trim(tr[d][s], [t1, t2]), [{k: _cut_of(v, d, s, n) for k, v in c.items()} for c in corr], names)
                for s in (0, 1))
        F = solve(l, r, d, [t1, t2])
        # nodes of the faces: index f (low corner) in lo .. hi+1 along d, lo .. hi across
        size = [g1["g"].shape[_ax(m)] - 2 + (m == d) for m in range(3)]
        ds = 0.0
        for o in node[d]:
            v = div
            for m in range(3):
                v = _cut_of(v, m, 1 + o[m], size[m])
            ds = ds + v
        av = dx * 0.1 * (0.25 * ds).clamp(max=0.0)
        keys = ["r", 0, 1, 2, "E", "re", None] + names
        for k, name in enumerate(keys):
            if name is None:
                continue
            v = Ub[k]
            for m in (t1, t2):
                v = _cut_of(v, m, 1, v.shape[_ax(m)] - 2)
            F[name] = F[name] + av * (_cut_of(v, d, 1, n) - _cut_of(v, d, 0, n))
        total = sum(F[k] for k in names)
        fac = torch.where(total != 0, F["r"] / total, torch.ones_like(total))
        for k in names:
            F[k] = F[k] * fac
        out.append((F, keys))
    return out


def _inner_all(U, cut):
    return torch.stack([_inner(c, cut, 0, 0) for c in U])


def _displaced(a, off):
    for m in range(3):
        a = _cut_of(a, m, 3 + off[m], a.shape[_ax(m)] - 6)
    return a


def _source(fl, dx):
    """fill_hydro_source from the final fluxes."""
    keys = fl[0][1]
    S = []
    for name in keys:
        if name is None:
            S.append(torch.zeros_like(S[0]))
            continue
        s = 0.0
        for d in range(3):
            f = fl[d][0]
            lo, hi = (_cut_of(f[name], d, o, f[name].shape[_ax(d)] - 1) for o in (0, 1))
            s = s + (lo - hi) / dx
            if name == "re":
                P, V = ([_cut_of(f[k], d, o, f[k].shape[_ax(d)] - 1) for o in (0, 1)] for k in ("P", "V"))
                s = s - 0.5 * (P[0] + P[1]) * (V[1] - V[0]) / dx
        S.append(s)
    return torch.stack(S)


def _initial(gas, inst):
    """initdata: the energy of the subzones inside the blast, the ambient gas elsewhere."""
    p = inst["problem"]
    dims = [h + 1 for h in inst["dom_hi"]]
    dx = (inst["probhi"][0] - inst["problo"][0]) / dims[0]
    X = torch.tensor((list(p["X"]) + [0.0] * len(gas.A))[:len(gas.A)], dtype=torch.float64, device=DEVICE)
    one = lambda v: torch.tensor([v], dtype=torch.float64, device=DEVICE)  # noqa: E731
    if p["ambient_from_T"]:
        ions, ye = gas.composition(X[:, None])
        T = one(p["T_ambient"])
    else:   # the reference inverts the pressure with the first species' composition
        ions, ye = 1.0 / gas.A[:1], gas.Z[:1] / gas.A[:1]
        T = gas.invert(one(p["dens_ambient"]), one(1e4), one(p["p_ambient"]), ions, ye, "p")
    e_amb = float(gas.eval(one(p["dens_ambient"]), T, ions, ye).e)
    r = p["r_init"]
    e_exp = p["exp_energy"] / (4.0 / 3.0 * math.pi * r ** 3) / p["dens_ambient"]
    sub = [(torch.arange(n, dtype=torch.float64, device=DEVICE)[:, None] + (torch.arange(10, device=DEVICE) + 0.5) / 10 - 0.5 * n) ** 2
           for n in dims]
    rr = (r / dx) ** 2
    inside = torch.zeros(dims[::-1], dtype=torch.float64, device=DEVICE)
    for a in range(10):
        for b in range(10):
            for c in range(10):
                inside += (sub[2][:, None, None, a] + sub[1][None, :, None, b] + sub[0][None, None, :, c]) <= rr
    e = (inside * e_exp + (1000.0 - inside) * e_amb) / 1000.0
    rho = torch.full_like(e, p["dens_ambient"])
    if p.get("pert") is not None:
        g = torch.from_numpy(np.ascontiguousarray(p["pert"].transpose(2, 1, 0))).to(DEVICE)
        rho = p["dens_ambient"] * (1.0 + p["pert_amp"] * g)
    zero = torch.zeros_like(e)
    return torch.stack([rho, zero, zero, zero, rho * e, rho * e, torch.full_like(e, p["T_init"])] + [x * rho for x in X]), dx


class _Level:
    def __init__(self, gas, inst):
        self.gas, self.inst = gas, inst
        self.U, self.dx = _initial(gas, inst)
        self.dt = 0.01 * 0.5 * _sound_dt(gas, self.U, self.dx)

    def step(self):
        U = _clean(self.gas, self.U)
        Sb = _grow(_clean(self.gas, U), self.inst["bc"])
        new = U + self.dt * _source(_fluxes(self.gas, Sb, self.dx, self.dt), self.dx)
        self.U = _clean(self.gas, _clean(self.gas, new))
        self.dt = min(0.5 * _sound_dt(self.gas, self.U, self.dx), 1.1 * self.dt)

    def boxes(self):
        out = []
        for lo, hi in self.inst["boxes"]:
            out.append(self.U[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1].reshape(-1))
        return out


def exact(case, seed):
    # the gradient is a sum over limiter branches, many of them on ties of the uniform ambient
    # gas where a one-sided derivative is as right as the other: no value to hold it to
    if case["kind"] == "adjoint":
        return None
    gas = _Gas(case.get("ns", 2))
    if case["kind"] == "box":
        U, dx, dt = _box_inputs(case, seed)
        fl = _fluxes(gas, _clean(gas, U), dx, dt)
        area = dx * dx
        flux = [torch.stack([dt * area * (f[k] if k is not None else torch.zeros_like(f["r"])) for k in keys]) for f, keys in fl]
        return dict(source=_source(fl, dx), fluxes=flux)
    levels = [_Level(gas, i) for i in _instances(case, seed)]
    if case["kind"] == "host":
        lev = levels[0]
        start = lev.U
        lev.step()           # the call that prepare() makes; its time step goes on, the state is uploaded again
        lev.U = start
        for _ in range(case["steps"]):
            lev.step()
        return torch.cat(lev.boxes()).cpu()
    flat = []
    for lev in levels:
        for _ in range(WARM_STEPS + case["steps"]):
            lev.step()
        flat += lev.boxes()
    if len(levels) == 1 and len(levels[0].inst["boxes"]) == 1:
        return list(flat[0].reshape(levels[0].U.shape[0], -1))
    return torch.cat(flat)
