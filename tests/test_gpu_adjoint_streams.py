"""The gradient's three streams against the same launches in one order.  A child process with CUDA_LAUNCH_BLOCKING=1
finishes every kernel before the next is launched, whatever stream it is on; the gradients of this process, where the
three directions of a stage overlap, must agree with it: 2 species whole and by slabs, a window of the last steps, 13
species, and two handles used in turn.

Scatter sums by FP64 atomics have no fixed order in either process, so repeats differ by rounding that the reverse sweep
amplifies.  The bound is that spread itself: at most 8 times what four repeats of the ordered process differ by (four
draws show the typical distance, not the largest), or 1e-13 of the largest value.  J has no atomics and must be equal."""
from __future__ import annotations

import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = ["whole", "slabs", "window", "13 species"]


def gradients(pkg, table, case, handles=1, repeats=1):
    """[(J, {name: array})] of `repeats` reverse sweeps of each handle, the handles' calls taken in turn."""
    K = pkg.castro
    if case == "13 species":
        cfg, steps, ckpt, kw, net = pkg.configs.reference(scale=8), 4, 2, {}, pkg.configs.NET13
    else:
        cfg, steps, ckpt, net = pkg.configs.adjoint64(scale=2, steps=6), 6, 3, pkg.configs.NET2
        kw = dict(whole={}, slabs=dict(slab_nz=8), window=dict(first_step=3))[case]
    L = K.init(*net, table)
    inst = cfg["instances"][0]
    p = inst["problem"]
    runs = [pkg.adjoint.SedovAdjoint(L, inst, steps, ckpt, **kw) for _ in range(handles)]
    J = [r.forward(p["exp_energy"] * (1.0 + 0.2 * m), p["dens_ambient"]) for m, r in enumerate(runs)]
    out = [[] for _ in runs]
    for _ in range(repeats):
        for m, r in enumerate(runs):
            dE, dR, dP = r.backward()
            out[m].append((J[m], dict(dE=np.array([dE]), dR=np.array([dR]), dP=dP.cpu().numpy(),
                                      dV=r.state_adjoint().cpu().numpy())))
    for r in runs:
        r.close()
    return out


def distance(a, b):
    return {k: float(np.abs(a[k] - b[k]).max() / max(np.abs(b[k]).max(), 1e-300)) for k in a}


@pytest.fixture(scope="module")
def ordered(tmp_path_factory):
    """Per case, per handle: J and four repeats of the gradient with one kernel at a time."""
    path = tmp_path_factory.mktemp("ordered") / "g.npz"
    env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1")
    subprocess.run([sys.executable, os.path.abspath(__file__), str(path)], check=True, env=env, timeout=600)
    z = np.load(path)

    def get(case, handle):
        return float(z[f"{case}/{handle}/J"]), [{k: z[f"{case}/{handle}/{m}/{k}"] for k in ("dE", "dR", "dP", "dV")}
                                                for m in range(4)]
    return get


@pytest.mark.parametrize("case", CASES)
def test_streams_match_one_order(pkg, table, ordered, case):
    for handle, runs in enumerate(gradients(pkg, table, case, handles=2, repeats=2)):
        J0, ref = ordered(case, handle)
        pairs = [distance(a, b) for i, a in enumerate(ref) for b in ref[:i]]
        spread = {k: max(p[k] for p in pairs) for k in pairs[0]}
        assert np.abs(ref[0]["dV"]).max() > 0
        for J, g in runs:
            assert J == J0
            d = distance(g, ref[0])
            for k in d:
                assert d[k] <= max(8.0 * spread[k], 1e-13), (handle, k, d[k], spread[k])


if __name__ == "__main__":
    sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
    from conftest import load_package

    pk = load_package()
    tab = pk.helm_table.ensure_table()
    save = {}
    for c in CASES:
        for h, res in enumerate(gradients(pk, tab, c, handles=2, repeats=4)):
            save[f"{c}/{h}/J"] = np.array(res[0][0])
            for m, (_, g) in enumerate(res):
                for k, v in g.items():
                    save[f"{c}/{h}/{m}/{k}"] = v
    np.savez(sys.argv[1], **save)
