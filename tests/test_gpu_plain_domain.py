"""A domain whose grown region has more than 2^31 points, cut into boxes: the per-box sequences number a box's points
only, so they take it (the batched and persistent step, which number the domain's, refuse it).  A column of 1 x 1 x
26,600,000 zones, 81 ghost-grown points a zone, 155 GB of Sborder; the two boxes beside the blast after one step must
equal, bit for bit, those of a short column with the same two boxes, since nothing else has moved and every coordinate
is exact in both."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTH = 100_000   # zones of a box


def column(pkg, nbox):
    n = nbox * LENGTH
    boxes = [((0, 0, b * LENGTH), (0, 0, (b + 1) * LENGTH - 1)) for b in range(nbox)]
    return dict(dom_lo=(0, 0, 0), dom_hi=(0, 0, n - 1), problo=(0.0, 0.0, 0.0), probhi=(1.0, 1.0, float(n)), bc=1,
                boxes=boxes, n=1, problem=pkg.configs.problem(r_init=4.0))


def test_domain_beyond_32_bits(pkg, table):
    import torch

    L = pkg.castro.init(*pkg.configs.NET2, table)
    long, short = column(pkg, 266), column(pkg, 2)
    with pytest.raises(Exception, match="2\\^31"):
        pkg.make_sim(L, dict(instances=[long]), pkg.castro.MODE_BATCHED)
    L.castro_clear_error()
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 168e9:
        pytest.skip("needs 168 GB of free device memory")
    near = []
    for inst, first in ((long, 132), (short, 0)):
        sim = pkg.make_sim(L, dict(instances=[inst]), pkg.castro.MODE_PLAIN_BOX)
        sim.init_data()
        sim.step(1)
        states = sim.box_states()[0][first:first + 2]
        sim.close()
        near.append(np.concatenate([np.asarray(x).ravel() for x in states]))
    assert np.isfinite(near[1]).all() and np.ptp(near[1][:LENGTH]) > 0
    np.testing.assert_array_equal(near[0], near[1])
