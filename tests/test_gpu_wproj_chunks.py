"""W-projection work items at the edges of their sizes.

A batch is gridded with the item size that its number of
samples gives and with the largest (a context with an allocation limit takes
that one).  Each record is summed once either way, so the grids agree within
the rounding of float32 sums in another order (1e-5 of the peak, the bound of
the other W-projection tests) and the counts are equal.  The sizes are just
below and at each change of the rule; the smallest has one sample.
"""
import numpy as np
import pytest

import casars_cuda as cc
from oracle import oracle as O

from gpu_common import arcsec, peak_norm_err, random_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 2 ** 17 - 1, 2 ** 17, 2 ** 19, 2 ** 21])
@pytest.mark.parametrize("law", [(3, 5), (4, 20)])
def test_item_sizes_agree(n, law):
    ctx = cc.Context(0)
    nx, cell, wmax = 200, arcsec(20.0), 2000.0
    gg = cc.StandardGridder(ctx, cc.ImageGeometry(nx, nx, cell, cell), 100)
    gw = cc.WProjector(gg, wmax, planes=8, sampling=4, support_law=law)
    og = O.StdGridder(O.Geometry(nx, nx, cell, cell), 100)
    rng = np.random.default_rng(n)
    u, v, w, wt, vis = random_batch(rng, n, og.gnx, og.du, margin=law[1] + 2, w_max=wmax)
    batch = cc.VisibilityBatch(u, v, vis, wt, w)
    out = []
    for limit in (0, 1 << 40):
        ctx.set_alloc_limit(limit)
        out.append(cc.grid_dirty(gg, batch, gw))
    (p0, d0, s0), (p1, d1, s1) = out
    assert s0.gridded_samples == s1.gridded_samples > 0
    assert peak_norm_err(p0, p1) <= 1e-5
    assert peak_norm_err(d0, d1) <= 1e-5
    ctx.close()
