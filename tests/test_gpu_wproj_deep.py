"""W-projection gridding of small batches against the general path.

Batches below 2^17 samples take the form that keeps eight records' kernel
values in flight.  The same samples followed by samples of zero weight, up to
2^17, give the same records and take the general form: the grids agree within
the rounding of float32 sums in another order (1e-5 of the peak, the bound of
the other W-projection tests) and the counts are equal.  The sizes leave one,
eight, nine and many records in a warp's batch; the largest is the last below
the change.  (test_residual_refresh_matches_oracle of test_gpu_wproj.py holds
the residual form to the oracle.)
"""
import numpy as np
import pytest

import casars_cuda as cc
from oracle import oracle as O

from gpu_common import arcsec, peak_norm_err, random_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8, 9, 33, 3000, 2 ** 17 - 1])
@pytest.mark.parametrize("law", [(3, 5), (4, 20)])
def test_small_batches_equal_the_general_form(n, law):
    ctx = cc.Context(0)
    nx, cell, wmax = 200, arcsec(20.0), 2000.0
    gg = cc.StandardGridder(ctx, cc.ImageGeometry(nx, nx, cell, cell), 100)
    gw = cc.WProjector(gg, wmax, planes=8, sampling=4, support_law=law)
    og = O.StdGridder(O.Geometry(nx, nx, cell, cell), 100)
    rng = np.random.default_rng(n)
    u, v, w, wt, vis = random_batch(rng, n, og.gnx, og.du, margin=law[1] + 2, w_max=wmax)
    pad = 2 ** 17 - n
    batch = cc.VisibilityBatch(u, v, vis, wt, w)
    padded = cc.VisibilityBatch(*(np.concatenate([a, np.zeros(pad, a.dtype)])
                                  for a in (u, v, vis, wt, w)))
    p0, d0, s0 = cc.grid_dirty(gg, batch, gw)
    p1, d1, s1 = cc.grid_dirty(gg, padded, gw)
    assert s0.gridded_samples == s1.gridded_samples > 0
    assert peak_norm_err(p0, p1) <= 1e-5
    assert peak_norm_err(d0, d1) <= 1e-5
    ctx.close()
