"""Cube planning with rows in uv order against row order.

A cube large enough for the uv order (262,144 rows and 2^24 samples) is
gridded in one call and, channel group by channel group, in calls too small
for it.  Planning decides each sample by itself and unit weights make every
density sum exact, so counts are equal and sums of weights agree to FP64
rounding (1e-12); the grids sum the same float32 terms in another order
(1e-5 of each channel's peak, the bound of the other cube tests).  Rows come
in random order, some share a point, one in a hundred lies outside the grid,
and some are zero or not finite.
"""
import numpy as np
import pytest

import casars_cuda as cc

from gpu_common import peak_norm_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,rows", [("natural", 2 ** 18), ("briggs", 2 ** 18 + 77)])
def test_uv_order_equals_row_order(mode, rows):
    ctx = cc.Context(0)
    image, channels, cell = 96, 64, 2.0e-5
    gg = cc.StandardGridder(ctx, cc.ImageGeometry(image, image, cell, cell), 32)
    gx, _ = gg.grid_shape()
    du = gg.info.du
    rng = np.random.default_rng(7)
    ls = np.linspace(1.0, 1.3, channels)
    u, v = (rng.normal(0.0, 0.12 * gx, rows) * du for _ in range(2))
    u[::3] = u[0]
    v[::3] = v[0]
    u[1::100] = 3.0 * gx * du
    u[5], v[6], u[7], v[8] = 0.0, 0.0, np.nan, np.inf
    vis = (rng.normal(size=(channels, rows)) + 1j * rng.normal(size=(channels, rows)))
    vis = vis.astype(np.complex64)
    flags = rng.random((channels, rows)) < 0.1
    whole = cc.cube_grid_dirty(gg, cc.CubeBatch(u, v, ls, vis, None, flags), mode, 0.5)
    for c in range(0, channels, 16):
        part = cc.cube_grid_dirty(
            gg, cc.CubeBatch(u, v, ls[c:c + 4], vis[c:c + 4], None, flags[c:c + 4]), mode, 0.5)
        for k in range(4):
            a, b = whole[2][c + k], part[2][k]
            assert a.gridded_samples == b.gridded_samples > 0
            assert a.skipped_samples == b.skipped_samples
            assert abs(a.normalization_sumwt - b.normalization_sumwt) <= \
                1e-12 * b.normalization_sumwt
            assert peak_norm_err(whole[0][c + k], part[0][k]) <= 1e-5
            assert peak_norm_err(whole[1][c + k], part[1][k]) <= 1e-5
    ctx.close()
