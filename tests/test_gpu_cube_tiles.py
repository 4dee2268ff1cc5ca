"""Cube gridding by runs at the edges of its tiles.

Samples start at chosen cells of a 32 x 32 tile: its corners and the cells
around x, y = 26, from which a 7 x 7 footprint reaches the next tile, in a
tile of the middle and in the grid's last, partly covered one.  The runs have
lengths around the four records that a warp sums at once and the 32 that it
decodes at once.  The grids agree with the FP64 oracle within the bound of a
float32 sum of n terms (n + 8 roundings: the additions, the two tap products,
the exchange between lanes and the tile), relative to the largest cell; n is
the number of samples, more than reach any one cell.
"""
import numpy as np
import pytest

import casars_cuda as cc
from oracle import oracle as O

pytestmark = pytest.mark.gpu

OS = 16
IMAGE = 101


@pytest.mark.parametrize("lengths", [(1,), (3,), (4,), (5,), (31,), (33,), (1, 2, 7, 40, 3)])
def test_runs_at_tile_edges(lengths):
    ctx = cc.Context(0)
    cell = 2.0e-5
    gg = cc.StandardGridder(ctx, cc.ImageGeometry(IMAGE, IMAGE, cell, cell), OS)
    gx, gy = gg.grid_shape()
    og = O.StdGridder(O.Geometry(IMAGE, IMAGE, cell, cell), OS)
    du, dv = gg.info.du, gg.info.dv
    edges = [32 + k for k in (0, 1, 25, 26, 27, 31)]
    starts = [(x, y) for x in edges for y in edges]
    starts += [(x, y) for x in (0, 5, gx - 9, gx - 8) for y in (0, 26, gy - 9, gy - 8)]
    rng = np.random.default_rng(5)
    sx = np.concatenate([np.repeat([s[0]], lengths[i % len(lengths)]) for i, s in enumerate(starts)])
    sy = np.concatenate([np.repeat([s[1]], lengths[i % len(lengths)]) for i, s in enumerate(starts)])
    order = rng.permutation(len(sx))
    sx, sy = sx[order], sy[order]
    u = (sx + 3 + rng.uniform(-0.4, 0.4, len(sx)) - gx / 2) * du
    v = -(sy + 3 + rng.uniform(-0.4, 0.4, len(sy)) - gy / 2) * dv
    ox, oy, _, _ = og.plan_many(u, v)
    np.testing.assert_array_equal(ox, sx)
    np.testing.assert_array_equal(oy, sy)
    n = len(u)
    vis = (rng.normal(size=(1, n)) + 1j * rng.normal(size=(1, n))).astype(np.complex64)
    wt = rng.uniform(0.5, 2.0, (1, n)).astype(np.float32)
    batch = cc.CubeBatch(u, v, np.ones(1), vis, wt, np.zeros((1, n), bool))
    psf, dirty, sums = cc.cube_grid_dirty(gg, batch, "natural", 0.0)
    p_o, d_o, acc = og.grid_dirty(u, v, wt[0], vis[0])
    a_o, _, _ = og.grid_dirty(u, v, wt[0] * np.abs(vis[0]), vis[0])
    tol = (n + 8) * 2.0 ** -24
    assert sums[0].gridded_samples == acc.gridded == n
    assert np.abs(psf[0] - p_o.real).max() <= tol * np.abs(p_o).max()
    assert np.abs(dirty[0] - d_o).max() <= 2 * tol * np.abs(a_o).max()
    assert not np.any(psf[0][p_o.real == 0.0])
    ctx.close()
