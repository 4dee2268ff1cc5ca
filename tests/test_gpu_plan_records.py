"""Sort and records at the sizes where their tiles, ranges and chains change.

The batches hold runs of equal keys that begin and end on, before and after
the boundaries of a warp's range (128 samples), a tile (1024) and a sort tile
(1024 and 4096), runs longer than several tiles, and samples that do not grid.
Counts, records and sums of weights are exact; grids and predictions are held
to the oracle's peak times 1e-5, as elsewhere.
"""
import numpy as np
import pytest

import casars_cuda as cc
from oracle import oracle as O

from gpu_common import peak_norm_err

pytestmark = pytest.mark.gpu
NX, CELL = 96, 2e-5


@pytest.fixture(scope="module")
def grid():
    ctx = cc.Context(0)
    gg = cc.StandardGridder(ctx, cc.ImageGeometry(NX, NX, CELL, CELL))
    og = O.StdGridder(O.Geometry(NX, NX, CELL, CELL))
    yield ctx, gg, og
    ctx.close()


def batch(n, runs, seed):
    """n samples of which `runs` lists the lengths of equal-coordinate runs;
    the rest are single samples, a few of them off the grid."""
    rng = np.random.default_rng(seed)
    half = 0.4 / CELL
    u, v = rng.uniform(-half, half, n), rng.uniform(-half, half, n)
    at = 0
    for length in runs:
        u[at:at + length] = rng.uniform(-half, half)
        v[at:at + length] = rng.uniform(-half, half)
        at += length
    u[rng.integers(0, n, max(n // 50, 1))] = 0.9 / CELL      # outside
    order = rng.permutation(n)
    wt = rng.integers(1, 9, n).astype(np.float32)
    wt[::97] = 0.0
    vis = (rng.normal(size=n) + 1j * rng.normal(size=n)).astype(np.complex64)
    return u[order], v[order], wt, vis


CASES = [(1, []), (2, [2]), (31, [31]), (127, [64, 63]), (128, [128]), (129, [128]),
         (1023, [500]), (1024, [127, 129]), (1025, [1025]), (4095, [1024, 1025, 1023]),
         (4096, [4096]), (4097, [3000, 300, 30, 3]), (20000, [9000, 129, 128, 127, 1]),
         (1 << 19, [200000, 4096, 1024]), ((1 << 19) - 1, [100000] * 3)]


@pytest.mark.parametrize("n,runs", CASES)
def test_records_and_grids(grid, n, runs):
    ctx, gg, og = grid
    u, v, wt, vis = batch(n, runs, n)
    b = cc.VisibilityBatch(u, v, vis, wt)
    psf, dirty, sums = cc.grid_dirty(gg, b)
    po, do, acc = og.grid_dirty(u, v, wt, vis, threads=8)
    assert (sums.gridded_samples, sums.skipped_samples) == (acc.gridded, acc.skipped)
    x0, y0, rx, ry = og.plan_many(u, v)
    ok = (x0 >= 0) & (wt > 0)
    assert sums.unique_records == len(set(zip(x0[ok], y0[ok], rx[ok], ry[ok])))
    assert sums.taps == 49 * sums.unique_records
    assert sums.normalization_sumwt == float(wt[ok].sum(dtype=np.float64))
    if not ok.any():
        return
    assert peak_norm_err(psf, po) <= 1e-5
    assert peak_norm_err(dirty, do) <= 1e-5
    # a kept plan gives the same records, and every sample its prediction
    p = cc.Plan(gg, b)
    assert p.sums.unique_records == sums.unique_records
    rng = np.random.default_rng(1)
    model = (rng.normal(size=po.shape) + 1j * rng.normal(size=po.shape)).astype(np.complex64)
    pred = p.degrid(model)
    ref = og.degrid(model, u, v)
    assert peak_norm_err(pred[ok], ref[ok]) <= 1e-5
    assert not np.any(pred[x0 < 0])
    res = p.grid_residual(model)
    r = np.where(np.isfinite(vis), vis - pred, 0).astype(np.complex64)
    _, ro, _ = og.grid_dirty(u, v, wt, r, threads=8)
    assert peak_norm_err(res, ro) <= 1e-5
