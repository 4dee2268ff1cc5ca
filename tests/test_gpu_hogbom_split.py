"""The register-resident Hogbom loop at the edges of its split.

Each shape sits where the split changes: one block, a partly filled column
group, odd sides, the smallest image of each register height, and images that
do not fit the registers (the global-memory loop).  Every decision and image
is bit-exact against the oracle, with ties across blocks, NaN and infinite
pixels, a mask, and the plane rules.
"""
import numpy as np
import pytest

import casars_cuda as cc
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = cc.Context(0)
    yield c
    c.close()


def inputs(nx, ny, masked):
    rng = np.random.default_rng(nx * 7919 + ny)
    x = np.arange(nx)[:, None] - nx // 2
    y = np.arange(ny)[None, :] - ny // 2
    psf = (np.exp(-(x * x + y * y) / 18.0) + 0.02 * rng.normal(size=(nx, ny))).astype(np.float32)
    psf[nx // 2, ny // 2] = 1.0
    res = (0.01 * rng.normal(size=(nx, ny))).astype(np.float32)
    for _ in range(12):
        res[rng.integers(0, nx), rng.integers(0, ny)] += rng.uniform(0.1, 1.0)
    res[0, 0] = -2.0
    res[nx - 1, ny - 1] = 2.0       # a tie with the first pixel, in the last block
    mask = (rng.uniform(size=(nx, ny)) > 0.05).astype(np.uint8) if masked else None
    return res, psf, mask


# 152 SMs hold 2432 warps: 32 columns by 4, 8, 16, 32, 56 or 96 rows each
SHAPES = [(1, 1), (3, 33), (4, 32), (5, 31), (200, 150), (129, 257), (601, 333), (700, 1001),
          (1400, 1400), (1600, 1500), (2048, 2048), (2100, 2050), (3, 80000), (3000, 2700)]


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_split_bit_exact(ctx, shape, masked):
    res, psf, mask = inputs(*shape, masked)
    n = 40 if shape[0] * shape[1] > 1 << 20 else 150
    ref = O.hogbom(res, psf, 0.15, n, threshold=0.004, mask=mask)
    out = cc.run_hogbom_minor_cycle(ctx, np.zeros_like(res), res, psf, 0.15, n, threshold=0.004,
                                    mask=mask)
    assert out.actual_updates == ref["actual"]
    np.testing.assert_array_equal(out.positions[:, 0], ref["x"])
    np.testing.assert_array_equal(out.positions[:, 1], ref["y"])
    np.testing.assert_array_equal(out.fluxes, ref["flux"])
    np.testing.assert_array_equal(out.residual, ref["residual"])
    np.testing.assert_array_equal(out.model, ref["model"])


def test_nan_never_wins_and_infinity_does(ctx):
    res, psf, _ = inputs(130, 90, False)
    res[7, 11] = np.nan
    ref = O.hogbom(res, psf, 0.1, 50)
    out = cc.run_hogbom_minor_cycle(ctx, np.zeros_like(res), res, psf, 0.1, 50)
    np.testing.assert_array_equal(out.residual, ref["residual"])
    assert not any((out.positions == (7, 11)).all(1))
    res[100, 80] = np.inf
    out = cc.run_hogbom_minor_cycle(ctx, np.zeros_like(res), res, psf, 0.1, 0)
    assert tuple(out.positions[0]) == (100, 80) and np.isinf(out.peaks[0])
    # under the plane rules only finite values are candidates
    out = cc.hogbom_plane_minor_cycle(ctx, np.zeros_like(res), res, psf, 0.1, 0, 0.0, 0.0)
    assert np.isfinite(out.peaks[0]) and abs(out.peaks[0]) == 2.0


def test_zero_budget_and_no_candidate_leave_the_images(ctx):
    res, psf, _ = inputs(70, 65, False)
    out = cc.run_hogbom_minor_cycle(ctx, np.zeros_like(res), res, psf, 0.1, 0, inclusive=False)
    assert out.actual_updates == 0 and out.stop_reason is None
    np.testing.assert_array_equal(out.residual, res)
    out = cc.run_hogbom_minor_cycle(ctx, np.zeros_like(res), res, psf, 0.1, 5,
                                    mask=np.zeros(res.shape, np.uint8))
    assert out.actual_updates == 0 and out.stop_reason == "NoCleanablePixels"
    np.testing.assert_array_equal(out.residual, res)
