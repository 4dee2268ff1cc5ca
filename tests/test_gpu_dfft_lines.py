"""The float-pair transforms over the kinds of line they handle differently.

Line lengths of one stage (2, 4), every power of two that changes the
shared-memory layout (2, 4, 8 and 16 dividing the length, below and from 1024
points on), a first radix of 2 and of 4, lines longer and shorter than a
block's threads, unequal sides, and odd image sides (a last column unpaired).
The reference is cuFFT in FP64; both round the same value to float32, so they
may differ by four float32 ulps of it (plus 1e-10 of the peak), as in
test_gpu_dfft.py.
"""
import numpy as np
import pytest

import casars_cuda as cc

pytestmark = pytest.mark.gpu

# image sides -> line lengths: 1 -> 2, 3 -> 4, 5 -> 6, 7 -> 8, 8 -> 10, 75 -> 90,
# 100 -> 120, 250 -> 300, 512 -> 640, 750 -> 900, 853 -> 1024, 1041 -> 1250,
# 1000 -> 1200, 1250 -> 1500, 1333 -> 1600, 1667 -> 2000
SIDES = [(1, 1), (1, 3), (3, 5), (8, 7), (75, 100), (100, 75), (250, 512), (853, 8), (7, 1041),
         (1000, 750), (1250, 1333), (1667, 250)]


@pytest.fixture(scope="module")
def ctx():
    c = cc.Context(0)
    yield c
    c.close()


def close(a, b):
    a, b = np.asarray(a), np.asarray(b)
    if np.iscomplexobj(b):
        return close(a.real, b.real) and close(a.imag, b.imag)
    bound = 4 * np.spacing(np.abs(b).astype(np.float32)) + 1e-10 * float(np.max(np.abs(b)))
    return bool(np.all(np.abs(a - b) <= bound))


@pytest.mark.parametrize("wproj", [False, True])
@pytest.mark.parametrize("nx,ny", SIDES)
def test_both_directions(ctx, nx, ny, wproj):
    if wproj and min(nx, ny) < 75:
        pytest.skip("no W kernels on so small a grid")
    rng = np.random.default_rng(1000 * nx + ny)
    gg = cc.StandardGridder(ctx, cc.ImageGeometry(nx, ny, 2e-5, 3e-5))
    gw = cc.WProjector(gg, 300.0, planes=2, sampling=2, support_law=(3, 4)) if wproj else None
    shape = gg.grid_shape()
    grid = (rng.normal(size=shape) + 1j * rng.normal(size=shape)).astype(np.complex64)
    model = rng.normal(size=(nx, ny)).astype(np.float32)

    def both():
        return (cc.grid_to_image(gg, grid, 0.5 * shape[0], gw), cc.image_to_grid(gg, model, gw))

    ctx.set_image_fft_engine("cufft")
    try:
        ref = both()
    finally:
        ctx.set_image_fft_engine("auto")
    got = both()
    assert close(got[0], ref[0])
    assert close(got[1], ref[1])


@pytest.mark.parametrize("nx,ny", [(75, 100), (101, 96), (512, 250)])
def test_pair_of_images(ctx, nx, ny):
    """The PSF and residual of a dirty image go through one pair of launches:
    the PSF's peak is one, and both agree with the two images transformed
    from the call's grids one at a time."""
    rng = np.random.default_rng(nx)
    cx, cy = 2e-5, 3e-5
    gg = cc.StandardGridder(ctx, cc.ImageGeometry(nx, ny, cx, cy))
    n = 3000
    u, v = rng.uniform(-0.3 / cx, 0.3 / cx, n), rng.uniform(-0.3 / cy, 0.3 / cy, n)
    vis = (rng.normal(size=n) + 1j * rng.normal(size=n)).astype(np.complex64)
    b = cc.VisibilityBatch(u, v, vis, np.ones(n, np.float32))
    psf, res, state, sums = cc.dirty_image(gg, b)
    assert float(np.max(np.abs(psf))) == 1.0
    gp, gd, _ = cc.grid_dirty(gg, b)
    # the two calls add the grids in different orders: 1e-5 of the peak
    for img, grid in ((psf, gp), (res, gd)):
        one = cc.grid_to_image(gg, grid, 1.0 / sums.normalization_sumwt) / state.psf_peak
        assert float(np.max(np.abs(one - img))) <= 1e-5 * float(np.max(np.abs(img)))
