"""Weight density collected in a table per block against the oracle.

Batches just below and above the size from which samples are collected by
cell (2^17), and one of several blocks per multiprocessor: successive samples
of some baselines share cells, others are scattered, on cell boundaries, on
the axes and in the first and last cells, where a cell's mirror is not the
reflected one.  Unit weights make every density sum exact, so the weights
equal the oracle's bit for bit, in both cell conventions.
"""
import numpy as np
import pytest

import casars_cuda as cc
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2 ** 17 - 1, 2 ** 17, 2 ** 20 + 5])
@pytest.mark.parametrize("image", [255, 512])
@pytest.mark.parametrize("convention", [0, 1])
def test_table_equals_direct_adds(n, image, convention):
    ctx = cc.Context(0)
    cell = 3.0e-5
    gg = cc.StandardGridder(ctx, cc.ImageGeometry(image, image, cell, cell), 16)
    rng = np.random.default_rng(n + image)
    unit = 1.0 / (image * cell)         # wavelengths a cell
    half = image / 2.0
    base = rng.uniform(-0.45 * image, 0.45 * image, (2, 97))
    t = np.arange(n) // 97
    x, y = (b[np.arange(n) % 97] + 0.01 * (t % 50) for b in base)
    k = rng.integers(0, n, n // 4)
    x[k], y[k] = rng.uniform(-half - 2, half + 2, (2, len(k)))
    k = rng.integers(0, n, n // 8)
    x[k] = rng.integers(-image // 2 - 1, image // 2 + 2, len(k))
    y[k] = rng.integers(-image // 2 - 1, image // 2 + 2, len(k)) + 0.5
    x[:100], y[50:150] = 0.0, 0.0
    u, v = x * unit, y * unit
    wt = np.ones(n, np.float32)
    wt[::501] = 0.0
    vis = np.zeros(n, np.complex64)
    for mode in ("uniform", "briggs"):
        got, f2 = cc.apply_weighting(gg, cc.VisibilityBatch(u, v, vis, wt), mode, 0.5,
                                     per_plane=convention == 1)
        want, f2_o, _ = O.apply_weighting(O.Geometry(image, image, cell, cell), u, v, wt, mode,
                                          0.5, convention=convention)
        np.testing.assert_array_equal(got, want)
    ctx.close()
