"""Row preparation at the edges of its tiles (2048 samples) and look-back.

Sample counts around one, two and 33 tiles (a look-back step covers 32),
everything flagged, nothing flagged, odd channel counts, and coordinates whose
float32 rounding is a tie, subnormal, overflowing or infinite.  The expected
values are numpy's float64 products and float32 conversions, bit for bit.
"""
import numpy as np
import pytest

import casars_cuda as cc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = cc.Context(0)
    yield c
    c.close()


def check(ctx, R, C, frac, seed, pair=True, spectrum=False):
    rng = np.random.default_rng(seed)
    K = 2
    uvw = rng.normal(0, 5000, (R, 3))
    special = [1.0 + 2.0 ** -24, 1.0 + 3 * 2.0 ** -24, -(1.0 + 2.0 ** -24), 1e-40, 1e39, -1e39, 0.0,
               -0.0, np.inf, 2.0 ** -126 * (1 - 2.0 ** -26), 2.0 ** 127 * (2 - 2.0 ** -25)]
    uvw[:min(R, len(special)), 0] = special[:R]
    uvw[:min(R, len(special)), 1] = special[::-1][:R]
    ls = np.ones(C)
    ls[1:] = rng.uniform(3.0, 6.0, C - 1)
    data = (rng.normal(size=(R, C, K)) + 1j * rng.normal(size=(R, C, K))).astype(np.complex64)
    flag = (rng.random((R, C, K)) < frac).astype(np.uint8)
    wt = rng.uniform(0.5, 2.0, (R, C, K) if spectrum else (R, K)).astype(np.float32)
    pol = cc.Polarization(0, 1, "half_sum", 2.0) if pair else cc.Polarization(1)
    b, du, dv = cc.prepare_row_runs(ctx, cc.RowRuns(uvw, ls, data, flag, None if spectrum else wt,
                                                    wt if spectrum else None), pol)
    used = flag.any(2) if pair else flag[:, :, 1] != 0
    r, c = np.nonzero(~used)
    assert len(b) == len(r)
    w3 = wt if spectrum else np.broadcast_to(wt[:, None, :], (R, C, K))
    with np.errstate(all="ignore"):
        for got, axis in ((b.u_lambda, 0), (b.v_lambda, 1), (b.w_lambda, 2)):
            np.testing.assert_array_equal(got, uvw[r, axis] * ls[c])
        ls32 = ls.astype(np.float32).astype(np.float64)
        for got, axis in ((du, 0), (dv, 1)):
            want = (uvw[r, axis] * ls32[c]).astype(np.float32).astype(np.float64)
            np.testing.assert_array_equal(got, want)
            np.testing.assert_array_equal(np.signbit(got), np.signbit(want))
    half = np.float32(0.5)
    weight = half * (w3[r, c, 0] + w3[r, c, 1]) if pair else w3[r, c, 1]
    vis = half * (data[r, c, 0] + data[r, c, 1]) if pair else data[r, c, 1]
    np.testing.assert_array_equal(b.weight, weight)
    np.testing.assert_array_equal(b.visibility, vis)


@pytest.mark.parametrize("R,C", [(1, 1), (2047, 1), (683, 3), (2049, 1), (32, 64), (4097, 1),
                                 (9655, 7), (33 * 2048 + 1, 1)])
@pytest.mark.parametrize("frac", [0.0, 0.3, 1.0])
def test_tiles(ctx, R, C, frac):
    check(ctx, R, C, frac, R + C)


@pytest.mark.parametrize("pair,spectrum", [(False, False), (False, True), (True, True)])
def test_forms(ctx, pair, spectrum):
    check(ctx, 3001, 5, 0.2, 9, pair, spectrum)
