"""The margins of the float32-pair decisions, emulated on the CPU.

The device's operations (cr_fixed.cuh: df_product, df_nearest, df_offset,
df_tap_span) in exact IEEE float32 arithmetic, on coordinates placed within
and beyond the margins of the anchor and offset boundaries (2^-26 to 2^-12 of
a cell or an oversampled cell away), for even and odd sizes, small and large
grids and oversamplings up to the largest accepted.  Every decision taken
equals the FP64 one (sample_tap_span, gridder.rs:1976-1995), and coordinates
more than 2^-15 away are decided.
"""
from fractions import Fraction

import numpy as np
import pytest

from test_fastpath_cpu import f32, fma32, pair, product

ANCHOR_MARGIN, OFFSET_MARGIN, OFFSET_REL = f32(2.0 ** -20), f32(2.0 ** -16), f32(2.0 ** -41)
LIMIT = f32(1048576.0)
MAGIC = f32(12582912.0)


def rint_magic(x):
    t = f32(x + MAGIC)
    r = f32(t - MAGIC)
    return r, int(r)


def nearest(p, e, h):
    if not abs(p) < LIMIT:
        return None
    q = p
    if h != 0.0:
        h = f32(h)
        q = f32(p + h)
        b = f32(q - p)
        e = f32(e + f32(f32(p - f32(q - b)) + f32(h - b)))
    r, n = rint_magic(q)
    f = f32(q - r)
    d = f32(f + e)
    if not abs(f32(abs(d) - f32(0.5))) > ANCHOR_MARGIN:
        return None
    if d > 0.5:
        n, f = n + 1, f32(f - f32(1.0))
    if d < -0.5:
        n, f = n - 1, f32(f + f32(1.0))
    return n, f, e


def tap_span(p, e, size, os_, rows):
    t = nearest(p, e, 0.5 if size & 1 else 0.0)
    if t is None:
        return None, None
    a, dh, e = t
    anchor = size // 2 + a
    if anchor - 3 < 0 or anchor + 3 >= size:
        return 0, None
    osf = f32(os_)
    v = -fma32(dh, osf, f32(e * osf))
    o, oi = rint_magic(v)
    if not f32(0.5) - abs(f32(v - o)) > fma32(f32(abs(p) * osf), OFFSET_REL, OFFSET_MARGIN):
        return None, None
    idx = oi + os_ // 2
    if idx < 0 or idx >= rows:
        return 0, None
    return 1, (anchor - 3, idx)


def away(x):
    """round half away from zero"""
    return int(np.floor(x + 0.5)) if x >= 0 else -int(np.floor(-x + 0.5))


def fp64_span(u, du, size, os_, rows):
    x = u / du + size / 2.0
    anchor = away(x)
    if anchor - 3 < 0 or anchor + 3 >= size:
        return 0, None
    idx = away((anchor - x) * os_) + os_ // 2
    if idx < 0 or idx >= rows:
        return 0, None
    return 1, (anchor - 3, idx)


@pytest.mark.parametrize("size,os_", [(101, 128), (128, 128), (4097, 254), (8192, 254),
                                      (32769, 63), (100000, 16)])
def test_decisions_near_boundaries_equal_fp64(size, os_):
    du = 37.3
    rows = 2 * (os_ // 2) + 1
    k = pair(Fraction(1) / Fraction(du))
    rng = np.random.default_rng(size)
    anchors = [3.5, size / 2.0 + 0.5 * (1 - size % 2), size - 3.5, 7.5, 64.5]
    anchors += [size // 2 + 2 ** j - 0.5 for j in range(1, 14) if 2 ** j < size // 2 - 4]
    bases = [(x, 1.0) for x in anchors]
    bases += [(rng.integers(4, size - 5) + (j + 0.5) / os_, 1.0 / os_)
              for j in rng.integers(-os_ // 2, os_ // 2, 40)]
    undecided = 0
    for base, unit in bases:
        for away_ in [0.0] + [2.0 ** -k for k in range(12, 27)]:
            for sign in (-1.0, 1.0):
                u = (base + sign * away_ * unit - size / 2.0) * du
                p, e = product(*pair(u), *k)
                got = tap_span(p, e, size, os_, rows)
                if got[0] is None:
                    undecided += 1
                    assert away_ < 2.0 ** -15 or unit == 1.0 or size > 32769, (base, away_)
                    continue
                assert got == fp64_span(u, du, size, os_, rows), (base, away_, sign)
    assert undecided > 0
