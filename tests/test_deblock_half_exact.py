"""Deblocking's half-precision filter path gives the reference's integers exactly.

At 8 and 10 bits deblock_kernel filters two lines per thread in packed half
precision.  Samples are held as 1024 + v, so the differences of two are exact
(integers below 1024).  This restates what the kernel decides and computes from
them in numpy, each operation computed exactly in float64 and rounded once to
float16 as the hardware does, and compares it with the integer arithmetic of
filter_mask and narrow_filter (src/loop_filter.rs:582-788) over every pair of
differences p1 - q1 and q0 - p0, every blimit that a level and a sharpness give,
and every sample that a result is added to.  Values that half precision rounds
lie beyond a bound or a clamp already.
"""
import numpy as np
import pytest

LEVELS = range(1, 64)


def _r(x):
    """One rounding to half precision of an exactly computed value, as float64 again."""
    return np.asarray(x, dtype=np.float64).astype(np.float16).astype(np.float64)


def _blimits():
    out = set()
    for sharp in range(8):
        sh = 2 if sharp > 4 else 1 if sharp > 0 else 0
        for lvl in LEVELS:
            limit = min(max(lvl >> sh, 1), 9 - sharp) if sharp > 0 else max(lvl >> sh, 1)
            out.add((2 * (lvl + 2) + limit) & 0xFF)
    return sorted(out)


@pytest.mark.parametrize("bd", [8, 10])
def test_filter_mask_step(bd):
    top, scale = (1 << bd) - 1, 1 << (bd - 8)
    a, b = np.arange(top + 1)[:, None], np.arange(top + 1)[None, :]  # |q0 - p0|, |p1 - q1|
    step = _r(a * 2.0 + _r(b * 0.5))
    exact = a * 2 + b // 2
    for blimit in _blimits():
        bound = _r(scale * blimit + 0.5)
        assert bound == scale * blimit + 0.5
        assert np.array_equal(step <= bound, exact <= scale * blimit), blimit


@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("hev", [False, True])
def test_narrow_filter(bd, hev):
    top = (1 << bd) - 1
    lo, hi = -(1 << (bd - 1)), (1 << (bd - 1)) - 1
    # the integers
    dp = np.arange(-top, top + 1)[:, None] if hev else np.zeros((1, 1), np.int64)
    dq = np.arange(-top, top + 1)[None, :]
    f = np.clip((np.clip(dp, lo, hi) if hev else 0) + 3 * dq, lo, hi)
    f1, f2 = np.clip(f + 4, lo, hi) >> 3, np.clip(f + 3, lo, hi) >> 3
    ff = (f1 + 1) >> 1
    # the kernel's sequence
    g = np.clip(dp.astype(np.float64), lo, hi) if hev else 0.0
    g = np.clip(_r(dq * 3.0 + g), lo, hi)
    cap = _r(hi - 3.5)
    g1 = _r(_r(np.minimum(_r(g + 0.5), cap) * 0.125 + 1536.0) - 1536.0)
    g2 = _r(_r(np.minimum(_r(g - 0.5), cap) * 0.125 + 1536.0) - 1536.0)
    gf = _r(_r(_r(g1 * 0.5 + 0.25) + 1536.0) - 1536.0)
    assert np.array_equal(g1, f1) and np.array_equal(g2, f2) and np.array_equal(gf, ff)


@pytest.mark.parametrize("bd", [8, 10])
def test_results_are_clamped_to_the_depth(bd):
    top, half = (1 << bd) - 1, 1 << (bd - 1)
    v = np.arange(top + 1)[:, None]
    d = np.arange(-(half >> 3) - 1, (half >> 3) + 2)[None, :]  # every f1, f2 and (f1 + 1) >> 1
    want = np.clip(v - half + d, -half, half - 1) + half
    got = np.minimum(np.maximum(_r(1024.0 + v + d), 1024.0), 1024.0 + top) - 1024.0
    assert np.array_equal(got, want)
