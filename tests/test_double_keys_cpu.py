"""The integer-key minimum and maximum of doubles (jmin / jmax<double>, hcc_internal.cuh) against Julia's rule for IEEE
floats, which the compare-based forms implement: NaN-propagating, -0 below +0. The arithmetic of the keys is restated
here with 64-bit integers."""
import numpy as np

NAN_RANGE = 0x000FFFFFFFFFFFFF
MASK = (1 << 64) - 1


def key(x):
    b = int(np.float64(x).view(np.int64))
    return (b ^ 0x7FFFFFFFFFFFFFFF) if b < 0 else b


def signed(v):
    v &= MASK
    return v - (1 << 64) if v >> 63 else v


def kmin(x, y):
    return y if signed(key(y) + NAN_RANGE) < signed(key(x) + NAN_RANGE) else x


def kmax(x, y):
    return y if signed(key(y) - NAN_RANGE) > signed(key(x) - NAN_RANGE) else x


def rule(x, y, smaller):
    sx, sy = np.signbit(x), np.signbit(y)
    take_y = (y < x) or (sy and not sx) if smaller else (y > x) or (not sy and sx)
    return (x if np.isnan(x) else y) if take_y else (y if np.isnan(y) else x)


def test_integer_keys_follow_the_compare_rule():
    tiny, big = 5e-324, np.finfo(np.float64).max
    payload = np.array([0x7FF0000000000001, 0x7FFFFFFFFFFFFFFF, 0xFFF0000000000001, 0xFFFFFFFFFFFFFFFF],
                       dtype=np.uint64).view(np.float64)
    vals = [0.0, -0.0, tiny, -tiny, 2.2250738585072014e-308, 1.0, -1.0, np.nextafter(1.0, 2.0), big, -big, np.inf,
            -np.inf, *payload]
    rng = np.random.default_rng(3)
    vals += list(rng.integers(0, 1 << 63, 40, dtype=np.int64).view(np.float64)) + list(-rng.random(20))
    for x in vals:
        for y in vals:
            x, y = np.float64(x), np.float64(y)
            for got, want in ((kmin(x, y), rule(x, y, True)), (kmax(x, y), rule(x, y, False))):
                if np.isnan(x) or np.isnan(y):
                    assert np.isnan(got) and np.isnan(want)
                else:
                    assert np.float64(got).view(np.int64) == np.float64(want).view(np.int64)
