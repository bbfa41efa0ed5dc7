"""The narrow deblocking filter's arithmetic on pairs (lpf_pair in
goav1_b200/csrc/pf_deblock.cu), restated in numpy: a sample n is the half
precision number n * 2^-24 as a bit pattern, and each operation rounds once to
half precision.  Every pair of differences (q0 - p0, p1 - q1) of 8- and 10-bit
samples, with and without a high edge variance, at both ends of the sample
range, against the integer form (loopfilter/sb.go:348-446)."""

import numpy as np
import pytest

UNIT = 2.0 ** -24


def half(v):
    """v (float64, in units, one operation's exact result) rounded to half precision."""
    return (v * UNIT).astype(np.float16).astype(np.float64) / UNIT


def clip(v, top):
    """The bit pattern as a signed 16-bit integer, held to 0..top."""
    bits = (v * UNIT).astype(np.float16).view(np.int16).astype(np.int64)
    return np.clip(bits, 0, top)


def narrow_half(d, e, hev, p0, q0, p1, q1, bd):
    up, top = bd - 8, (1 << bd) - 1
    lo, hi = -float(256 << up), float((256 << up) - 9)
    base = np.maximum(np.minimum(half(e + e), half(np.float64(hi + 7))), lo) * hev
    f = np.maximum(half(6 * d + base), lo)
    g1, g2 = np.minimum(half(f + 1), hi), np.minimum(half(f - 1), hi)
    f1 = half(g1 / 16)
    r = half(2 * f1 + 1)
    return [clip(half(g2 / 16 + p0), top), clip(half(-g1 / 16 + q0), top),
            p1 if hev else clip(half(r / 4 + p1), top), q1 if hev else clip(half(-r / 4 + q1), top)]


def narrow_int(d, e, hev, p0, q0, p1, q1, bd):
    lo, hi, top = -128 << (bd - 8), (128 << (bd - 8)) - 1, (1 << bd) - 1
    f = np.clip((np.clip(e, lo, hi) if hev else 0) + 3 * d, lo, hi)
    f1, f2 = np.minimum(f + 4, hi) >> 3, np.minimum(f + 3, hi) >> 3
    f = (f1 + 1) >> 1
    return [np.clip(p0 + f2, 0, top), np.clip(q0 - f1, 0, top), p1 if hev else np.clip(p1 + f, 0, top),
            q1 if hev else np.clip(q1 - f, 0, top)]


@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("hev", [0, 1])
@pytest.mark.parametrize("end", ["low", "high"])
def test_narrow_filter(bd, hev, end):
    top = (1 << bd) - 1
    e = np.arange(-top, top + 1)
    for d in range(-top, top + 1):
        dd = np.full_like(e, d)
        if end == "low":
            p0, q1 = max(0, -d), np.maximum(0, -e)
        else:
            p0, q1 = min(top, top - d), np.minimum(top, top - e)
        q0, p1 = p0 + d, q1 + e
        p0, q0 = np.full_like(e, p0), np.full_like(e, q0)
        want = narrow_int(dd, e, hev, p0, q0, p1, q1, bd)
        got = narrow_half(dd.astype(np.float64), e.astype(np.float64), hev, p0.astype(np.float64), q0.astype(np.float64),
                          p1.astype(np.float64), q1.astype(np.float64), bd)
        for name, a, b in zip(("p0", "q0", "p1", "q1"), want, got):
            assert np.array_equal(a, b), (d, name, e[a != b][:4])


@pytest.mark.parametrize("bd", [8, 10])
def test_edge_limit(bd):
    """4 |q0 - p0| + |p1 - q1| <= 2 E + 1 for every pair of differences and the
    limits of every level and sharpness: sums past 2,047 round, but stay past
    the largest limit."""
    top = (1 << bd) - 1
    d, e = np.meshgrid(np.arange(top + 1), np.arange(top + 1), indexing="ij")
    s = half((4 * d + e).astype(np.float64))
    exact, twice = 4 * d + e, 2 * d + (e >> 1)
    limits = set()
    for level in range(1, 64):
        for sharp in range(8):
            limit = level >> ((sharp > 0) + (sharp > 4))
            limit = max(1, min(limit, 9 - sharp) if sharp else limit)
            limits.add((2 * (level + 2) + limit) << (bd - 8))
    assert 2 * max(limits) + 1 < 2047
    for E in sorted(limits)[:: max(1, len(limits) // 24)] + [min(limits), max(limits)]:
        assert np.array_equal(twice <= E, s <= 2 * E + 1), E
    assert np.array_equal(exact[exact < 2048], s[exact < 2048])
