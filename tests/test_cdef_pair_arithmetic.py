"""The CDEF kernels' packed fp16 arithmetic, restated on the CPU.

pair_constrain and pair_round in goav1_b200/csrc/pf_cdef_dev.cuh compute the
reference's integer constrain() (cdef/filter.go:603-612) and its final
rounding (cdef/filter.go:150-169) on samples held as fp16 values.  Each
instruction is modelled as the exact result rounded once to fp16 (numpy's
conversion from float64 rounds to nearest even, as the hardware does, and
every exact result here fits a float64), and compared with the integers over
every difference, strength and shift of 8- and 10-bit frames.
"""

import numpy as np
import pytest

Q = 2.0 ** -10


def f16(x):
    return np.asarray(x, np.float64).astype(np.float16).astype(np.float64)


def from_bits(b):
    return float(np.array([b & 0xFFFF], np.uint16).view(np.float16)[0])


def pair_tap(thr, shift):
    """PairTap's three constants, from the bits the kernel forms."""
    o = 0x8000 + ((shift + 3) << 10) + 1024 - (2048 >> shift) if shift else 0
    return from_bits(0x3C00 + thr), from_bits(0xBC00 - (shift << 10)), from_bits(o)


def pair_constrain(d, tap):
    k, m, o = tap
    a = np.abs(d)
    v = f16(f16(a + o) * m + k)
    c = np.minimum(np.clip(f16(v - 1.0), 0.0, 1.0), a)
    return np.copysign(c, d)


def pair_round(x, s):
    return f16(s * from_bits(0x2C01) + x)


def constrain_shift(thr, damping):
    return max(0, damping - (thr.bit_length() - 1)) if thr else 0


@pytest.mark.parametrize("bd", [8, 10])
def test_constrain_every_difference(bd):
    top, scale = (1 << bd) - 1, bd - 8
    n = np.arange(-top, top + 1)
    # Luma strengths are adjusted by the variance, so any value up to the
    # largest occurs; damping 3..6 in the bitstream, one less for chroma.
    for thr in range((15 << scale) + 2):
        for damping in range(2 + scale, 7 + scale):
            shift = constrain_shift(thr, damping)
            a = np.abs(n)
            want = np.sign(n) * np.minimum(a, np.maximum(0, thr - (a >> shift)))
            d = f16(f16(1 + (n + top) % (top + 1) * Q) - f16(1 + ((n + top) % (top + 1) - n) * Q))
            assert np.array_equal(d, n * Q)
            assert np.array_equal(pair_constrain(d, pair_tap(thr, shift)) / Q, want)
            # An absent sample (-3) against every sample: no contribution.
            x = f16(1 + np.arange(top + 1) * Q)
            assert not pair_constrain(f16(-3.0 - x), pair_tap(thr, shift)).any()


@pytest.mark.parametrize("bd", [8, 10])
def test_rounding_and_clamp(bd):
    top, scale = (1 << bd) - 1, bd - 8
    most = 12 * (15 << scale) + 12 * (4 << scale)
    s = np.arange(-most, most + 1)
    assert np.array_equal(f16(s * Q), s * Q)
    for x in list(range(0, top + 1, 7 if bd == 10 else 1)) + [top]:
        want = x + ((8 + s - (s < 0)) >> 4)
        y = pair_round(f16(1 + x * Q), s * Q)
        # One filter alone stays between its samples: the rounded value itself.
        between = (16 * x + s >= 0) & (16 * x + s <= 16 * top)
        assert np.array_equal((y[between] - 1) / Q, want[between])
        # Both filters: clamped to a range around x inside the sample range.
        for lo in {0, x // 2, x}:
            for hi in {x, (x + top) // 2, top}:
                got = (np.clip(y, 1 + lo * Q, 1 + hi * Q) - 1) / Q
                assert np.array_equal(got, np.clip(want, lo, hi))


def test_sample_order_in_16_bit_integers():
    """The clamp compares bit patterns: samples in order, an absent one below
    them all signed and above them all unsigned."""
    b = np.arange(1024) | 0x3C00
    v = b.astype(np.uint16).view(np.float16).astype(np.float64)
    assert np.array_equal(v, 1 + np.arange(1024) * Q)
    none = np.array([0xC200], np.uint16)
    assert float(none.view(np.float16)[0]) == -3.0
    assert none.view(np.int16)[0] < b.astype(np.uint16).view(np.int16).min() and none[0] > b.max()
