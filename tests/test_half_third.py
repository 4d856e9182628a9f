"""CPU: x / 6 == 0.5 * (x / 3) in IEEE arithmetic, wherever the D3Q27 MRT population
transform forms x / 6 as half of the correctly rounded x / 3 inside an FMA
(populations_d3q27, lb-cube_b200/csrc/collide.cuh): every FP32 x of at least 2^-123 in
magnitude, every FP64 x of at least 2^-960.

x / 6 and x / 3 have the same significand quotient, one binade apart, so they round alike as long
as x / 6 is a normal number; the halving is then exact. FP32: every pattern of the
binades from 2^-123 to 2^-99 (where x / 6 comes next to the subnormals), of [1, 2) and of the
top binade, both signs; in between every value is a normal number scaled by a
power of two. FP64: random patterns over every exponent from 2^-960 on, and quotients next
to rounding midpoints."""
import numpy as np


def test_fp32():
    binades = list(range(127 - 123, 127 - 98)) + [127, 254]
    mantissa = np.arange(1 << 23, dtype=np.uint32)
    for e in binades:
        x = (mantissa | np.uint32(e << 23)).view(np.float32)
        for s in (x, -x):
            six, half = s / np.float32(6), np.float32(0.5) * (s / np.float32(3))
            assert np.array_equal(six.view(np.uint32), half.view(np.uint32)), e


def test_fp32_bound_is_needed():
    """Below 2^-123 the halves round a second time."""
    x = (np.arange(1 << 23, dtype=np.uint32) | np.uint32((127 - 124) << 23)).view(np.float32)
    assert not np.array_equal(x / np.float32(6), np.float32(0.5) * (x / np.float32(3)))


def test_fp64():
    rng = np.random.default_rng(11)
    for _ in range(8):
        bits = rng.integers(0, 1 << 52, 1 << 20, dtype=np.uint64)
        x = (bits | rng.integers(1023 - 960, 2047, 1 << 20, dtype=np.uint64) << np.uint64(52)).view(np.float64)
        # 3 q and 6 q next to the midpoint of two doubles: q odd in the 54th bit
        q = (rng.integers(0, 1 << 51, 1 << 20, dtype=np.uint64) << np.uint64(1) | np.uint64(1)).astype(np.float64) * 1.5
        for v in (x, -x, q, q * 2.0 ** -500):
            assert np.array_equal((v / 6.0).view(np.uint64), (0.5 * (v / 3.0)).view(np.uint64))
