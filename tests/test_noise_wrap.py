"""Noise-cell wrap arithmetic of the packed taps (NoiseCells, kWrapMask / kWrapMul), restated in
FP32 and 32-bit integers on the CPU against floor and the integer remainder, for every extent:
u + 1.5 * 2^23 rounded down holds floor(u) in its low bits, the multiply-high quotient is exact
below 2^21, and the clamp is the cell a NaN position reads in the general form."""
import numpy as np
import pytest

REACH = 1 << 19
MAGIC = np.float32(12582912.0)
BITS = np.uint32(0x4B400000)


def add_down(u):
    """FP32 u + MAGIC rounded toward minus infinity: the nearest sum, one step down when its
    distance from MAGIC (exact) exceeds u."""
    f = (u.astype(np.float64) + np.float64(MAGIC)).astype(np.float32)
    over = f.astype(np.float64) - np.float64(MAGIC) > u.astype(np.float64)
    return np.where(over, np.nextafter(f, np.float32(-np.inf)), f).astype(np.float32)


def constants(m):
    r = (1 << 24) % m
    clamp = -float(((REACH - r) // m) * m + r)
    off = ((REACH + m - 1) // m) * m
    mul = (1 << 32) // m + 1 if m > 1 else 0
    return clamp, off, mul


def coordinates(m, rng):
    whole = rng.integers(-REACH + 4096, REACH - 4096, 200).astype(np.float32)
    edge = np.array([-m, -1, 0, 1, m - 1, m, m + 1, -REACH + 4096, REACH - 4096], np.float32)
    base = np.concatenate([whole, edge])
    return np.concatenate([base, base - np.float32(0.5), np.nextafter(base, np.float32(-np.inf)),
                           np.nextafter(base, np.float32(np.inf)), rng.uniform(-4 * m, 4 * m, 200).astype(np.float32)])


@pytest.mark.parametrize("first", range(1, 2049, 256))
def test_wrap_matches_floor_and_remainder(first):
    rng = np.random.default_rng(first)
    for m in range(first, min(first + 256, 2049)):
        clamp, off, mul = constants(m)
        u = np.maximum(coordinates(m, rng), np.float32(clamp))
        t = add_down(u)
        fl = t - MAGIC
        np.testing.assert_array_equal(fl, np.floor(u))
        want = np.mod(np.floor(u).astype(np.int64), m)
        if m & (m - 1) == 0:
            np.testing.assert_array_equal(t.view(np.uint32) & np.uint32(m - 1), want)
        if m > 1:
            b = (t.view(np.uint32) - BITS + np.uint32(off)).astype(np.uint64)
            assert int(b.max()) < 1 << 21
            q = (b * np.uint64(mul)) >> np.uint64(32)
            np.testing.assert_array_equal(b - q * np.uint64(m), want)


def test_nan_positions_read_the_general_forms_cell():
    for m in range(1, 2049):
        clamp, _, _ = constants(m)
        assert -REACH <= clamp < -REACH + 4096 and clamp == int(clamp)
        assert int(clamp) % m == (-(1 << 24)) % m
