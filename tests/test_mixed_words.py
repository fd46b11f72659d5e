"""The 6-byte mixed format (grg_b200.h, GRG_B200_MIXED) restated in NumPy: the leading 32 bits of a
value as an FP32 number plus its next 16 mantissa bits, rounded to nearest even.  On CPU: the
rounding bound, exact integers, the edges of the exponent range, and the walk's way of decoding
(integer shifts into a double that is the value x 2^-896, scaled back)."""

from __future__ import annotations

import numpy as np
import pytest


def encode(v: np.ndarray) -> tuple[np.ndarray, np.ndarray]:
    v = np.asarray(v, dtype=np.float64)
    with np.errstate(under="ignore"):
        bits = (v * 2.0**-896).view(np.uint64)
    sign = (bits >> np.uint64(32)).astype(np.uint32) & np.uint32(0x80000000)
    m = bits & np.uint64(0x7FFFFFFFFFFFFFFF)
    m = (m + np.uint64(0xFFF) + ((m >> np.uint64(13)) & np.uint64(1))) >> np.uint64(13)
    over = m >= np.uint64(255 << 39)
    m = np.where(over, np.where(np.isnan(v), np.uint64(511 << 38), np.uint64(255 << 39)), m)
    return sign | (m >> np.uint64(16)).astype(np.uint32), (m & np.uint64(0xFFFF)).astype(np.uint32)


def decode(hi: np.ndarray, lo: np.ndarray) -> np.ndarray:
    high = (hi.view(np.int32) >> 3).view(np.uint32) & np.uint32(0x8FFFFFFF)
    low = (hi << np.uint32(29)) | (lo << np.uint32(13))
    scaled = ((high.astype(np.uint64) << np.uint64(32)) | low.astype(np.uint64)).view(np.float64)
    special = (hi & np.uint32(0x7F800000)) == np.uint32(0x7F800000)
    return np.where(special, hi.view(np.float32).astype(np.float64), scaled * 2.0**896)


def bound(v: np.ndarray) -> np.ndarray:
    """Half a unit of the 40 significant bits; below 2^-126 half of 2^-165, plus the rounding of the
    scaled double to its own subnormal spacing (2^-1074 against 2^-1061)."""
    return np.maximum(np.abs(v) * 2.0**-40, 2.0**-166 * (1 + 2.0**-13))


@pytest.mark.parametrize("scale", [1e-37, 1e-20, 1.0, 1e20, 1e37])
def test_rounding_bound(scale):
    v = np.random.default_rng(0).standard_normal(200_000) * scale
    back = decode(*encode(v))
    assert np.all(np.abs(back - v) <= bound(v))


def test_integers_are_exact():
    rng = np.random.default_rng(1)
    for v in (np.arange(-5000, 5000, dtype=np.float64), np.arange(2**24, 2**24 + 20_000, dtype=np.float64),
              rng.integers(-(2**40), 2**40 + 1, 200_000).astype(np.float64)):
        np.testing.assert_array_equal(decode(*encode(v)), v)


def test_edges_of_the_range():
    with np.errstate(over="ignore", under="ignore"):
        top = np.asarray([2.0**128 * (1 - 2.0**-40), np.finfo(np.float32).max, 2.0**-126, 2.0**-149, 2.0**-165, -0.0, 0.0])
        np.testing.assert_array_equal(decode(*encode(top)), top)
        assert np.signbit(decode(*encode(np.asarray([-0.0])))[0])
        special = np.asarray([np.inf, -np.inf, 2.0**128, -1e300])
        np.testing.assert_array_equal(decode(*encode(special)), [np.inf, -np.inf, np.inf, -np.inf])
        assert np.isnan(decode(*encode(np.asarray([np.nan, -np.nan])))).all()
        small = np.random.default_rng(2).standard_normal(10_000) * 2.0**-130
        assert np.all(np.abs(decode(*encode(small)) - small) <= bound(small))
