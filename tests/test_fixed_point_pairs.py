"""The integer form of r^-3 and r^-2 of the FP64 pair field, restated with
exact integers: its error stays below plain FP64's for every seed that the
reciprocal square root's error bound allows."""
import math
from fractions import Fraction

import numpy as np
import pytest

ONE = 1 << 52


def r2_fixed(d):
    """Units of 2^-56 from differences in units of 2^-59 (truncations as in the kernel)."""
    s = c = q = 0
    for v in d:
        h, l = v >> 32, v & 0xFFFFFFFF
        s += h * h
        c += h * (l >> 1)
        q += l * l >> 32
    return (s << 2) + (c >> 28) + (q >> 30)


def clz32(v):
    return 32 - v.bit_length()


def inverse(r2, seed_error):
    """(r^-3, r^-2) as the kernel forms them; seed_error: relative error of the hardware's y."""
    lz = clz32(r2 >> 32) & ~1
    n = r2 << lz
    assert 1 << 62 <= n < 1 << 64
    n1, n0 = n >> 32, n & 0xFFFFFFFF
    y = np.float32((1.0 + seed_error) / math.sqrt(float(np.float32(n1))))
    m = int(y * np.float32(70368744177664.0 * (1.0 - 1.5 / 4194304.0)))
    mm = m * m
    assert mm % (1 << 12) == 0
    l, h = (mm >> 12) & 0xFFFFFFFF, mm >> 44
    t = (n1 * l + n0 * h + (n0 * l >> 32) + ((n1 * h) << 32)) & ((1 << 64) - 1)
    e = -t & ((1 << 64) - 1)
    assert e < 1 << 61          # e >= 0, below 2^-19
    e60 = e >> 20
    e2 = (e >> 32) ** 2 >> 32
    m3 = (mm >> 32) * m + ((mm & 0xFFFFFFFF) * m >> 32)
    w = m3 + (m3 * ((e60 + (e60 >> 1) + ((e2 * 15) >> 7)) << 4) >> 64)
    v = mm + (mm * ((e60 + (e2 >> 4)) << 4) >> 64)
    assert w < 1 << 64 and v < 1 << 64

    def rounded(x, ex):
        k = x.bit_length() - 53
        return math.ldexp((x >> k) + ((x >> (k - 1)) & 1), ex + k)
    return rounded(w, -70 + 3 * (lz >> 1)), rounded(v, -68 + lz)


@pytest.mark.parametrize("seed_error", [-(2.0 ** -22.9), 0.0, 2.0 ** -22.9])
def test_inverse_is_rounded_once(seed_error):
    rng = np.random.default_rng(3)
    r2s = [1 << 56, (1 << 56) - 1, (1 << 56) + 1, 1 << 58, (1 << 58) - 1, 1 << 54, 1 << 62, (1 << 64) - 1, 1 << 53]
    r2s += [int(v) for v in 2.0 ** rng.uniform(53, 63.99, 4000)]
    for r2 in r2s:
        i3, i2 = inverse(r2, seed_error)
        x = Fraction(r2, 1 << 56)
        # one rounding (2^-53) and the truncated terms of the series and of the products (2^-56)
        assert abs(Fraction(i2) * x - 1) < Fraction(1, 1 << 53) * Fraction(9, 8)
        assert abs(Fraction(i3) ** 2 * x ** 3 - 1) < Fraction(2, 1 << 53) * Fraction(9, 8)


def test_squared_distance():
    rng = np.random.default_rng(4)
    for _ in range(4000):
        d = [int(v * ONE) << 7 for v in rng.uniform(-9.1, 9.1, 3) * 2.0 ** rng.uniform(-6, 0)]
        exact = Fraction(sum(v * v for v in d), 1 << 118)
        got = Fraction(r2_fixed(d), 1 << 56)
        assert 0 <= exact - got < Fraction(3, 1 << 56)
        assert r2_fixed(d) < 1 << 64


def test_reach_keeps_the_square_in_range():
    """Sites within 2.7 sigma of their cells' centres, cells 12 A apart."""
    d = 2 * 2.7 + 12.0 / 3.166
    assert 3 * d * d < 256.0
