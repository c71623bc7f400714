"""The integer form of r^-3 and r^-2 of the FP64 pair field, restated with
exact integers: its error stays below plain FP64's for every seed that the
reciprocal square root's error bound allows."""
import math
from fractions import Fraction

import numpy as np
import pytest

ONE = 1 << 52


def halves(v):
    """h 2^32 + 2 l of a difference whose low 7 bits are zero, l signed."""
    l = (v & 0xFFFFFFFF) - ((v & 0x80000000) << 1)
    h = (v - l) >> 32
    assert v == (h << 32) + l and l % 2 == 0 and -(1 << 31) <= h < 1 << 31
    return h, l >> 1


def r2_fixed(d):
    """Units of 2^-56 from differences in units of 2^-59 (as in the kernel)."""
    hl = [halves(v) for v in d]
    s = sum(h * h for h, _ in hl)
    c = sum(h * l for h, l in hl) + 3 * (1 << 27)
    assert abs(c) < 1 << 63
    return (s << 2) + (c >> 28)


def clz32(v):
    return 32 - v.bit_length()


def inverse(r2, seed_error):
    """(w, lz, mm, e60, e2) as the kernel forms them; seed_error: relative error of the hardware's y."""
    lz = clz32(r2 >> 32 | 1 << 21) & ~1
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
    k = (e60 + (e60 >> 1) + ((e2 * 15) >> 7)) << 4
    assert k < 1 << 46
    kh, kl, mh, ml = k >> 32, k & 0xFFFFFFFF, m3 >> 32, m3 & 0xFFFFFFFF
    w = m3 + mh * kh + ((mh * kl + ml * kh) >> 32)
    assert mh * kl + ml * kh < 1 << 64
    return w, lz, mm, e60, e2


def rounded(x, ex):
    assert x < 1 << 64
    k = x.bit_length() - 53
    return math.ldexp((x >> k) + ((x >> (k - 1)) & 1), ex + k)


def term(w, lz):
    """r^-3 in units of 2^-57 and its halves."""
    k = 3 * lz // 2
    w4 = (w + (4096 >> k)) << 2
    assert w4 < 1 << 64
    v = w4 >> (15 - k)
    h, l = v >> 31, v & 0x7FFFFFFF
    assert h < 1 << 31
    return v, h, l


@pytest.mark.parametrize("seed_error", [-(2.0 ** -22.9), 0.0, 2.0 ** -22.9])
def test_inverse_is_rounded_once(seed_error):
    rng = np.random.default_rng(3)
    r2s = [1 << 56, (1 << 56) - 1, (1 << 56) + 1, 1 << 58, (1 << 58) - 1, 1 << 54, 1 << 62, (1 << 64) - 1, 1 << 53]
    r2s += [int(v) for v in 2.0 ** rng.uniform(53, 63.99, 4000)]
    for r2 in r2s:
        w, lz, mm, e60, e2 = inverse(r2, seed_error)
        i3 = rounded(w, -70 + 3 * (lz >> 1))
        i2 = rounded(mm + (mm * ((e60 + (e2 >> 4)) << 4) >> 64), -68 + lz)
        x = Fraction(r2, 1 << 56)
        # one rounding (2^-53) and the truncated terms of the series and of the products (2^-56)
        assert abs(Fraction(i2) * x - 1) < Fraction(1, 1 << 53) * Fraction(9, 8)
        assert abs(Fraction(i3) ** 2 * x ** 3 - 1) < Fraction(2, 1 << 53) * Fraction(9, 8)


def differences(rng):
    return [int(v * ONE) << 7 for v in rng.uniform(-9.1, 9.1, 3) * 2.0 ** rng.uniform(-6, 0)]


def test_squared_distance():
    rng = np.random.default_rng(4)
    for _ in range(4000):
        d = differences(rng)
        exact = Fraction(sum(v * v for v in d), 1 << 118)
        got = Fraction(r2_fixed(d), 1 << 56)
        # left out: three squares of up to a unit and a truncation, less 1.5 units
        assert Fraction(-3, 1 << 57) <= exact - got < Fraction(5, 1 << 57)
        assert r2_fixed(d) < 1 << 64


def test_force_term_is_within_a_unit():
    """d r^-3 in units of 2^-53: the rounding of r^-3 to 2^-57 (half a unit
    times |d| < 9.2), the product of the low halves (half a unit), the
    rounding (half), the reciprocal's 2^-53 of a term of at most 8 (2^3)."""
    rng = np.random.default_rng(5)
    total = 0.0
    for _ in range(4000):
        d = differences(rng)
        r2 = r2_fixed(d)
        if r2 < 1 << 53:
            continue
        w, lz = inverse(r2, 0.0)[:2]
        _, th, tl = term(w, lz)
        r3 = Fraction(1 << 124, int(math.isqrt(r2 ** 3 << 80)))   # (2^56 / r2)^(3/2) to 2^-80
        for v in d:
            h, l = halves(v)
            c = h * tl + l * th + (1 << 30)
            assert abs(c) < 1 << 63 and abs(h * th) < 1 << 62
            got = h * th + (c >> 31)
            exact = Fraction(v, 1 << 59) * r3 * (1 << 53)
            err = float(got - exact)
            assert abs(err) < 0.5 * 9.2 / 16 + 0.5 + 0.5 + abs(float(exact)) * 2.0 ** -52
            total += err
    assert abs(total) < 4.0 * 0.4 * math.sqrt(3 * 4000)   # no bias: four times the spread of 12,000 such errors


def test_reach_keeps_the_square_in_range():
    """Sites within 2.7 sigma of their cells' centres, cells 12 A apart."""
    d = 2 * 2.7 + 12.0 / 3.166
    assert 3 * d * d < 256.0
