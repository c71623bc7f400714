"""Precision of the FP64 pair field's fixed point where a site has only far
partners: coordinates are the state's own, and the summed terms keep FP64's
accuracy at every distance (restated with exact integers, and on the GPU)."""
import dataclasses
import math
from fractions import Fraction

import numpy as np
import pytest

from surfactant_enhanced_spreading_gb300 import system as S
from test_fixed_point_pairs import halves, inverse, r2_fixed


def fix_of(v):
    """Units of 2^-59 modulo 2^64, rounded to 2^-58 (as in the kernel)."""
    b = int(np.float64(v).view(np.int64))
    e = b >> 52 & 0x7FF
    s = e - (1023 + 52 - 58)
    m = (b & ((1 << 52) - 1)) | (int(e != 0) << 52)
    u = (m << (s & 63)) % (1 << 64) if s >= 0 else (m + (1 << (-s - 1))) >> -s if s > -55 else 0
    return ((-u if b < 0 else u) << 1) % (1 << 64)


def signed(v):
    v %= 1 << 64
    return v - (1 << 64) if v >> 63 else v


def term(w, lz):
    """r^-3 of r >= 1 in units of 2^-61 and its halves."""
    k = 3 * lz // 2
    assert k <= 9
    v = (w + (256 >> k)) >> (9 - k)
    h, l = v >> 31, v & 0x7FFFFFFF
    assert w < 1 << 63 and h < 1 << 31
    return v, h, l


def test_coordinates_are_the_states_own():
    """Differences of nearby coordinates, anywhere in a box: exact down to 2^-58."""
    rng = np.random.default_rng(1)
    for _ in range(4000):
        c = float(rng.uniform(-1, 1) * 2.0 ** rng.uniform(0, 20))
        p = c + float(rng.uniform(-9, 9) * 2.0 ** rng.uniform(-30, 0))
        d = signed(fix_of(p) - fix_of(c))
        exact = (Fraction(p) - Fraction(c)) * (1 << 59)
        assert d % 2 == 0
        if min(abs(p), abs(c)) >= 2.0 ** -6:
            assert d == exact
        else:
            assert abs(d - exact) <= 2
    for v in (0.0, -0.0, 2.0 ** -58, 2.0 ** -59, 2.0 ** -60, 2.0 ** -70, -(2.0 ** -6), 1.0, 1e6, -1e6, 5e-324):
        assert abs(signed(fix_of(v)) - Fraction(v) * (1 << 59)) <= 1 if abs(v) < 16 else True


def test_terms_are_within_a_unit():
    """d r^-3 of pairs at least 1 sigma apart in units of 2^-57: the rounding
    of r^-3 to 2^-61 (half a unit times |d| < 9.2), the product of the low
    halves and the rounding (half a unit each), the reciprocal's 2^-53."""
    rng = np.random.default_rng(5)
    seen = 0
    for _ in range(6000):
        d = [int(v * 2.0 ** 58) << 1 for v in rng.uniform(-9.1, 9.1, 3) * 2.0 ** rng.uniform(-4, 0)]
        r2 = r2_fixed(d)
        if r2 < 1 << 56:
            continue
        seen += 1
        w, lz = inverse(r2, 0.0)[:2]
        _, th, tl = term(w, lz)
        r3 = Fraction(1 << 124, int(math.isqrt(r2 ** 3 << 80)))
        for v in d:
            h, l = halves(v)
            c = h * tl + l * th + (1 << 30)
            assert abs(c) < 1 << 63 and abs(h * th) < 1 << 62
            got = h * th + (c >> 31)
            exact = Fraction(v, 1 << 59) * r3 * (1 << 57)
            assert abs(float(got - exact)) < 0.5 * 9.2 / 16 + 0.5 + 0.5 + abs(float(exact)) * 2.0 ** -52
            assert abs(got) <= (1 << 57) + 2        # 32 of them fit
    assert seen > 2000


def water_pairs(r, n, seed):
    """n pairs of waters r sigma apart, both in or beside one another's cells (8 cells of 12 A an axis)."""
    rng = np.random.default_rng(seed)
    tmpl = S.water_template() / S.SIGMA
    cell = S.RS
    out = []
    for _ in range(n):
        u = 1.0 + 0.2 * rng.uniform(-1, 1, 3)
        u /= np.linalg.norm(u)
        rot = S._rand_rots(rng, 2)
        a = cell * rng.integers(-2, 1, 3) + rng.uniform(0.6, 1.4, 3)     # towards a cell's lower corner
        out.append(np.concatenate([tmpl @ rot[0].T + a, tmpl @ rot[1].T + a + r * u]))
    return out


def pair_force(pos, dtype):
    """Coulomb force between the two waters of pos, in dtype: (6, 3)."""
    x = pos.astype(dtype)
    q = np.array([-0.82, 0.41, 0.41] * 2).astype(dtype)
    f = np.zeros((6, 3), dtype=dtype)
    for i in range(6):
        for j in (range(3, 6) if i < 3 else range(3)):
            d = x[i] - x[j]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            inv = dtype(1) / np.sqrt(r2)
            f[i] += (q[i] * dtype(np.float32(675.05)) * q[j] * inv * inv * inv) * d
    return f


@pytest.mark.gpu
@pytest.mark.parametrize("r", [4.0, 6.0, 8.0])
def test_far_waters_are_as_accurate_as_fp64(r):
    """Waters beyond the LJ cutoff with no other partner: the median error
    against extended precision is at most twice that of FP64 arithmetic (the
    sums over cells and rows add a rounding or two to the pair terms')."""
    from surfactant_enhanced_spreading_gb300 import config_preset as C
    from surfactant_enhanced_spreading_gb300 import engine as E
    base = C.config_droplet(200, 0, cells=(8, 8, 8), seed=1, graphite_layers=0)
    pairs = water_pairs(r, 150, int(r))
    systems = [dataclasses.replace(base, n_water=2, pos=p, vel=np.zeros((6, 3))) for p in pairs]
    f = E.Engine(systems, E.PLAIN_FP64).force(True, terms=E.T_NEAR).reshape(-1, 6, 3)
    err, ref = [], []
    for k, p in enumerate(pairs):
        exact = pair_force(p, np.longdouble)
        size = np.linalg.norm(exact.astype(np.float64), axis=1)
        err.append(np.linalg.norm((f[k] - exact).astype(np.float64), axis=1) / size)
        ref.append(np.linalg.norm((pair_force(p, np.float64) - exact).astype(np.float64), axis=1) / size)
    assert np.median(err) <= 2.0 * np.median(ref)
