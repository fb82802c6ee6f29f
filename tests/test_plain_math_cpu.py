"""The FP64 form's cheaper operations (pic_plain_math.cuh, fx_split in
pic_internal.cuh), restated with exactly rounded operations on the host: they
give the bits of the operations they stand for."""
from fractions import Fraction

import numpy as np


def rn(x):
    """a rational number correctly rounded to FP64"""
    return x.numerator / x.denominator


def fma(a, b, c):
    return rn(Fraction(a) * Fraction(b) + Fraction(c))


def div_by(a, h, rh):
    q = a * rh
    q = fma(fma(-q, h, a), rh, q)
    return fma(fma(-q, h, a), rh, q)


def test_division_by_the_cell_size_is_exact():
    rng = np.random.default_rng(1)
    sizes = [0.1, 0.011424, 0.0125, 1.0 / 3.0, 1.0, 0.7, 1.1424 / 100, 6.4 / 64, np.nextafter(1.0, 2.0),
             np.nextafter(2.0, 1.0)]
    for h in sizes + list(rng.uniform(1e-3, 10.0, 20)):
        h = float(h)
        rh = 1.0 / h
        near = np.arange(0, 60) * h
        a = np.concatenate([rng.uniform(0, 64 * h, 300), rng.uniform(0, h, 200), near, np.nextafter(near, 1e9),
                            np.nextafter(near[1:], 0.0), h * 2.0 ** -rng.uniform(0, 60, 50), [0.0]])
        for x in a:
            x = float(x)
            assert div_by(x, h, rh) == x / h, (x, h)


def test_truncation_by_adding_2_52_rounded_down():
    """dadd_rd(t, 2^52): the exact sum rounded down to an integer (ulp 1 in
    [2^52, 2^53)); its low word is (int)t and the difference is floor(t)."""
    rng = np.random.default_rng(2)
    t = np.concatenate([rng.uniform(0, 8, 2000), rng.uniform(0, 1e6, 500), np.arange(20.0), np.nextafter(np.arange(1, 20.0), 0),
                        np.nextafter(np.arange(20.0), 99), [2.0 ** 32 - 1]])
    for v in t:
        m = Fraction(float(v)) + 2 ** 52
        down = float(m.numerator // m.denominator)   # exact: below 2^53
        bits = np.float64(down).view(np.uint64)
        assert int(bits) & 0xFFFFFFFF == int(v) and int(bits) >> 32 == 0x43300000
        assert down - 2.0 ** 52 == np.floor(v)
    # a negative or huge argument never passes for an index: the high word differs
    for v in (-1e-9, -0.5, -2.0, 2.0 ** 32, 2.0 ** 32 + 2.0, 1e300, np.inf, np.nan):
        with np.errstate(all="ignore"):
            m = np.float64(v) + 2.0 ** 52 if not (-1 < v < 0) else np.nextafter(2.0 ** 52, 0.0)
        assert int(np.float64(m).view(np.uint64)) >> 32 != 0x43300000


def test_rounding_by_adding_three_halves_2_52():
    """u = s + 1.5 * 2^52, |s| < 2^51: the low bits are rint(s), s - (u - 1.5 * 2^52) is the exact remainder"""
    rng = np.random.default_rng(3)
    s = np.concatenate([rng.standard_normal(2000) * 2.0 ** rng.uniform(-10, 49, 2000), [0.5, 1.5, -0.5, -2.5, 0.0, 2.0 ** 51 - 1]])
    for v in s:
        v = float(v)
        u = v + 1.5 * 2.0 ** 52
        ih = int(np.float64(u).view(np.int64)) - 0x4338000000000000
        assert ih == int(np.rint(v))
        r = v - (u - 1.5 * 2.0 ** 52)
        assert Fraction(r) == Fraction(v) - ih and abs(r) <= 0.5
