"""The FP64 form's cheaper operations (pic_plain_math.cuh, the fixed-point words of
pic_internal.cuh) as the kernels run them, against exact arithmetic."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from device_math_build import load

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dm(tmp_path_factory):
    return load(str(tmp_path_factory.mktemp("device_math")))


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def test_division_by_the_cell_size_is_the_ieee_quotient(dm):
    rng = np.random.default_rng(1)
    sizes = np.concatenate([[0.1, 0.011424, 0.0125, 1.0 / 3.0, 1.0, 0.7, 6.4 / 64, np.nextafter(1.0, 2.0),
                             np.nextafter(2.0, 1.0)], rng.uniform(1e-3, 10.0, 200)])
    a, h = [], []
    for s in sizes:
        near = np.arange(-2, 600) * s
        v = np.concatenate([rng.uniform(-s, 512 * s, 4000), near, np.nextafter(near, 1e9), np.nextafter(near, -1e9),
                            s * 2.0 ** -rng.uniform(0, 60, 200)])
        a.append(v)
        h.append(np.full(v.size, s))
    a, h = np.concatenate(a), np.concatenate(h)
    out = np.zeros(a.size)
    assert dm.dm_gpu_div(a.size, ptr(a), ptr(h), ptr(out)) == 0
    assert np.array_equal(out, a / h)


def test_truncations(dm):
    rng = np.random.default_rng(2)
    ints = np.concatenate([np.arange(0.0, 600.0), [2.0 ** 31, 2.0 ** 32 - 1]])
    t = np.concatenate([rng.uniform(0, 8, 4000), rng.uniform(0, 2.0 ** 32 - 1, 4000), ints, np.nextafter(ints, 1e10),
                        np.nextafter(ints[1:], 0.0)])
    bad = np.concatenate([-rng.uniform(0, 4, 1000), [-1e-9, -0.5, -1.0, -2.0, -1e300, 2.0 ** 32, 2.0 ** 32 + 2.0, 2.0 ** 51,
                                                      2.0 ** 52 * 3, 1e300, np.inf, -np.inf, np.nan]])
    both = np.concatenate([t, bad])
    fi, ti, ex = (np.zeros(both.size, np.int32) for _ in range(3))
    fv = np.zeros(both.size)
    assert dm.dm_gpu_trunc(both.size, ptr(both), ptr(fi), ptr(fv), ptr(ti), ptr(ex)) == 0
    n = t.size
    want = t.astype(np.uint32)
    assert np.array_equal(fi[:n].view(np.uint32), want) and np.array_equal(ti[:n].view(np.uint32), want)
    assert np.array_equal(fv[:n], np.floor(t)) and ex[:n].all()
    assert not ex[n:].any()  # an index that is not one is told apart


@pytest.mark.parametrize("bits", [7, 14, 21, 24])
def test_rounded_sums(dm, bits):
    """two contributions below 2^51 quanta, either sign: high word the sum of the
    roundings to nearest even, low word that of the exact remainders in units of
    2^-40 or 2^-bits, rounded to nearest even"""
    rng = np.random.default_rng(3 + bits)
    n = 4000
    s, r = (rng.choice([-1.0, 1.0], n) * rng.uniform(1.0, 2.0, n) * 2.0 ** rng.uniform(-60, 50, n) for _ in range(2))
    s[:8] = [0.5, 1.5, -0.5, -2.5, 0.0, 2.0 ** 51 - 1, -(2.0 ** 51 - 1), 2.0 ** 31 - 0.5]
    r[:8] = [0.5, -1.5, -0.5, 2.5, -0.0, 1.0, -1.0, 0.25]
    wide, narrow = np.zeros((n, 2), np.int64), np.zeros((n, 2), np.int64)
    assert dm.dm_gpu_split(n, ptr(s), ptr(r), bits, ptr(wide), ptr(narrow)) == 0

    def words(v, b):
        hi = round(Fraction(v))  # half to even
        return hi, round((Fraction(v) - hi) * 2 ** b)

    for i in range(n):
        for b, got in ((40, wide[i]), (bits, narrow[i])):
            a, c = words(float(s[i]), b), words(float(r[i]), b)
            assert (a[0] + c[0], a[1] + c[1]) == (got[0], got[1])
