"""Accuracy of the wet sum of r (k_mean_fix): a thread's sum, taken in fixed point with
94 bits below sqrt(sum r^2), is the exact sum rounded to a double, as a compensated
FP64 sum is. Restates the kernel's arithmetic in Python integers.

The bound: conversions lose less than 2^-94 of the bound B a cell, and the sum's way
to a double rounds its high word (exact below 2^53), its low word and their sum, at
most one ulp of the sum and 2^11 units of 2^-94 B where they cancel."""
import math
import struct
from fractions import Fraction

import numpy as np
import pytest


def _fix(v, k, up):
    """to_fix_wide: the significand `up` bits up, shifted down, towards zero."""
    u = struct.unpack("<Q", struct.pack("<d", v))[0]
    ex = (u >> 52) & 0x7FF
    n = min(max(1075 + up - k - ex, 0), 127)
    r = (((u & 0x000FFFFFFFFFFFFF) | 0x0010000000000000) << up) >> n
    return -r if u >> 63 else r


def _to_double(v):
    """int_to_double: 2^64 times the high word plus the low one."""
    hi, lo = v >> 64, v & 0xFFFFFFFFFFFFFFFF
    return float(hi) * 18446744073709551616.0 + float(lo)


def _thread_sums(r, k, up, threads):
    for t in range(threads):
        cells = [float(v) for v in r[t::threads]]
        yield _to_double(sum(_fix(v, k, up) for v in cells)) * 2.0 ** -k, sum(Fraction(v) for v in cells), len(cells)


def _fields():
    rng = np.random.default_rng(2)
    n = 60000
    white = rng.standard_normal(n)
    steep = white * np.exp(rng.uniform(-30, 0, n))
    dipole = white * 1e-9
    dipole[[7, 40007]] = 1e6, -1e6
    tiny = np.concatenate([white[:1000] * 2.0 ** -530, np.zeros(n - 1000)])
    return {"white": white, "steep": steep, "dipole": dipole, "tiny": tiny, "zero": np.zeros(n)}


@pytest.mark.parametrize("name", list(_fields()))
def test_thread_sums_are_exact_sums_rounded_once(name):
    r = _fields()[name]
    sq = float(np.sum(r * r))
    e2 = math.frexp(sq)[1] if sq > 0 else 0
    E = (e2 + 1) >> 1
    unit = Fraction(2) ** (E - 94)
    for got, exact, n in _thread_sums(r, 94 - E, 42, 997):
        bound = Fraction(math.ulp(float(exact))) + (n + 2 ** 11) * unit
        assert abs(Fraction(got) - exact) <= bound, (name, got, float(exact))


def test_58_bits_would_not_do():
    """The dipole field: what a grid of 58 bits loses is more than the sum's own rounding."""
    r = _fields()["dipole"]
    E = (math.frexp(float(np.sum(r * r)))[1] + 1) >> 1
    worst = 0.0
    for got, exact, n in _thread_sums(r, 58 - E, 6, 997):
        worst = max(worst, float(abs(Fraction(got) - exact) / Fraction(math.ulp(float(exact)))))
    assert worst > 100.0
