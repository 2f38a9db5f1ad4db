"""CPU restatement of the assembled operator's fixed-point products
(gade_cuda.cu: fx_from, fx_split and the 30-product row sums) in exact
integers: the limbs hold a value to 2^-56 (2^-58 for vector entries) of its
group's largest, no 64-bit sum overflows, and a row's sum is within the bound
that follows from those roundings of the exact rational sum."""
from fractions import Fraction

import numpy as np
import pytest

LB, UPA, UPX = 29, 4, 5
I64 = 1 << 63


def _exp(v):
    return (int(np.float64(v).view(np.uint64)) >> 52) & 0x7FF


def _fx(v, em, up):
    b = int(np.float64(v).view(np.uint64))
    ev, m = (b >> 52) & 0x7FF, b & ((1 << 52) - 1)
    m, ev = (m | 1 << 52, ev) if ev else (m, 1)
    d = em - ev
    n = ((m << up >> (d - 1)) + 1) >> 1 if d else m << up
    return -n if b >> 63 else n


def _split(n):
    hi = (n + (1 << (LB - 1))) >> LB
    lo = n - (hi << LB)
    assert -(1 << 31) <= hi < 1 << 31 and abs(lo) <= 1 << (LB - 1)
    return hi, lo


def _row(a, x):
    """sum a x as the kernel forms it, and 2^e of its unit."""
    ea, ex = max(max(map(_exp, a)), 1), max(max(map(_exp, x)), 1)
    h = m = 0
    for av, xv in zip(a, x):
        (ah, al), (xh, xl) = _split(_fx(av, ea, UPA)), _split(_fx(xv, ex, UPX))
        h += ah * xh
        m += ah * xl + al * xh
        assert abs(h) < I64 and abs(m) < I64
    v = h + ((m + (1 << (LB - 1))) >> LB)
    assert abs(v) < I64
    return Fraction(v) * Fraction(2) ** (ea + ex - 2101)


@pytest.mark.parametrize("spread", [0, 8, 40, 300])
@pytest.mark.parametrize("scale", [0, -250, 250])
def test_row_sum_within_bound(spread, scale):
    rng = np.random.default_rng(100 * spread + scale + 1000)
    for _ in range(20):
        a = rng.uniform(-1, 1, 30) * 2.0 ** (rng.uniform(-spread, 0, 30) + scale)
        x = rng.uniform(-1, 1, 30) * 2.0 ** rng.uniform(-spread, 0, 30)
        exact = sum(Fraction(float(p)) * Fraction(float(q)) for p, q in zip(a, x))
        big = 4 * Fraction(float(np.abs(a).max())) * Fraction(float(np.abs(x).max()))
        # |a| and |x| truncated at 2^-56 and 2^-58 of their group's power of
        # two, the lo lo products below 2^-57, the final shift below 2^-56
        bound = (30 * (Fraction(1, 2 ** 56) + Fraction(1, 2 ** 58) + Fraction(1, 2 ** 57)) + Fraction(1, 2 ** 56)) * big
        assert abs(_row(a, x) - exact) <= bound


def test_largest_values_do_not_overflow():
    top = np.nextafter(2.0, 0.0)
    for sa in (1, -1):
        for sx in (1, -1):
            r = _row(np.full(30, sa * top), np.full(30, sx * top))
            assert abs(r - sa * sx * 30 * Fraction(float(top)) ** 2) < Fraction(1, 2 ** 40)


def test_zeros_and_denormals():
    assert _row(np.zeros(30), np.ones(30)) == 0
    tiny = np.full(30, 5e-324)
    assert abs(_row(tiny, np.ones(30)) - 30 * Fraction(5e-324)) <= Fraction(5e-324)
