"""CPU restatement of the assembled operator's arithmetic (gade_fx.cuh: words
with an exponent of their own, sums aligned to their largest product; the
assembly of a value from its three factors) in exact integers: no 64-bit sum
overflows, and every row's sum is as close to the exact rational one as FP64's
rounding of its own terms, however its entries are spread."""
import math
from fractions import Fraction

import numpy as np
import pytest

OFF, LB, GS = 127, 30, 8
I64 = 1 << 63
ZERO = -100000


def _bits(v):
    b = int(np.float64(v).view(np.uint64))
    ev, m = (b >> 52) & 0x7FF, b & ((1 << 52) - 1)
    m, ev = (m | 1 << 52, ev) if ev else (m, 1)
    return m, ev, b >> 63


def _pow2(e):
    return Fraction(2) ** e


def _word(v, e):
    """(N 2^7, offset) of v in a group of exponent e."""
    m, ev, neg = _bits(v)
    if m == 0:
        return 0, OFF
    off, t = e - ev, m << 10
    if off > OFF:
        t, off = t >> min(off - OFF, 63), OFF
    t = (-t if neg else t) & ~127
    assert off >= 0 and -I64 <= t < I64
    return t, off


def _take(w, s):
    t = (w[0] | w[1]) >> min(s + 6, 64)
    h, lo = t >> LB, (t & ((1 << LB) - 1)) | 1
    assert -(1 << 31) <= h < 1 << 31
    return h, lo


def _limbs(x):
    h = (x + (1 << (LB - 1))) >> LB
    return h, x - (h << LB)


def _sum(products):
    h = m = 0
    for (ah, al), (xh, xl) in products:
        h += ah * xh
        m += ah * xl + al * xh
        assert abs(h) < I64 and abs(m) < I64
    return h, m


def _row(words, ea, x):
    """sum of the words and the real entries x as k_apply_asm forms it."""
    fac = []
    for v in x:
        m, ev, neg = _bits(v)
        fac.append((_limbs((-m if neg else m) << 5), ev if m else -20000))
    S, E = 0, -40000
    for half in (0, 15):
        for g0 in (half, half + GS):
            idx = range(g0, min(g0 + GS, half + 15))
            C = max([fac[i][1] - words[i][1] for i in idx] + [-40000])
            h, m = _sum((_take(words[i], C - fac[i][1] + words[i][1]), fac[i][0]) for i in idx)
            s = (h << 2) + (m >> (LB - 2))
            S = (S >> min(max(C - E, 0), 64)) + (s >> min(max(E - C, 0), 64))
            E = max(E, C)
            assert abs(S) < 1 << 62
    return Fraction(S) * _pow2(ea + E - 2101)


def _fp64(a, x):
    s = 0.0
    for av, xv in zip(a, x):
        s = math.fma(av, xv, s) if hasattr(math, "fma") else s + av * xv
    return Fraction(s)


# products of 53-bit values; the shift of a value leaves 2^-57 of the largest
# product's power of two, the lo lo products 2^-54, the alignment of the four
# groups and their last bit 2^-55 each: below 30 x 2^-54 + 8 x 2^-55 of four
# times the largest product in the worst case; the typical row is held to
# FP64's own unit, 2^-52 of the sum of the magnitudes
@pytest.mark.parametrize("sa", [0, 10, 60])
@pytest.mark.parametrize("sx", [0, 10, 60, 300])
def test_rows(sa, sx):
    rng = np.random.default_rng(100 * sa + sx)
    for _ in range(60):
        a = rng.uniform(-1, 1, 30) * 2.0 ** rng.uniform(-sa, 0, 30)
        x = rng.uniform(-1, 1, 30) * 2.0 ** rng.uniform(-sx, 0, 30)
        e = max(_bits(v)[1] for v in a) + 1
        got = _row([_word(v, e) for v in a], e, x)
        terms = [Fraction(float(p)) * Fraction(float(q)) for p, q in zip(a, x)]
        assert abs(got - sum(terms)) <= _pow2(-52) * sum(map(abs, terms))


def test_opposed_powers():
    """Entries that fall along the row against entries that rise: the products
    are all of one size, far below the largest value times the largest entry."""
    rng = np.random.default_rng(1)
    for step in (1, 2, 4):
        a = rng.uniform(0.5, 1, 30) * 2.0 ** (-step * np.arange(30.0))
        x = rng.uniform(0.5, 1, 30) * 2.0 ** (step * np.arange(30.0))
        e = max(_bits(v)[1] for v in a)
        terms = [Fraction(float(p)) * Fraction(float(q)) for p, q in zip(a, x)]
        assert abs(_row([_word(v, e) for v in a], e, x) - sum(terms)) <= _pow2(-52) * sum(terms)


def test_largest_values_do_not_overflow():
    top = np.nextafter(2.0, 0.0)
    for sa in (1, -1):
        for sx in (1, -1):
            r = _row([_word(sa * top, 1023)] * 30, 1023, [sx * top] * 30)
            assert abs(r - sa * sx * 30 * Fraction(float(top)) ** 2) < Fraction(1, 2 ** 44)


def test_zero_entries():
    a = np.zeros(30)
    a[4] = 3.0
    x = np.zeros(30)
    assert _row([_word(v, 1025) for v in a], 1025, x) == 0
    x[4] = 5.0
    assert abs(_row([_word(v, 1025) for v in a], 1025, x) - 15) <= 15 * _pow2(-52)


def _bound(v):
    """upper 16 bits of a double >= |v|"""
    b = int(np.float64(abs(v)).view(np.uint64))
    return (b + (1 << 48) - 1) >> 48


def _assemble(kwords, ek, w, ea):
    """word of sum_ia w_ia K_ia as k_assemble forms it."""
    fac = []
    for v in w:
        m, ev, neg = _bits(v)
        fac.append((_limbs((-m if neg else m) << 4), ev if m else ZERO))
    keys = [f[1] + e - k[1] for f, e, k in zip(fac, ek, kwords)]
    C = max(keys)
    h, m = _sum((_take(k, C - key), f[0]) for k, key, f in zip(kwords, keys, fac))
    S = (h << 5) + (m >> (LB - 5))
    assert abs(S) < 1 << 61
    z = 64 - (S ^ (S >> 63)).bit_length()
    off = ea + 1017 - C + z
    if S == 0 or off >= OFF + 56:
        return 0, OFF
    T = (S << (z - 1)) >> max(off - OFF, 0)
    assert off >= 0 and -I64 <= T < I64
    return (T & ~127, min(off, OFF)) if T else (0, OFF)


@pytest.mark.parametrize("spread", [0, 8, 50])
def test_assembled_values(spread):
    """A value from its three factors to FP64's unit of its largest term,
    2^-52, with the row's exponents of the three tables far apart and a
    factor that is zero."""
    rng = np.random.default_rng(spread)
    for trial in range(200):
        rows = rng.uniform(-1, 1, (3, 5)) * 2.0 ** rng.uniform(-spread, 0, (3, 5)) * 2.0 ** rng.integers(-40, 40, (3, 1))
        rows[rng.integers(3), rng.integers(5)] = 0.0
        w = rng.uniform(-1, 1, 3) * 2.0 ** rng.uniform(-spread, 0, 3)
        if trial % 3 == 0:
            w[rng.integers(3)] = 0.0
        bits = [_bound(np.abs(r).max()) for r in rows]
        ek = [max(u >> 4, 1) for u in bits]
        b = 0.0
        for wv, u in zip(w, bits):
            b += abs(wv) * float(np.uint64(u << 48).view(np.float64))
        ea = _bits(b)[1] + 1
        for t in range(5):
            word = _assemble([_word(r[t], e) for r, e in zip(rows, ek)], ek, w, ea)
            terms = [Fraction(float(p)) * Fraction(float(r[t])) for p, r in zip(w, rows)]
            got = Fraction(word[0] >> 7) * _pow2(ea - 1078 - word[1])
            assert abs(got - sum(terms)) <= _pow2(-52) * max(map(abs, terms))
            # three quarters of the words' 57 bits are in use wherever the terms do not cancel
            if word[1] < OFF and abs(sum(terms)) > max(map(abs, terms)) / 8:
                assert 1 << 55 <= abs(word[0] >> 7) <= 1 << 56


def test_zero_factors_give_zero_words():
    assert _assemble([_word(v, 1023) for v in (1.0, 0.5, 0.25)], [1023] * 3, np.zeros(3), 1) == (0, OFF)
    assert _assemble([(0, OFF)] * 3, [1023] * 3, np.ones(3), 1025) == (0, OFF)
