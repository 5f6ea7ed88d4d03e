"""CPU: the double-float arithmetic of the mixed projection's right-hand side
(df_split_bits and df_dot in step.cu), restated in exact integers and in numpy."""
from fractions import Fraction

import numpy as np
import pytest

f32 = np.float32


def split_bits(x):
    """df_split_bits on the bits of x: (hi, lo) as float32."""
    b = int(np.float64(x).view(np.uint64))
    hi, lo, sg = (b >> 32) & 0x7FFFFFFF, b & 0xFFFFFFFF, b >> 63
    e = hi >> 20
    rest = lo & 0x1FFFFFFF
    up = rest >> 28
    m = (((hi & 0xFFFFF) << 3) | (lo >> 29)) + up
    fe = e - 896
    if e >= 896 + 255:
        return f32(np.nan), f32(np.nan)
    h = np.uint32((sg << 31) | ((fe << 23) + m if fe > 0 else 0)).view(f32)
    rb = int(f32(rest - (up << 29)).view(np.uint32))
    le = ((rb >> 23) & 0xFF) + e - 1075
    if rb == 0 or le <= 0:
        return h, f32(0)
    return h, np.uint32(((rb + ((e - 1075) << 23)) & 0xFFFFFFFF) ^ (sg << 31)).view(f32)


def test_split_keeps_49_bits():
    rng = np.random.default_rng(3)
    xs = list(rng.standard_normal(4000) * 10.0 ** rng.uniform(-25, 30, 4000))
    xs += [0.0, -0.0, 1.0, -1.0, 1.0 - 2.0 ** -53, 1.0 + 2.0 ** -24, 1.0 + 2.0 ** -52, 2.0 ** 24 - 0.5]
    for x in xs:
        h, l = split_bits(x)
        assert abs(Fraction(float(h)) - Fraction(x)) <= Fraction(abs(float(h))) / 2 ** 24
        # lo is the rest rounded to 24 bits
        assert abs(Fraction(float(h)) + Fraction(float(l)) - Fraction(x)) <= abs(Fraction(x)) / 2 ** 48
    for x in (np.inf, -np.inf, np.nan, 1e39):
        assert all(np.isnan(split_bits(x)))
    assert split_bits(1e-45) == (0, 0)


def _fma(a, b, c):
    """float32 fma of arrays: the product is exact in float64, the sum is in long double."""
    return (np.longdouble(a) * np.longdouble(b) + np.longdouble(c)).astype(f32)


@pytest.mark.parametrize("n", [1, 2, 17, 49, 97])
def test_bounded_dot_product(n):
    rng = np.random.default_rng(n)
    cols = 400
    a = rng.standard_normal(n) * 10.0 ** rng.uniform(-3, 3, n)
    b = rng.standard_normal((n, cols)) * 10.0 ** rng.uniform(-6, 3, (n, cols))
    q = 2.0 ** rng.integers(0, 8, n)  # level weights
    bound = 2.0 ** np.ceil(np.log2(np.sum(np.abs(a) / q)))
    ah, bh = a.astype(f32), b.astype(f32)
    al, bl = (a - ah).astype(f32), (b - bh).astype(f32)
    cm = 2.0 ** (np.floor(np.log2(np.max(np.abs(bh) * f32(1) * q[:, None].astype(f32), axis=0))) + 1)
    c = (3 * cm * bound).astype(f32)
    hi, lo = c.copy(), np.zeros(cols, f32)
    for j in range(n):
        t = _fma(ah[j], bh[j], hi)
        z = hi - t
        lo = lo + _fma(ah[j], bh[j], z)
        lo = _fma(ah[j], bl[j], lo)
        lo = _fma(al[j], bh[j], lo)
        hi = t
        assert np.all(hi >= c / 3 * 2) and np.all(hi <= c / 3 * 4)  # the start stays the larger addend
    got = np.longdouble(hi - c) + np.longdouble(lo)
    exact = np.sum(np.longdouble(a)[:, None] * np.longdouble(b), axis=0)
    # per term 2^-23 of the bound goes to lo (|hi| < 4 cm bound, half an ulp),
    # so lo stays below n 2^-22 cm bound and each of its 3 roundings below
    # 2^-24 of that; the operands' own 2^-48 and lo lo add 2^-46 of the terms
    tol = (3 * n * n * 2.0 ** -46 + 2.0 ** -45) * cm * bound
    assert np.all(np.abs(got - exact) <= tol)
