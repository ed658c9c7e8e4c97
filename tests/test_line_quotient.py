"""The line solve's quotient from a stored reciprocal (lsgs.cu:quotient) is the
correctly rounded a / b: its four operations in exact rational arithmetic,
rounded to 24 bits as the device rounds them, against the rounded quotient,
over the ranges in which the device uses it."""
import random
from fractions import Fraction

import pytest


def rn(x: Fraction) -> Fraction:
    """round to nearest even, 24 bits, FP32's exponents (subnormals too)"""
    if x == 0:
        return Fraction(0)
    s, x = (-1, -x) if x < 0 else (1, x)
    e = x.numerator.bit_length() - x.denominator.bit_length()
    while Fraction(2) ** e > x:
        e -= 1
    while Fraction(2) ** (e + 1) <= x:
        e += 1
    ulp = Fraction(2) ** (max(e, -126) - 23)
    q, r = divmod(x, ulp)
    q += 1 if r * 2 > ulp or (r * 2 == ulp and q % 2) else 0
    return s * q * ulp


def quotient(a, b):
    y = rn(1 / b)
    yl = rn(rn(1 - b * y) * y)
    q = rn(a * y + rn(a * yl))
    return rn(rn(a - b * q) * y + q)


def draw(r, lo, hi):
    m = r.choice([r.getrandbits(23), 0, 1, 2**23 - 1, 2**23 - 2, r.getrandbits(4), 2**23 - 1 - r.getrandbits(4)])
    return r.choice([1, -1]) * Fraction(2**23 + m) * Fraction(2) ** (r.randint(lo, hi) - 23)


@pytest.mark.parametrize("seed", range(4))
def test_quotient_is_correctly_rounded(seed):
    r = random.Random(seed)
    for _ in range(4000):
        b = draw(r, -36, 27)
        a = r.choice([draw(r, -74, 80), draw(r, -74, -70), rn(draw(r, -30, 30) * b)])
        assert quotient(a, b) == rn(a / b), (a, b)


@pytest.mark.parametrize("seed", range(4))
def test_quotient_of_small_operands(seed):
    """pivots down to 2^-100, dividends down to 2^-90"""
    r = random.Random(100 + seed)
    for _ in range(4000):
        b = draw(r, *r.choice([(-100, 27), (-100, -98), (26, 27)]))
        a = r.choice([draw(r, -90, 20), draw(r, -90, -88), rn(draw(r, -20, 20) * b)])
        if abs(a) >= Fraction(1, 2**90) and abs(a / b) < 2**120:  # overflow ends in a NaN
            assert quotient(a, b) == rn(a / b), (a, b)
