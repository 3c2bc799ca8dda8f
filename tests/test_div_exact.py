"""The quotient the kernels form from a correctly rounded reciprocal (an
approximation and two corrections, Markstein 1990) is the correctly rounded
one: the same steps with exact rational arithmetic between the roundings."""
import random
from fractions import Fraction

import numpy as np


def rn(x):
    """Fraction rounded to the nearest float32, ties to even (normal range)."""
    if x == 0:
        return Fraction(0)
    s, x = (-1, -x) if x < 0 else (1, x)
    e = x.numerator.bit_length() - x.denominator.bit_length()
    if Fraction(2) ** e > x:
        e -= 1
    u = Fraction(2) ** (e - 23)
    n, r = divmod(x, u)
    if 2 * r > u or (2 * r == u and n % 2):
        n += 1
    return s * n * u


def div_exact(a, b, y):
    q = rn(a * y)
    q = rn(rn(a - b * q) * y + q)
    return rn(rn(a - b * q) * y + q)


def test_quotient_is_correctly_rounded():
    rng = random.Random(5)
    ones = (1 << 24) - 1
    mant = [1 << 23, (1 << 23) + 1, ones, ones - 1] + [rng.randrange(1 << 23, 1 << 24) for _ in range(60)]
    fixed = [Fraction(float(np.float32(v))) for v in (5.0, 32767.0, 0.02, 0.016, 0.032, 200.0, 125.0, 62.5, 1 / 0.005)]
    for b in fixed + [Fraction(m) for m in mant]:
        y = rn(1 / b)
        for m in mant + [rng.randrange(1 << 23, 1 << 24) for _ in range(40)]:
            for a in (Fraction(m), -Fraction(m) / 1024):
                assert div_exact(a, b, y) == rn(a / b), (a, b)


def test_every_16_bit_code():
    """code / 32767 of the 16-bit formats: one correction rounds every code's
    quotient correctly."""
    b = Fraction(32767)
    y = rn(1 / b)
    assert float(y) == float(np.float32(1.0) / np.float32(32767.0))
    for c in range(1, 32769):
        q = rn(c * y)
        assert rn(rn(c - b * q) * y + q) == rn(Fraction(c, 32767)), c
