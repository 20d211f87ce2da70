"""The FP64 fit's quotients from a reciprocal (div_by): restated with exactly rounded operations, equal to IEEE division."""
from fractions import Fraction

import numpy as np


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))      # one rounding to nearest even


def div_by(a, b):
    y = 1.0 / b
    q = a * y
    q = fma(fma(-q, b, a), y, q)
    return fma(fma(-q, b, a), y, q)


def test_quotients_equal_division():
    rng = np.random.default_rng(2)
    for _ in range(6000):
        a = float(rng.uniform(1, 2) * 2.0 ** rng.integers(-60, 60)) * (1 if rng.random() < 0.5 else -1)
        b = float(rng.uniform(1, 2) * 2.0 ** rng.integers(-20, 20))
        assert div_by(a, b) == a / b, (a, b)
    one = float(np.nextafter(1.0, 2.0))
    edge = [1.0, one, float(np.nextafter(2.0, 1.0)), 1.5, float(np.nextafter(1.5, 2.0)), 3.0, 19.0, 1.0 / 3.0]
    for a in edge:
        for b in edge:                                         # quotients next to a power of two and to halfway cases
            for k in (-3, 0, 7):
                assert div_by(a * 2.0 ** k, b) == a * 2.0 ** k / b, (a, b, k)
    for _ in range(2000):                                      # a = b * q rounded: quotients next to representable ones
        b, q = float(rng.uniform(5, 40)), float(rng.uniform(-60, 60))
        for a in (b * q, float(np.nextafter(b * q, 1e9)), float(np.nextafter(b * q, -1e9))):
            assert div_by(a, b) == a / b, (a, b)
