"""The division of the triangular factors: a quotient from the correctly
rounded reciprocal and one residual step (Markstein 1990) is the correctly
rounded quotient. Restated here with exact rationals for the two fused
operations."""
from fractions import Fraction

import numpy as np


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _div_by(a, b):
    r = 1.0 / b
    q = a * r
    return _fma(_fma(-q, b, a), r, q)


def test_quotient_is_correctly_rounded():
    rng = np.random.default_rng(3)
    m = 1.0 + rng.random((4000, 2))
    a = m[:, 0] * 2.0 ** rng.integers(-300, 300, 4000)
    b = m[:, 1] * 2.0 ** rng.integers(-40, 200, 4000)
    # mantissas next to one and two, where the reciprocal is least accurate
    edge = 1.0 + np.arange(-4, 5) * 2.0 ** -52
    a = np.concatenate([a * rng.choice([-1, 1], 4000), np.repeat(edge, 9)])
    b = np.concatenate([b, np.tile(edge, 9)])
    for x, y in zip(a.tolist(), b.tolist()):
        assert _div_by(x, y) == x / y
