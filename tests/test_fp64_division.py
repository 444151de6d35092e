"""Quotients of the FP64 sweeps (div_rn_geo, div_rn_3, div_rn_6 in
f3d_common.cuh), restated with exact rational arithmetic: correctly rounded
over the numerators that take the short way, its lower ends included."""
import math
import random
from fractions import Fraction

import pytest


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))  # one rounding, to nearest even


def _geo(a, b):
    y = 1.0 / b
    q = a * y
    q = _fma(_fma(-q, b, a), y, q)
    return _fma(_fma(-q, b, a), y, q)


def _known(a, z):
    return _fma(a, z, a * (z * 2.0 ** -54))


def _numerators(low, rng, n):
    for _ in range(n):
        yield rng.choice((-1, 1)) * (1.0 + rng.getrandbits(52) * 2.0 ** -52) * 2.0 ** rng.randint(low, 900)
    for m in (1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 1.5):
        yield m * 2.0 ** low


@pytest.mark.parametrize("b", [1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 5559.7463322, 250.0, 2.0 ** 100, 2.0 ** -100, 3e-7])
def test_by_a_spacing(b):
    rng = random.Random(1)
    for a in _numerators(-900, rng, 3000):
        if math.frexp(a / b)[1] < 1000:
            assert _geo(a, b) == float(Fraction(a) / Fraction(b)), (a, b)


def test_by_three_and_six():
    rng = random.Random(2)
    for a in _numerators(-960, rng, 20000):
        assert _known(a, float(Fraction(1, 3))) == float(Fraction(a) / 3), a
        assert _known(a, float(Fraction(1, 6))) == float(Fraction(a) / 6), a
