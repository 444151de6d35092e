"""The FP64 sweeps' quotients at small numerators (f3d_common.cuh), restated
with exact rational arithmetic: the short forms down to the limits the device
uses (div_small, kSmall36, read from the source), and the scaled form below
them, subnormal results and their ties included."""
import math
import os
import random
import re
from fractions import Fraction

import pytest

from fall3d_b200 import build as B
from tests.test_fp64_division import _fma, _geo, _known

SRC = open(os.path.join(B.CSRC, "f3d_common.cuh")).read()
NEAR, FAR = re.search(r"most <= 0x1p50 \? 0x1p(-\d+) : 0x1p(-\d+);", SRC).groups()
SMALL36 = re.search(r"kSmall36 = \(1023u - (\d+)u\) << 20", SRC).group(1)
RECIP36 = {3.0: float(Fraction(1, 3)), 6.0: float(Fraction(1, 6))}


def _scaled(a, b):
    y = 1.0 / b
    sa = a * 2.0 ** 400
    q = sa * y
    q = _fma(_fma(-q, b, sa), y, q)
    q = _fma(_fma(-q, b, sa), y, q)
    res = q * 2.0 ** -400
    rem, d = _fma(-q, b, sa), _fma(-res, 2.0 ** 400, q)
    if abs(d) == 2.0 ** -675 and rem != 0.0 and (d > 0.0) == ((rem > 0.0) == (b > 0.0)):
        res += math.copysign(2.0 ** -1074, d)
    return res


def _at(low, high, rng, n):
    for _ in range(n):
        yield rng.choice((-1, 1)) * (1.0 + rng.getrandbits(52) * 2.0 ** -52) * 2.0 ** rng.randint(low, high)
    for m in (1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 1.5):
        yield m * 2.0 ** low


@pytest.mark.parametrize("b", [1.0, 2.0 - 2.0 ** -52, 5559.7463322, 250.0, 2.0 ** 50, 1.9 * 2.0 ** 49, 2.0 ** -100, 3e-7,
                               2.0 ** 100, 1.1 * 2.0 ** 99])
def test_short_form_down_to_its_limit(b):
    rng = random.Random(3)
    low = int(NEAR if b <= 2.0 ** 50 else FAR)
    for a in _at(low, low + 60, rng, 4000):
        assert _geo(a, b) == float(Fraction(a) / Fraction(b)), (a, b)


def test_three_and_six_down_to_their_limit():
    rng = random.Random(4)
    for a in _at(-int(SMALL36), -int(SMALL36) + 60, rng, 20000):
        for b, z in RECIP36.items():
            assert _known(a, z) == float(Fraction(a) / Fraction(b)), a


@pytest.mark.parametrize("b", [3.0, 6.0, 1.0 + 2.0 ** -52, 5559.7463322, 250.0, 2.0 ** 50, 2.0 ** 100, 2.0 ** -100, 3e-7])
def test_scaled_form(b):
    rng = random.Random(5)
    shift = math.frexp(b)[1]
    for low, high in ((-1074, -1000), (-1074 + shift, -1010 + shift), (-700, 499)):
        if high < -1074:
            continue  # no such numerators: the quotient by this spacing is normal
        for _ in range(3000):
            e = rng.randint(max(low, -1074), high)
            a = math.ldexp(rng.choice((-1, 1)) * rng.randrange(1 << 52, 1 << 53), max(e - 52, -1126))
            if a and math.frexp(a / b)[1] < 990:
                assert _scaled(a, b) == float(Fraction(a) / Fraction(b)), (a, b)
    # quotients that lie at or beside the middle of two subnormals, and just below 2^-1022
    for _ in range(3000):
        k = rng.choice((rng.randrange(1, 1 << 52), rng.randrange(1, 64), (1 << 52) - 1, (1 << 52)))
        a = float(Fraction(b) * Fraction(2 * k + 1, 2) * Fraction(2) ** -1074)
        for c in (a, math.nextafter(a, math.inf), math.nextafter(a, 0.0)):
            if c:
                assert _scaled(c, b) == float(Fraction(c) / Fraction(b)), (c, b)
