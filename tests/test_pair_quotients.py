"""CPU check of the pair field's quotients (f64::recip, f64::quot) in exact arithmetic.

The device forms a / q, a / q^2 and a / q^3 of an image from one reciprocal y of q: the
squares' and cubes' reciprocals are y y and (y y) y, and a quotient is q0 = a y,
q0 + (a - b q0) y with fused multiply-adds.  Each must be the correctly rounded quotient,
except where a / b lies nearer to the middle of two doubles than the reciprocal's error
lets the last step tell apart: 2^-51, 2^-48 and 2^-47 of their distance.
"""
import math
import random
from fractions import Fraction as Fr

import pytest


def fma(a, b, c):
    return float(Fr(a) * Fr(b) + Fr(c))


def recip(b, seed_error):
    y = float(Fr(1) / Fr(b) * (1 + Fr(seed_error)))  # the hardware's estimate
    for _ in range(2):
        y = fma(y, fma(-b, y, 1.0), y)
    return y


def quot(a, b, y):
    q0 = a * y
    return fma(fma(-b, q0, a), y, q0)


def distance_to_middle(a, b, q):
    """Of a / b from the middle of the two doubles around it, in their distances."""
    exact = Fr(a) / Fr(b)
    low = q if Fr(q) <= exact else math.nextafter(q, -math.inf)
    high = math.nextafter(low, math.inf)
    return abs((exact - Fr(low)) / (Fr(high) - Fr(low)) - Fr(1, 2))


@pytest.mark.parametrize("power,bound", [(1, 2.0 ** -51), (2, 2.0 ** -48), (3, 2.0 ** -47)])
def test_quotients_correctly_rounded(power, bound):
    rng = random.Random(power)
    for _ in range(4000):
        q = math.exp(rng.uniform(math.log(1e-5), math.log(1e12)))
        if rng.random() < 0.2:
            q = math.nextafter(2.0 ** rng.randrange(-16, 40), rng.choice([0.0, math.inf]))
        y = recip(q, rng.uniform(-1, 1) * 2.0 ** -20)
        b, yb = q, y
        if power >= 2:
            b, yb = q * q, y * y
        if power == 3:
            b, yb = float(Fr(q) ** 3), yb * y  # (rounded once)
        a = rng.choice([-1, 1]) * math.exp(rng.uniform(math.log(1e-30), math.log(1e30)))
        got, want = quot(a, b, yb), float(Fr(a) / Fr(b))
        assert abs(got - want) <= math.ulp(want)
        assert got == want or distance_to_middle(a, b, got) <= bound
        # and beside a middle: a numerator whose quotient by b is next to one
        m = Fr(want) + Fr(math.ulp(want)) / 2
        a = float(m * Fr(b))
        got, want = quot(a, b, yb), float(Fr(a) / Fr(b))
        assert got == want or distance_to_middle(a, b, got) <= bound
