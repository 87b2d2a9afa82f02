"""Division by a constant as the stress kernel does it (reciprocal product,
remainder, one correction) gives the correctly rounded quotient: checked in
exact arithmetic for the constants it is used with."""
import math
import random
from fractions import Fraction

import pytest


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


@pytest.mark.parametrize("b", [3.0, 6.0, math.sqrt(3.0)])
def test_quotient_is_correctly_rounded(b):
    rb, rng = 1.0 / b, random.Random(7)
    for _ in range(20000):
        x = math.ldexp(rng.choice([-1, 1]) * (1 + rng.random()), rng.randint(-60, 60))
        q = x * rb
        assert fma(fma(-b, q, x), rb, q) == x / b
    for k in range(1, 2000):            # quotients next to powers of two, small multiples
        for x in (b * k, math.nextafter(b * k, 0.0), math.nextafter(b * k, math.inf), float(k)):
            q = x * rb
            assert fma(fma(-b, q, x), rb, q) == x / b
    assert math.sqrt(3.0) == 1.7320508075688772
