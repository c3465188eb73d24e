"""The two-operation quotient of kernels_brinkman.cu (br_div) equals the
correctly rounded x / d for every divisor its host rule (br_divisor) accepts:
the arithmetic modelled exactly with rationals."""
import math
import random
from fractions import Fraction

import pytest


def odd_part(d):
    m = int(math.ldexp(abs(math.frexp(d)[0]), 53))
    while m % 2 == 0:
        m //= 2
    return m


def quotient(x, d):
    zh = 1.0 / d
    zl = float(1 - Fraction(zh) * Fraction(d)) / d
    q1 = float(Fraction(x) * Fraction(zl))
    return float(Fraction(x) * Fraction(zh) + Fraction(q1))


@pytest.mark.parametrize("d", [6.0, 1.0e8 + 6.0, 1.0e5 + 6.0, 3.0, 7.5, -6.0, float(2 ** 40 - 1), 0.375])
def test_quotient_is_correctly_rounded(d):
    assert odd_part(d) < 2 ** 40
    rng = random.Random(int(abs(d)))
    xs = [math.ldexp(rng.uniform(1.0, 2.0), rng.randint(-599, 598)) * rng.choice((-1, 1)) for _ in range(4000)]
    # next to the rounding boundaries: neighbours of d times 54-bit odd numbers
    for _ in range(4000):
        x = float(Fraction(2 * rng.randrange(2 ** 52, 2 ** 53) + 1) * Fraction(d) / 2 ** rng.randint(0, 90))
        xs += [x, math.nextafter(x, math.inf), math.nextafter(x, -math.inf)]
    for x in xs:
        if 2.0 ** -600 <= abs(x) < 2.0 ** 600:
            assert quotient(x, d) == x / d
