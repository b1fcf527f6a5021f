"""The short quotient of csrc/cvlbm_math.cuh (quot) rounds as the division does.

The device forms a/b from y = RN(1/b) and e = RN(RN(1 - b y) y) with two fused
multiply-adds.  Here the same steps run in exact rational arithmetic (every
rounding is the correctly rounded conversion of a Fraction to a float), on random
operands and on the ones that are hard for such a scheme: significands at both
ends of the binade, divisors next to powers of two, quotients next to a midpoint.
"""

from __future__ import annotations

from fractions import Fraction as Fr

import numpy as np


def fma(a, b, c):
    return float(Fr(a) * Fr(b) + Fr(c))


def quot(a, b):
    y = 1.0 / b
    e = fma(-b, y, 1.0) * y
    q = fma(a, y, a * e)
    return fma(fma(-b, q, a), y, q)


def _operands():
    rng = np.random.default_rng(5)
    hard = [1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 1.5, 4.0 / 3.0, 1.0 + 2.0 ** -26,
            1.0 + 2.0 ** -27, 2.0 - 2.0 ** -26, float(np.nextafter(1.5, 2.0))]
    for a in hard:
        for b in hard:
            yield a, b
            yield -a * 2.0 ** 40, b * 2.0 ** -30
    for _ in range(4000):
        yield (float(rng.uniform(1, 2) * 2.0 ** rng.integers(-850, 800)),
               float(rng.choice((-1, 1)) * rng.uniform(1, 2) * 2.0 ** rng.integers(-99, 99)))
    for _ in range(2000):  # a next to the product of b and a midpoint between two doubles
        b = float(rng.uniform(1, 2))
        m = Fr(float(rng.uniform(1, 2))) + Fr(1, 2 ** 53)
        a = float(m * Fr(b))
        yield a, b
        yield float(np.nextafter(a, 4.0)), b
    for k in range(1, 400):  # the constants of the solvers: steps, lattice constants, weights
        yield 1.1 / k, 1.0 + k * 1e-5
        yield float(rng.uniform(-1, 1)), 2.0 * (1.1 / (60 + k))
        yield float(rng.uniform(-1, 1)), 6.0


def test_quotient_rounds_as_the_division():
    for a, b in _operands():
        assert quot(a, b) == a / b, (a.hex(), b.hex())


def test_zero_numerator():
    for b in (3.0, -7.0, 1.0 + 2.0 ** -52):
        assert quot(0.0, b) == 0.0 and quot(-0.0, b) == 0.0
