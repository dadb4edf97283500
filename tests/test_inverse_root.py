"""The FP64 inverse root of the grid build and the FIRE scalars (inv_sqrt64 in
mmff_device.cuh), restated with exactly rounded operations: from an approximate root
within 2^-19 of the exact one, its one series step ends within one unit in the last
place, the bound that is stated there."""
import math
import random
from fractions import Fraction

import numpy as np


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def inv_sqrt64(x, y):
    e = fma(-(x * y), y, 1.0)
    return fma(y * e, fma(e, fma(e, 0.3125, 0.375), 0.5), y)


def test_series_step_is_within_one_unit():
    rng = random.Random(1)
    worst = 0.0
    for _ in range(3000):
        x = math.exp(rng.uniform(math.log(1e-6), math.log(1e6)))
        d = rng.choice([rng.uniform(-2.0 ** -19, 2.0 ** -19), 2.0 ** -19, -2.0 ** -19])
        r = inv_sqrt64(x, (1.0 / math.sqrt(x)) * (1.0 + d))
        # 200 bits of the exact value
        n = Fraction(1) / Fraction(x)
        k = 1 << 200
        exact = Fraction(math.isqrt(n.numerator * k * k // n.denominator), k)
        worst = max(worst, float(abs(Fraction(r) - exact) / Fraction(float(np.spacing(r)))))
    assert worst <= 1.0, worst
