"""z / q of the training network's silu (silu_f in mmff_mlp.cu), restated with exactly
rounded FP32 operations: Markstein's correction of z times the rounded reciprocal gives
the exactly rounded quotient in all but rare cases, and never misses it by more than one
unit in the last place."""
import math
import random
from fractions import Fraction

import numpy as np

f32 = np.float32


def rnd(x):
    """Fraction -> FP32, round to nearest (through FP64: inexact twice only within 2^-29 of a tie)."""
    return f32(float(x))


def test_corrected_quotient():
    rng = random.Random(3)
    off = 0
    n = 4000
    for _ in range(n):
        z = f32(rng.choice([rng.uniform(-60, 60), rng.uniform(-3, 3), rng.gauss(0, 0.1)]))
        q = f32(1) + f32(math.exp(-float(z)))
        if not q < f32(1e30):
            continue
        s = rnd(Fraction(1) / Fraction(float(q)))
        v = z * s
        r = rnd(Fraction(float(z)) - Fraction(float(q)) * Fraction(float(v)))
        got = rnd(Fraction(float(r)) * Fraction(float(s)) + Fraction(float(v)))
        want = rnd(Fraction(float(z)) / Fraction(float(q)))
        if got != want:
            off += 1
            assert abs(float(got) - float(want)) <= float(np.spacing(np.abs(want)))
    assert off <= n // 1000, off
