"""The step of inv_sqrt_to_float (csrc/wd_device.cuh), restated with exactly rounded arithmetic: where its guard lets the result through, the result is that of
(float)(1.0 / sqrt(z)), for every estimate within 2^-21, with z next to the arguments whose result lies between two floats."""
import math
import random
from fractions import Fraction

import numpy as np

GUARD = 64


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))      # float() of a fraction rounds to nearest


def step(z, y):
    e = fma(-(z * y), y, 1.0)
    return fma(y * e, fma(e, 0.375, 0.5), y)


def lets_through(r):
    low = int(np.array([r], np.float64).view(np.uint64)[0]) & 0x1fffffff
    return (low - (0x10000000 - GUARD)) % (1 << 32) > 2 * GUARD


def test_what_the_guard_lets_through_rounds_as_the_expression():
    rng = random.Random(5)
    guarded = 0
    for _ in range(400):
        m = np.float32(math.ldexp(rng.uniform(1.0, 2.0), rng.randint(-49, 49)))
        middle = (Fraction(float(m)) + Fraction(float(np.nextafter(m, np.float32(np.inf))))) / 2
        z0 = float(1 / (middle * middle))                       # 1 / sqrt(z0) is next to the middle between two floats
        for k in (0, 1, -1, 2, -3, 9, -40, 300, -5000, rng.randint(-10**7, 10**7)):
            z = z0
            z = float(np.array([np.array([z0]).view(np.int64)[0] + k], np.int64).view(np.float64)[0])
            want = np.float32(1.0 / math.sqrt(z))
            for err in (0.0, 2.0**-21, -2.0**-21, rng.uniform(-1, 1) * 2.0**-22):
                y = float(np.float32((1.0 + err * 0.9) / math.sqrt(z)))
                r = step(z, y)
                if lets_through(r):
                    assert np.float32(r) == want
                else:
                    guarded += 1
    assert guarded > 1000                                       # the arguments next to a middle take the expression itself
