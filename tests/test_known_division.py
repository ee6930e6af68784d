"""Division by a known divisor (setup.cu: div_known): a (1/b) in two operations,
1/b held in two doubles, against the correctly rounded quotient.  The sum before
its rounding is off by 2^-105 of the quotient, so a quotient of random operands
rounds the other way once in 2^52 times; the sum is formed exactly here."""
from fractions import Fraction as Fr

import numpy as np


def _fma(a, b, c):
    return float(Fr(a) * Fr(b) + Fr(c))


def test_quotients_are_the_divisions():
    rng = np.random.default_rng(0)
    for b in np.concatenate([rng.uniform(0.01, 1.0, 40), np.sqrt(rng.uniform(1e-4, 2.0, 40)), [0.5, 0.05, 1.0 / 34.0]]):
        b = float(b)
        zh = 1.0 / b
        zl = _fma(-b, zh, 1.0) * zh
        for a in np.concatenate([rng.uniform(-1.0, 1.0, 100) * b, rng.standard_normal(100), [0.0, b, -b, 1.0]]):
            a = float(a)
            assert _fma(a, zh, a * zl) == a / b, (a, b)
