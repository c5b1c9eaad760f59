"""The generator's quotient dist / beta as one product and one correction by its
exact residual: equal to the correctly rounded division (exact rationals stand
in for the fused multiply-adds)."""
from fractions import Fraction

import numpy as np
import pytest


def _quotient(d, b):
    rb = 1.0 / b
    x = d * rb
    residual = float(Fraction(d) - Fraction(x) * Fraction(b))  # fma(-x, b, d)
    return float(Fraction(x) + Fraction(residual) * Fraction(rb))  # fma(residual, rb, x)


@pytest.mark.parametrize("scale", [1e-150, 1e-3, 1.0, 1e120])
def test_corrected_product_is_the_correctly_rounded_quotient(scale):
    rng = np.random.default_rng(5)
    for _ in range(4000):
        b = float(np.exp(rng.uniform(np.log(1e-3), np.log(50.0)))) * scale
        x = float(np.exp(rng.uniform(np.log(2.0 ** -20), np.log(2.0 ** 9))))  # the table's range
        d = x * b
        assert _quotient(d, b) == d / b
