"""The division-free quotients of the list builders: RN(a y) corrected by one
exact remainder equals the IEEE quotient a / d for y = RN(1 / d) (the formula
of `quotient` in hfx_gb300/csrc/lists_device.cuh), in exact rational
arithmetic with one rounding per operation."""
from fractions import Fraction

import numpy as np
import pytest


def _rn(x: Fraction) -> np.float32:
    return np.float32(float(x))


@pytest.mark.parametrize("d", [1.0005079, 0.02, 0.0137, 1.0, 2.0, 3.0, 4.0])
def test_corrected_quotient_is_the_ieee_quotient(d):
    d = np.float32(d)
    y = np.float32(1.0) / d
    rng = np.random.default_rng(7)
    bits = rng.integers(np.float32(2.0 ** -12).view(np.uint32), np.float32(2.0 ** 22).view(np.uint32), 4000)
    near = (np.arange(2000, dtype=np.float32) + np.float32(0.5)) * d  # quotients near half-integers
    for a in np.concatenate([bits.astype(np.uint32).view(np.float32), near, -near[:50]]):
        q = _rn(Fraction(float(a)) * Fraction(float(y)))
        rem = _rn(Fraction(float(a)) - Fraction(float(q)) * Fraction(float(d)))
        got = _rn(Fraction(float(rem)) * Fraction(float(y)) + Fraction(float(q)))
        assert got == a / d, (a, got, a / d)
