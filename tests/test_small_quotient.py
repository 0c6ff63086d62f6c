"""small_quotient of kinship_mixed.cu: x r corrected once by its remainder, r the rounded 1 / d, is the
correctly rounded x / d for every integer |x| <= 128 and d = 254, 254^2 (the digits' weights), so that the
mixed form's sums are those of a division.  The device's operations (IEEE products and fused multiply-adds)
in exact rational arithmetic, rounded once each."""
from fractions import Fraction

import pytest


def small_quotient(x, d):
    r = 1.0 / d
    q = x * r
    rest = float(Fraction(-d) * Fraction(q) + Fraction(x))
    return float(Fraction(rest) * Fraction(r) + Fraction(q))


@pytest.mark.parametrize("d", [254, 254 * 254])
def test_correctly_rounded(d):
    for x in range(-128, 129):
        assert small_quotient(float(x), d) == float(Fraction(x, d))
