"""div_const (st_spix_gb300/csrc/k_color.cu) rounds x / b correctly for every x that neither
over- nor underflows, for each of its constants.

With y = RN(1 / b), q = RN(x y), r = x - b q (exact) the result is RN(q + r y).  With the
relative error d <= 2^-53 of y, |x / b - q| <= (x / b) (d + 2^-53), so q + r y differs from x / b
by at most (x / b) d (d + 2^-53), which is at most 4 2^-53 of half an ulp.  A quotient of
53-bit integers X 2^s / B that is not itself a midpoint M (an odd 54-bit integer) lies
|X 2^s - M B| / B > k 2^-53 from it for k = |X 2^s - M B|: only X with k <= 4 can round
wrongly.  All of them (up to k = 8) are tried in exact arithmetic."""
import math
import os
import re
from fractions import Fraction

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CONSTANTS = (12.92, 1.055, 116.0, 0.950456, 1.088754)


def div_const(x, b):
    y = 1.0 / b
    q = x * y
    r = Fraction(x) - Fraction(b) * Fraction(q)
    assert Fraction(float(r)) == r                  # the first fused multiply-add is exact
    return float(Fraction(q) + r * Fraction(y))


def nearest_to_midpoints(b, kmax):
    """The 53-bit integers X whose quotient by b's mantissa lies nearest to a midpoint."""
    B = int(math.frexp(b)[0] * 2 ** 53)
    out = []
    for s in (53, 54):                              # X 2^s / B in [2^53, 2^54)
        g = math.gcd(2 ** s, B)
        n = B // g
        for k in range(-kmax, kmax + 1):
            if k == 0 or k % g:
                continue
            x = (k // g) * pow(2 ** s // g, -1, n) % n
            for X in range(x + -(-(2 ** 52 - x) // n) * n, 2 ** 53, n):
                M = (X * 2 ** s - k) // B
                if M % 2 and 2 ** 53 <= M < 2 ** 54:
                    out.append(X)
    return out


@pytest.mark.parametrize("b", CONSTANTS)
def test_quotients_nearest_to_a_midpoint(b):
    y = Fraction(1.0 / b)
    d = abs(y * Fraction(b) - 1)
    assert d <= Fraction(1, 2 ** 53) and 2 * d * (d + Fraction(1, 2 ** 53)) * 2 ** 53 <= Fraction(8, 2 ** 53)
    for X in nearest_to_midpoints(b, 8):
        for e in (-60, -52, 0, 40):
            x = math.ldexp(X, e)
            assert div_const(x, b) == x / b and div_const(-x, b) == -x / b


def test_the_constants_are_those_of_the_conversion():
    with open(os.path.join(ROOT, "st_spix_gb300", "csrc", "k_color.cu")) as f:
        src = f.read()
    used = set(re.findall(r"DIV_CONST\([^;]*?, ([0-9.]+)\)", src))
    assert {float(u) for u in used} == set(CONSTANTS)
