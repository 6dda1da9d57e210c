"""The window's depth gate without its quotient (k_statmc.cu, depth_far) against the quotient.

fl(num / m) > t, decided as fma(-t, m, num) > m h with h half an ulp of t, restated with exact
rationals: the fused difference is rounded once from its exact value. Pairs are drawn on and around
the threshold, where a rounding could flip the decision.
"""
from __future__ import annotations

import math
from fractions import Fraction

import numpy as np
import pytest

F32 = np.float32


def round_f32(x: Fraction) -> Fraction:
    """x rounded to the nearest single (ties to even; normal and subnormal range)."""
    if x == 0:
        return x
    s, a = (1, x) if x > 0 else (-1, -x)
    e = math.floor(math.log2(a.numerator) - math.log2(a.denominator)) - 1
    while Fraction(2) ** (e + 1) <= a:
        e += 1
    unit = Fraction(2) ** (max(e, -126) - 23)
    q, r = divmod(a, unit)
    if 2 * r > unit or (2 * r == unit and q % 2 == 1):
        q += 1
    return s * q * unit


@pytest.mark.parametrize("threshold", [0.2, 0.25, 0.1, 1.0, 0.33333334, 1e-3, 1e-21, 3.0000002])
def test_gate_equals_the_quotient(threshold):
    rng = np.random.default_rng(7)
    t = F32(threshold)
    h = Fraction(float(np.nextafter(t, F32(np.inf)))) / 2 - Fraction(float(t)) / 2
    for _ in range(1500):
        m = F32(rng.uniform(1.0, 2.0) * 2.0 ** rng.integers(-26, 20))
        num = F32(float(t) * float(m))
        for _ in range(int(rng.integers(0, 4))):  # the product, or a few ulps beside it
            num = np.nextafter(num, F32(np.inf) if rng.random() < 0.5 else F32(0))
        if rng.random() < 0.2:
            num = F32(float(num) * rng.uniform(0.0, 3.0))
        quotient = round_f32(Fraction(float(num)) / Fraction(float(m)))
        fused = round_f32(Fraction(float(num)) - Fraction(float(t)) * Fraction(float(m)))
        assert (fused > Fraction(float(m)) * h) == (quotient > Fraction(float(t))), (num, m, t)
