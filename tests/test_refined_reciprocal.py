"""The refined reciprocal of the f64 arithmetic, 1/x from a hardware
estimate r0 by r0 (1 + e + e^2), e = 1 - r0 x, each operation one rounding
(fused multiply-adds): exact rational arithmetic shows its error for every
estimate within the documented bounds."""

from __future__ import annotations

from fractions import Fraction

import numpy as np
import pytest


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))   # Fraction -> float rounds correctly


def refined(x, r0):
    e = fma(-x, r0, 1.0)
    return fma(r0, fma(e, e, e), r0)


# (bits of the estimate's relative error, worst error of the result in ulp):
# f32 rcp.approx is within 2^-22 (its result and its operand rounded to f32
# included); the result is off by half an ulp for its own rounding and
# the iteration's e^3. rcp.approx.ftz.f64 keeps 20 mantissa bits of its operand
# and of its result: within 2^-19, e^3 is up to 2^-57, 1/16 ulp
@pytest.mark.parametrize("bits,ulp", [(22, 0.5 + 2.0 ** -12), (19, 0.5 + 2.0 ** -4 + 2.0 ** -12)])
def test_refined_reciprocal_error(bits, ulp):
    rng = np.random.default_rng(bits)
    x = np.concatenate([rng.uniform(1.0, 2.0, 400), 1.0 + np.arange(8) * 2.0 ** -52, 2.0 - np.arange(1, 8) * 2.0 ** -52])
    x = np.concatenate([x, x * 2.0 ** rng.integers(-100, 100, x.size)])
    for v in x:
        for err in (-1.0, 1.0, rng.uniform(-1, 1)):
            v = float(v)
            r0 = float(Fraction(1) / Fraction(v) * (1 + Fraction(err) * Fraction(1, 2 ** bits)))
            got = refined(v, r0)
            exact = Fraction(1) / Fraction(v)
            size = Fraction(float(np.spacing(float(exact))))
            assert abs(Fraction(got) - exact) <= Fraction(ulp) * size
