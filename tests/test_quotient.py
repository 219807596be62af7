"""The quotient by a stored reciprocal (mg_tail.cuh, quotient()): two residual
corrections of n * (1/d) give the correctly rounded n / d, restated here in exact
arithmetic for both precisions over random and awkward operands, and its stated
limits: near the subnormal range the last bits may differ, an infinite numerator
gives NaN."""
import math
from fractions import Fraction

import numpy as np
import pytest


def rounded(x, T):
    """A fraction rounded to nearest in T (double: Python's own rounding)."""
    if T is np.float64:
        return np.float64(float(x))
    if x == 0:
        return np.float32(0)
    e = max(math.frexp(float(x))[1] - 24, -149)  # the spacing of floats at x
    k = x / (Fraction(2) ** e)
    return np.float32(float(Fraction(round(k)) * Fraction(2) ** e))  # (round: ties to even)


def fma(a, b, c, T):
    return rounded(Fraction(float(a)) * Fraction(float(b)) + Fraction(float(c)), T)


def quotient(n, d, T):
    r = T(1) / d
    q = n * r
    q = fma(fma(-q, d, n, T), r, q, T)
    return fma(fma(-q, d, n, T), r, q, T)


def operands(T, rng):
    top = 2.0 ** (52 if T is np.float64 else 23)
    mant = [1.0, 2 - 1 / top, 1 + 1 / top, 1.5, 4 / 3, 5 / 3] + list(1 + rng.random(400))
    for a in mant:
        for b in rng.choice(mant, 8):
            yield T(a * 2.0 ** rng.integers(-40, 40) * rng.choice([-1, 1])), T(b * 2.0 ** rng.integers(-40, 40) * rng.choice([-1, 1]))


@pytest.mark.parametrize("T", [np.float64, np.float32])
def test_equals_the_division(T):
    for n, d in operands(T, np.random.default_rng(5)):
        assert quotient(n, d, T) == n / d, (n, d)
    assert quotient(T(0), T(-3), T) == 0


@pytest.mark.parametrize("T", [np.float64, np.float32])
def test_near_the_subnormal_range(T):
    """Within two spacings of the subnormals, where the residual underflows."""
    rng = np.random.default_rng(6)
    info = np.finfo(T)
    for _ in range(500):
        n = T(info.tiny * rng.uniform(0.01, 8))
        d = T(rng.uniform(1, 4) * 2.0 ** rng.integers(-3, 4))
        assert abs(float(quotient(n, d, T)) - float(n) / float(d)) <= max(2 * float(info.smallest_subnormal), 2 * float(np.spacing(n / d)))


def test_infinite_numerator_is_not_finite():
    with np.errstate(invalid="ignore"):
        q = np.float64(np.inf) * (np.float64(1) / np.float64(3))
        assert not np.isfinite(-q * np.float64(3) + np.float64(np.inf))
