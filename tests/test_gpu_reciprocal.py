"""The reciprocal of the factorisation's pivots (factor.cu: one third-order Householder step
on the hardware's approximation, the division outside its window) against exact quotients
and CUDA's division.

With a start of 20 fraction bits, e = 1 - d y is below 2^-19 and exact, the terms left out
are below e^3 = 2^-57 of the result, at most an eighth of its last place's half, and the
last FMA rounds once: within 0.5 + 2^-57 / 2^-53 x 2 = 0.625 ulp of 1 / d, so at most one
unit beside the correctly rounded quotient."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mantissas(rng, n):
    m = 1.0 + rng.random(n)
    m[:8] = [1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), 1.5, 4.0 / 3.0, 1.0 + 2.0 ** -20, 1.25, 1.75]
    return m


# biased exponents: the window's edges 24 and 2020 from both sides, and between
@pytest.mark.parametrize("lo,hi", [(1, 23), (22, 26), (24, 1000), (1015, 1031), (1000, 2020), (2018, 2023), (2021, 2046)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_within_a_unit_of_the_quotient(elhl, lo, hi, sign):
    rng = np.random.default_rng(lo * 4096 + hi)
    n = 200_000
    x = sign * np.ldexp(_mantissas(rng, n), rng.integers(lo, hi + 1, n) - 1023)
    assert np.isfinite(x).all() and (np.abs(x) >= np.finfo(float).tiny).all()
    y, q = elhl.debug_reciprocal(x)
    assert np.array_equal(q, 1.0 / x)  # both correctly rounded
    assert np.abs(y.view(np.int64) - q.view(np.int64)).max() <= 1
    for i in range(0, n, n // 500):
        exact = 1 / Fraction(float(x[i]))
        ulp = Fraction(float(np.spacing(np.abs(q[i]))))
        assert abs(Fraction(float(y[i])) - exact) <= Fraction(5, 8) * ulp


def test_outside_the_window_is_the_division(elhl):
    tiny = np.finfo(float).tiny
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, tiny / 2, tiny, -tiny, np.finfo(float).max,
                  2.0 ** 1023, 2.0 ** -1022])
    y, q = elhl.debug_reciprocal(x)
    assert np.array_equal(y.view(np.int64)[~np.isnan(x)], q.view(np.int64)[~np.isnan(x)])
    assert np.isnan(y[np.isnan(x)]).all()
    with np.errstate(divide="ignore", over="ignore"):
        ref = 1.0 / x[~np.isnan(x)]
    assert np.array_equal(q[~np.isnan(x)], ref)
