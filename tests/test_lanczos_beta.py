"""lanczos_rows_kernel takes beta^2 as |p|^2 - alpha^2 where that keeps its digits and sums
|p - alpha q|^2 elsewhere.  Host replay at the line between the two (read from the source)
and on either side: beta is within four times the summed residual's rounding bound."""
import os
import re

import numpy as np
import pytest

SRC = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dynemol_gb300", "csrc",
                        "lanczos.cu")).read()


def _line():
    assert "s_sc[1] = b2 > kLrCancel * p2 ? 1.0 : 0.0;" in SRC
    return float(re.search(r"constexpr double kLrCancel = ([0-9.e-]+);", SRC).group(1))


@pytest.mark.parametrize("n", [62, 450, 1860])
@pytest.mark.parametrize("factor", [1e-10, 1e-4, 0.1, 0.999, 1.001, 2.0, 4.0])
def test_beta_keeps_its_digits(n, factor):
    rng = np.random.default_rng(n)
    ratio = _line() * factor  # beta^2 / |p|^2
    q = rng.standard_normal(n)
    q /= np.linalg.norm(q)
    r = rng.standard_normal(n)
    r -= (r @ q) * q
    r *= np.sqrt(ratio) / np.linalg.norm(r)
    p = np.sqrt(1.0 - ratio) * q + r
    alpha = p @ q
    p2 = p @ p
    b2 = p2 - alpha * alpha
    beta = np.sqrt(b2) if b2 > _line() * p2 else np.linalg.norm(p - alpha * q)
    pl, ql = p.astype(np.longdouble), q.astype(np.longdouble)
    exact = np.sqrt(np.sum((pl - np.sum(pl * ql) * ql) ** 2))
    # the residual's own rounding: one unit of |p| per element beside beta, pairwise sums
    bound = np.finfo(float).eps * (1.0 / np.sqrt(ratio) + 8.0)
    if ratio > _line():
        bound = 4 * np.finfo(float).eps * 8.0
    assert abs(beta - exact) <= bound * exact
