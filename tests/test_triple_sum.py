"""Host replay of the epilogue sums of the tensor-core block product (ts_add and ts_round in
dynemol_gb300/csrc/df64.cuh, FP32 round-to-nearest throughout): the partial products of a
K split summed as FP32 triples, doubled, less the vector before last, and rounded to FP32.
Against exact sums it is never further off than the same in FP64, and it rounds to nearest
within 2^-60 of the largest term."""
import os
import re
from fractions import Fraction

import numpy as np
import pytest

SRC = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dynemol_gb300", "csrc",
                        "df64.cuh")).read()
f32 = np.float32


def two_sum(a, b):
    s = a + b
    z = s - a
    return s, (a - (s - z)) + (b - z)


def ts_add(s, y):
    s0, y = two_sum(s[0], y)
    s1, y = two_sum(s[1], y)
    return s0, s1, s[2] + y


def ts_round(a, b, c):
    a, b = two_sum(a, b)
    b, c = two_sum(b, c)
    bits = b.view(np.int32)
    step = np.where((bits ^ c.view(np.int32)) < 0, np.int32(-1), np.int32(1))
    odd = np.where((c != 0) & (bits & 1 == 0), bits + step, bits).astype(np.int32)
    return a + odd.view(f32)


def test_replay_is_the_source():
    body = re.sub(r"\s+", " ", SRC)
    assert "two_sum(s[0], y); two_sum(s[1], y); s[2] = __fadd_rn(s[2], y);" in body
    assert "two_sum(a, b); two_sum(b, c); int i = __float_as_int(b);" in body
    assert "if (c != 0.f && !(i & 1)) i += (i ^ __float_as_int(c)) < 0 ? -1 : 1;" in body
    assert "return __fadd_rn(a, __int_as_float(i));" in body


def _cases(kind, rng, n, m):
    y = rng.standard_normal((n, m)).astype(f32)
    w = rng.standard_normal(m).astype(f32)
    if kind == "spread":      # partial products of very different size
        y *= np.ldexp(f32(1), rng.integers(-30, 1, (n, m))).astype(f32)
    if kind == "cancel":      # 2 y close to w
        w = (2.0 * y.astype(np.float64).sum(0)).astype(f32)
        w = np.where(rng.random(m) < 0.5, w, np.nextafter(w, f32(0)))
    if kind == "tie":         # half a last place of the rest, then a small last partial
        y[-1] = np.ldexp(f32(1), -40) * rng.choice([-1, 0, 1], m).astype(f32)
        if n > 1:
            y[0] = 1.0 + np.ldexp(f32(1), -23) * rng.integers(0, 8, m).astype(f32)
            y[1:-1] = 0.0
            y[min(1, n - 1)] += np.ldexp(f32(1), -24) if n > 2 else f32(0)
        w = np.zeros(m, f32)
    return y, w


@pytest.mark.parametrize("kind", ["plain", "spread", "cancel", "tie"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 10, 16])
def test_no_further_off_than_fp64(kind, n):
    rng = np.random.default_rng(n + 100 * len(kind))
    m = 1500
    y, w = _cases(kind, rng, n, m)
    s = (y[0], np.zeros(m, f32), np.zeros(m, f32))
    for q in range(1, n):
        s = ts_add(s, y[q])
    first = ts_round(*s)
    s = tuple(f32(2) * x for x in s)
    v = ts_round(*ts_add(s, -w))
    y64 = np.zeros(m)
    for q in range(n):
        y64 = y64 + y[q].astype(np.float64)
    v64 = (2.0 * y64 - w.astype(np.float64)).astype(f32)
    for got, ref, scale in ((first, y64.astype(f32), 0), (v, v64, 1)):
        assert got.dtype == f32
        for j in range(m):
            exact = sum((Fraction(float(x)) for x in y[:, j]), Fraction(0))
            if scale:
                exact = 2 * exact - Fraction(float(w[j]))
            e, e64 = abs(Fraction(float(got[j])) - exact), abs(Fraction(float(ref[j])) - exact)
            assert e <= e64 or e - e64 <= Fraction(1, 2 ** 60) * max(abs(Fraction(float(x))) for x in y[:, j])
            near = Fraction(float(np.spacing(np.abs(got[j])))) / 2 if got[j] else Fraction(0)
            big = max([abs(Fraction(float(x))) for x in y[:, j]] + [abs(Fraction(float(w[j])))])
            assert e <= near + Fraction(1, 2 ** 60) * big
