"""The factorisation's diagonal-block leaf (one cluster of four CTAs) over block counts
and remainders, through the drop-in's H' = S^-1 h and its positive-definiteness check."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H_BAR = 6.58264e-4


def _system(n, seed=0):
    rng = np.random.default_rng(1000 * seed + n)
    x = rng.standard_normal((n, n))
    S = x @ x.T / n + 0.5 * np.eye(n)
    h = rng.standard_normal((n, n))
    return S, (h + h.T) / 2


def _call(elhl, S, h):
    n = len(S)
    z = np.ones(n, complex) / np.sqrt(n)
    return elhl.propagationelhl_gpucaller(S, h, z.copy(), z.copy(), 0.0, 1e-6, 1e-6 / H_BAR)


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 33, 40, 48, 55, 56, 57, 63, 64, 65, 72, 127, 129])
def test_h_prime_and_ao_bra(elhl, n):
    """S^-1 h = G^T (G h) and AO_bra = S^-1 bra: relative 1e-11, cond(S) <= 30 times some
    n roundings of 1e-16 on both sides."""
    S, h = _system(n)
    Hp, ao_bra, bra, _, _ = _call(elhl, S, h)
    ref = np.linalg.solve(S, h)
    assert np.abs(Hp - ref).max() <= 1e-11 * np.abs(ref).max()
    ao = np.linalg.solve(S, bra)
    assert np.abs(ao_bra - ao).max() <= 1e-11 * np.abs(ao).max()


@pytest.mark.parametrize("n,bad", [(1, 0), (9, 8), (64, 0), (64, 37), (64, 63), (130, 100)])
def test_non_positive_pivot_is_reported(elhl, n, bad):
    """A leading block that stops being positive definite at one column ends the call with
    ELHL_ERR_NOT_POSITIVE_DEFINITE, and the next call works."""
    S, h = _system(n, seed=1)
    T = S.copy()
    T[bad, bad] = -1.0
    with pytest.raises(elhl.ElhlError) as e:
        _call(elhl, T, h)
    assert e.value.status == elhl.ERR_NOT_PD
    _call(elhl, S, h)
