"""The factorisation's smallest products (8 x 4 tiles, every eighth k per warp) over blocks
around their tiles, through the drop-in's H' = S^-1 h and S^-1 bra."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H_BAR = 6.58264e-4


@pytest.mark.parametrize("n", [2, 9, 65, 66, 68, 71, 73, 127, 128, 130, 190, 192, 193, 200, 255, 256, 257, 261, 320])
def test_factor_and_products(elhl, n):
    """Splits into blocks of 64 and a remainder of 1 to 64 rows.  Relative 1e-11: cond(S)
    <= 30 times some n roundings of 1e-16 on both sides."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, n))
    S = x @ x.T / n + 0.5 * np.eye(n)
    h = rng.standard_normal((n, n))
    h = (h + h.T) / 2
    z = np.ones(n, complex) / np.sqrt(n)
    Hp, ao_bra, bra, _, _ = elhl.propagationelhl_gpucaller(S, h, z.copy(), z.copy(), 0.0, 1e-6, 1e-6 / H_BAR)
    ref = np.linalg.solve(S, h)
    assert np.abs(Hp - ref).max() <= 1e-11 * np.abs(ref).max()
    ao = np.linalg.solve(S, bra)
    assert np.abs(ao_bra - ao).max() <= 1e-11 * np.abs(ao).max()
