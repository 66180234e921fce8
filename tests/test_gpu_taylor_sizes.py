"""The Taylor kernel's forms over the sizes where they change, against the oracle.

H' stays in shared memory up to N = 1264 for one particle (the kernel's footprint:
pad8(N) (4 + 2 rows) doubles and the warps' sums, rows = ceil(N / 152), against
220 KB); above that the rows are read from L2 every round.  Below 304 rows fewer
CTAs than SMs take part (two rows each); eight rows are one epilogue unit, more
take several; columns come in groups of eight."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H_BAR = 6.58264e-4


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 31, 33, 303, 304, 305, 465, 1216, 1217, 1264, 1265])
def test_taylor_sizes_vs_oracle(elhl, oracle_mod, n):
    """One particle over several sub-steps with a non-symmetric H' (bra and ket see
    different matrices).  Same accepted tau; Psi to 1e-11: a run of at most a few
    hundred orders, each with rounding below 16 eps |H'| tau on vectors of norm 1
    (2e-15 times 300 orders, times an order of magnitude)."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) / np.sqrt(n)
    Hp = np.asfortranarray((a + a.T) * 2.0 + 0.1 * rng.standard_normal((n, n)) / np.sqrt(n) + np.diag(rng.uniform(-15.0, -5.0, n)))
    bra, ket = (rng.standard_normal(n) + 1j * rng.standard_normal(n) for _ in range(2))
    bra /= np.linalg.norm(bra)
    ket /= np.linalg.norm(ket)
    dt = 2.0e-4
    rb, rk, _, rtau, _ = oracle_mod.propagate(Hp, bra, ket, 0.0, dt, dt / H_BAR)
    gb, gk, gtau = elhl.propagation_gpucaller(Hp, bra.copy(), ket.copy(), 0.0, dt, dt / H_BAR)
    assert abs(gtau - rtau) <= 1e-12 * abs(rtau)
    assert np.abs(gb - rb).max() < 1e-11 and np.abs(gk - rk).max() < 1e-11
