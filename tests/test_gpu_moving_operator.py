"""Moving nuclei with the explicit H~ = G h G^T in FP64, DF64 and FP32: a step
through new coordinates, then fixed steps on the operator it left behind."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec_name,tol", [("fp64", 1e-11), ("df64", 1e-10), ("oz64", 1e-11), ("fp32", 5e-6)])
@pytest.mark.parametrize("n_atoms", [16, 110])  # N = 50 (FP64-pipe products), N = 340 (sliced products)
def test_moving_then_fixed_vs_exact(elhl, oracle_mod, prec_name, tol, n_atoms):
    """One moving step at the geometry the run goes on with, then three fixed steps,
    against the exact propagator of that geometry.  FP64 results to a few hundred
    roundings of the 1e-14 truncation (1e-11), DF64's 48-bit pairs to 1e-10, FP32
    to the 5e-6 of its other operator tests."""
    prec = {"fp64": elhl.PREC_FP64, "df64": elhl.PREC_DF64, "oz64": elhl.PREC_OZ64, "fp32": elhl.PREC_FP32}[prec_name]
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=5, frag_atoms=6)
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    S = oracle_mod.overlap(sysm)
    bra, ket = oracle_mod.initial_states(sysm, S, homo + 1, homo)
    tr = elhl.Trajectory(sysm, dt=2e-4, method=elhl.METHOD_CHEBYSHEV, precision=prec, ncols=4, cheb_tol=1e-14)
    tr.set_psi(bra, ket)
    pops = np.concatenate([tr.step(sysm.coords, nsteps=1), tr.step(None, nsteps=3)])
    assert tr.stats().phases == 1
    gb, gk = tr.get_psi()
    tr.close()
    ex = oracle_mod.ExactPropagator(S, oracle_mod.huckel(sysm, S))
    for q in range(4):
        ref = oracle_mod.exact_populations(sysm, S, ex.ket(ket, 2e-4 * (q + 1)))
        assert np.abs(pops[q] - ref.T).max() < tol
    k4 = ex.ket(ket, 8e-4)
    assert np.abs(gk - k4).max() < 10 * tol and np.abs(gb - S @ k4).max() < 10 * tol
