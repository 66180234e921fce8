"""Moving and fixed steps by turns: the plan of the propagation is kept, with new read-out
matrices, and every step agrees with exact propagation on its geometry."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


# the row kernel, the general kernel (4 x 1302 columns), the tensor cores, FP32, and FP64 short
# steps on the factors
@pytest.mark.parametrize("prec,n_atoms,dt,tol", [("PREC_FP64", 64, 2e-4, 1e-11), ("PREC_FP64", 420, 2e-4, 1e-11),
                                                 ("PREC_OZ64", 200, 2e-4, 1e-11), ("PREC_FP32", 64, 2e-4, 5e-6),
                                                 ("PREC_FP32", 420, 2e-4, 5e-6), ("PREC_FP64", 420, 2e-5, 1e-11),
                                                 ("PREC_DF64", 64, 2e-4, 1e-10)])
def test_alternating_steps_vs_exact(elhl, oracle_mod, prec, n_atoms, dt, tol):
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=5)
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    geo = [systems.perturbed_coords(sysm.coords, i, seed=3) for i in range(4)]
    bra, ket = oracle_mod.initial_states(sysm, oracle_mod.overlap(sysm, geo[0]), homo + 1, homo)
    tr = elhl.Trajectory(sysm, coords=geo[0], dt=dt, method=elhl.METHOD_CHEBYSHEV, precision=getattr(elhl, prec),
                         ncols=4, cheb_tol=1e-14)
    tr.set_psi(bra, ket)
    for g in geo[1:]:
        got = [tr.step(g, nsteps=1), tr.step(None, nsteps=1), tr.step(None, nsteps=2)[1:]]
        S = oracle_mod.overlap(sysm, g)
        ex = oracle_mod.ExactPropagator(S, oracle_mod.huckel(sysm, S))
        for pops, steps in zip(got, (1, 1, 2)):
            bra, ket = S @ ex.ket(np.linalg.solve(S, bra), steps * dt), ex.ket(ket, steps * dt)
            ref = np.stack([oracle_mod.populations(sysm, bra[:, p], ket[:, p]) for p in range(2)])
            assert np.abs(pops[0] - ref).max() < tol
    tr.close()
