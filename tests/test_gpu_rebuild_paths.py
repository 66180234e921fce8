"""Paths of the moving-nuclei rebuild and of the read-out that the other tests' sizes do not
take: the reduced precisions on the factors G h G^T (large bases, short steps), the block
regime through moving steps and back to fixed ones (the operator packed again, read-out
matrices made late, the step graph recorded anew), and the one-launch read-out of one particle."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


def _run(elhl, sysm, geo, prec, P, ncols, dt, states, calls):
    tr = elhl.Trajectory(sysm, coords=geo[0], dt=dt, method=elhl.METHOD_CHEBYSHEV, precision=getattr(elhl, prec),
                         nparticles=P, ncols=ncols, cheb_tol=1e-12)
    tr.init_fmo_states(states)
    pops, phases, at = [], [], 1
    for moving, n in calls:
        pops.append(tr.step(np.stack(geo[at:at + n]) if moving else None, nsteps=n))
        at += n if moving else 0
        phases.append(tr.stats().phases)
    psi = tr.get_psi()
    tr.close()
    return np.concatenate(pops), phases, psi


@pytest.mark.parametrize("prec", ["PREC_FP32", "PREC_BF16X3"])
def test_reduced_precision_on_the_factors(elhl, prec):
    """N = 5580, 21 orders a step: FP32 applies the factors; against DF64's run of the same."""
    sysm = systems.cubic_cluster(n_atoms=1800, seed=7)
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    geo = [systems.perturbed_coords(sysm.coords, i, seed=3) for i in range(3)]
    calls = [(True, 2), (False, 2)]
    p0, _, (b0, k0) = _run(elhl, sysm, geo, "PREC_DF64", 2, 4, 2e-5, [homo + 1, homo], calls)
    p1, ph, (b1, k1) = _run(elhl, sysm, geo, prec, 2, 4, 2e-5, [homo + 1, homo], calls)
    assert ph[0] == 3
    assert np.abs(p1 - p0).max() < 5e-6  # the FP32 bar of the other operator tests
    assert np.abs(k1 - k0).max() < 5e-5


@pytest.mark.parametrize("prec,n_atoms,dt", [("PREC_BF16X3", 670, 1e-4), ("PREC_FP32", 670, 1e-4),
                                             ("PREC_BF16X3", 1800, 2e-5)])
def test_block_regime_moving_then_fixed(elhl, prec, n_atoms, dt):
    """Fixed, moving and fixed steps of 16 ket columns (one matrix product per order at fixed
    nuclei) against the FP64 (DF64 at N = 5580) row kernels; the largest basis leaves its
    moving steps on the factors and forms H~ for the fixed ones."""
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=7)
    geo = [systems.perturbed_coords(sysm.coords, i, seed=3) for i in range(4)]
    states = list(range(1, 17))
    calls = [(False, 2), (True, 2), (False, 2), (True, 1), (False, 1)]
    p0, _, (_, k0) = _run(elhl, sysm, geo, "PREC_FP64" if n_atoms < 1000 else "PREC_DF64", 16, 16, dt, states, calls)
    p1, _, (_, k1) = _run(elhl, sysm, geo, prec, 16, 16, dt, states, calls)
    # the reduced precisions hold each particle's total, which ket columns alone (bra = S ket)
    # change with the geometry; FP64 and DF64 report it as it is
    k0 = k0 / np.sqrt(p0[-1, :, -1])
    p0 = p0 / p0[:, :, -1:]
    assert np.abs(p1 - p0).max() < 2e-6 * 2  # the block tests' bars, twice their steps
    assert np.abs(k1 - k0).max() < 5e-5


@pytest.mark.parametrize("n_atoms", [16, 64, 200])
def test_one_particle_read_out(elhl, oracle_mod, n_atoms):
    """One particle with bra and ket columns: two columns on the row kernel, P = 1 in its read-out."""
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=5, frag_atoms=6)
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    S = oracle_mod.overlap(sysm)
    _, ket = oracle_mod.initial_states(sysm, S, homo + 1, homo)
    tr = elhl.Trajectory(sysm, dt=1e-4, method=elhl.METHOD_CHEBYSHEV, precision=elhl.PREC_FP64, nparticles=1, ncols=2,
                         cheb_tol=1e-14)
    tr.init_fmo_states([homo + 1])
    pops = tr.step(None, nsteps=10)
    b, k = tr.get_psi()
    tr.close()
    ex = oracle_mod.ExactPropagator(S, oracle_mod.huckel(sysm, S))
    for q in (0, 9):
        kt = ex.ket(ket[:, :1], (q + 1) * 1e-4)
        assert np.abs(pops[q] - oracle_mod.exact_populations(sysm, S, kt).T).max() < 1e-11
    # the eigensolver's column may differ from the oracle's by its sign
    sign = np.sign(np.real(np.vdot(kt[:, 0], k[:, 0])))
    assert np.abs(sign * k - kt).max() < 1e-10 and np.abs(sign * b - S @ kt).max() < 1e-10
