"""ELHL_PREC_OZ64 where its propagation runs on the tensor cores (oz_cheb_kernel, beyond the
sizes that the FP64 row kernel takes over, 608 AOs with four columns, 912 with two): fixed and
moving nuclei against exact propagation in the generalized eigenbasis at the FP64 bars, and
many steps.  One order is one hand-over of tagged partial sums whose tags come round after
1,023 orders, and the step count covers that within a launch of many orders too."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


def _exact(oracle_mod, sysm, bra, ket, geometry, t):
    """bra and ket after t on one geometry: exp(-i H'^T t) and exp(-i H' t), H' = S^-1 h."""
    S = oracle_mod.overlap(sysm, geometry)
    ex = oracle_mod.ExactPropagator(S, oracle_mod.huckel(sysm, S))
    return S @ ex.ket(np.linalg.solve(S, bra), t), ex.ket(ket, t)


def _pops(oracle_mod, sysm, bra, ket):
    return np.stack([oracle_mod.populations(sysm, bra[:, p], ket[:, p]) for p in range(ket.shape[1])])


def _system(n_atoms):
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=11)
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    return sysm, homo


# row tiles of 128: nine with 3 rows in the last, five with 108, ten with 88
@pytest.mark.parametrize("n_atoms,ncols", [(331, 2), (200, 4), (400, 4)])
def test_fixed_nuclei_vs_exact(elhl, oracle_mod, n_atoms, ncols):
    sysm, homo = _system(n_atoms)
    S = oracle_mod.overlap(sysm)
    bra, ket = oracle_mod.initial_states(sysm, S, homo + 1, homo)
    tr = elhl.Trajectory(sysm, dt=1e-4, method=elhl.METHOD_CHEBYSHEV, precision=elhl.PREC_OZ64, ncols=ncols,
                         cheb_tol=1e-14)
    tr.init_fmo(homo + 1, homo)
    pops = tr.step(None, nsteps=20)
    b, k = tr.get_psi()
    st = tr.stats()
    tr.close()
    eb, ek = _exact(oracle_mod, sysm, bra, ket, None, 20 * 1e-4)
    assert np.abs(pops[-1] - _pops(oracle_mod, sysm, eb, ek)).max() < 1e-10
    assert np.abs(np.sum(np.conj(b) * k, axis=0) - np.sum(np.conj(eb) * ek, axis=0)).max() < 1e-10
    assert st.norm_drift < 1e-10 and st.phases == 1


def test_many_steps_and_many_orders(elhl, oracle_mod):
    """300 steps of about 40 orders, then one step of 6 fs: more than 1,023 orders in a launch."""
    sysm, homo = _system(300)
    S = oracle_mod.overlap(sysm)
    bra, ket = oracle_mod.initial_states(sysm, S, homo + 1, homo)
    for dt, nsteps, orders in ((1e-4, 300, 0), (6e-3, 1, 1024)):
        tr = elhl.Trajectory(sysm, dt=dt, method=elhl.METHOD_CHEBYSHEV, precision=elhl.PREC_OZ64, ncols=2,
                             cheb_tol=1e-14)
        tr.init_fmo(homo + 1, homo)
        pops = tr.step(None, nsteps=nsteps)
        st = tr.stats()
        tr.close()
        eb, ek = _exact(oracle_mod, sysm, bra, ket, None, nsteps * dt)
        assert np.abs(pops[-1] - _pops(oracle_mod, sysm, eb, ek)).max() < 1e-10
        assert st.orders // (2 * nsteps) > orders


@pytest.mark.parametrize("n_atoms,ncols", [(200, 4), (331, 2)])
def test_moving_then_fixed_vs_exact(elhl, oracle_mod, n_atoms, ncols):
    sysm, homo = _system(n_atoms)
    coords = np.stack([systems.perturbed_coords(sysm.coords, i, seed=3) for i in range(3)])
    S0 = oracle_mod.overlap(sysm, coords[0])
    bra, ket = oracle_mod.initial_states(sysm, S0, homo + 1, homo)
    tr = elhl.Trajectory(sysm, coords=coords[0], dt=5e-4, method=elhl.METHOD_CHEBYSHEV, precision=elhl.PREC_OZ64,
                         ncols=ncols, cheb_tol=1e-14)
    tr.set_psi(bra, ket)
    pops = list(tr.step(coords[1:], nsteps=2))
    if ncols == 4:  # with ket columns alone a fixed step takes bra = S ket
        pops += list(tr.step(None, nsteps=2))
    tr.close()
    geo = [coords[1], coords[2], coords[2], coords[2]]
    for p, g in zip(pops, geo):
        if ncols == 2:
            bra = oracle_mod.overlap(sysm, g) @ ket
        bra, ket = _exact(oracle_mod, sysm, bra, ket, g, 5e-4)
        assert np.abs(p - _pops(oracle_mod, sysm, bra, ket)).max() < 1e-10


@pytest.mark.parametrize("n_atoms,ncols,on_tensor_cores", [(294, 2, False), (295, 2, True), (196, 4, False), (197, 4, True)])
def test_line_between_the_kernels(elhl, n_atoms, ncols, on_tensor_cores):
    """The last size of the FP64 row kernel and the first of the tensor cores, by the column
    counts: both agree with the FP64 path; which kernel ran shows in the launches of a step."""
    sysm, homo = _system(n_atoms)
    assert (sysm.nao > (912 if ncols == 2 else 608)) == on_tensor_cores
    out = {}
    for prec in ("PREC_FP64", "PREC_OZ64"):
        tr = elhl.Trajectory(sysm, dt=1e-4, method=elhl.METHOD_CHEBYSHEV, precision=getattr(elhl, prec), ncols=ncols,
                             cheb_tol=1e-14)
        tr.init_fmo(homo + 1, homo)
        tr.step(None, nsteps=1)
        before = elhl.kernel_launches()
        pops = tr.step(None, nsteps=4)
        launches = elhl.kernel_launches() - before
        out[prec] = (pops, tr.get_psi()[1], launches)
        tr.close()
    assert np.abs(out["PREC_OZ64"][0] - out["PREC_FP64"][0]).max() < 1e-12
    assert np.abs(out["PREC_OZ64"][1] - out["PREC_FP64"][1]).max() < 1e-11
    # the row kernel's step is two launches, the tensor cores' one and the separate read-out's
    assert out["PREC_FP64"][2] == 8
    assert (out["PREC_OZ64"][2] == 8) != on_tensor_cores
