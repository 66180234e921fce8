"""A moving step whose geometry cannot be factored (two atoms at one place) is refused, and the
trajectory stays where it was: its next steps, fixed or moving, equal those of a run without
the attempt, bit for bit."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


# H~ on the row kernel, on the tensor cores, FP32, DF64, the factors in short steps, the block regime
@pytest.mark.parametrize("prec,n_atoms,ncols,dt", [("PREC_FP64", 64, 4, 5e-4), ("PREC_OZ64", 200, 4, 5e-4),
                                                   ("PREC_FP32", 64, 4, 5e-4), ("PREC_DF64", 64, 4, 5e-4),
                                                   ("PREC_FP64", 450, 2, 2e-5), ("PREC_BF16X3", 670, 16, 1e-4)])
@pytest.mark.parametrize("moved_before,then_moving", [(True, False), (True, True), (False, False)])
def test_refused_geometry_leaves_the_state(elhl, prec, n_atoms, ncols, dt, moved_before, then_moving):
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=7)
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    geo = [systems.perturbed_coords(sysm.coords, i, seed=3) for i in range(4)]
    bad = geo[2].copy()
    bad[1] = bad[0]
    P = 2 if ncols <= 4 else ncols
    out = []
    for attempt in (False, True):
        tr = elhl.Trajectory(sysm, coords=geo[0], dt=dt, method=elhl.METHOD_CHEBYSHEV, precision=getattr(elhl, prec),
                             ncols=ncols, nparticles=P, cheb_tol=1e-12)
        tr.init_fmo_states([homo + 1, homo] if P == 2 else list(range(1, P + 1)))
        if moved_before:
            tr.step(geo[1], nsteps=1)
        else:
            tr.step(None, nsteps=1)
        if attempt:
            with pytest.raises(elhl.ElhlError) as e:
                tr.step(bad, nsteps=1)
            assert e.value.status == elhl.ERR_NOT_PD
        pops = tr.step(np.stack(geo[2:4]) if then_moving else None, nsteps=2)
        st = tr.stats()
        out.append((pops, *tr.get_psi(), np.array([st.t, st.it, st.emin, st.emax])))
        tr.close()
    assert np.isfinite(out[0][0]).all()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_refused_after_a_good_step_of_the_call(elhl):
    """The step before the refused one counts; the next call goes on from it."""
    sysm = systems.cubic_cluster(n_atoms=64, seed=7)
    geo = [systems.perturbed_coords(sysm.coords, i, seed=3) for i in range(3)]
    bad = geo[2].copy()
    bad[5] = bad[9]
    out = []
    for attempt in (False, True):
        tr = elhl.Trajectory(sysm, coords=geo[0], dt=5e-4, method=elhl.METHOD_CHEBYSHEV, precision=elhl.PREC_FP64,
                             ncols=4, cheb_tol=1e-12)
        tr.init_fmo(41, 40)
        if attempt:
            with pytest.raises(elhl.ElhlError):
                tr.step(np.stack([geo[1], bad]), nsteps=2)
        else:
            tr.step(geo[1], nsteps=1)
        pops = tr.step(None, nsteps=2)
        out.append((pops, *tr.get_psi(), np.array([tr.stats().t, tr.stats().it])))
        tr.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
