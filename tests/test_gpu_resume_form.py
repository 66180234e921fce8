"""A checkpoint between moving and fixed steps: the restored trajectory goes on with the
operator in the form the steps before left it in and on their spectral interval, so its
fixed steps equal the uninterrupted run's bit for bit (DF64 is created on the factors
G h G^T and moves on H~; FP64 with large bases and short steps the other way round)."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n_atoms,ncols,dt", [("PREC_DF64", 64, 4, 5e-4), ("PREC_DF64", 300, 2, 5e-4),
                                                   ("PREC_FP32", 64, 4, 5e-4), ("PREC_FP64", 64, 4, 5e-4),
                                                   ("PREC_FP64", 450, 2, 2e-5), ("PREC_OZ64", 200, 2, 5e-4)])
def test_moving_then_fixed_resume_is_exact(elhl, tmp_path, prec, n_atoms, ncols, dt):
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=7)
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    coords = np.stack([systems.perturbed_coords(sysm.coords, i, seed=3) for i in range(3)])
    kw = dict(dt=dt, method=elhl.METHOD_CHEBYSHEV, precision=getattr(elhl, prec), ncols=ncols, cheb_tol=1e-14)
    path = str(tmp_path / "Security_copy.dat")
    a = elhl.Trajectory(sysm, coords=coords[0], **kw)
    a.init_fmo(homo + 1, homo)
    a.step(coords[1:], nsteps=2)
    a.snapshot(path)
    pa = a.step(None, nsteps=3)
    ba, ka = a.get_psi()
    sa = a.stats()
    a.close()
    b = elhl.Trajectory(sysm, coords=coords[2], **kw)
    b.restore(path)
    pb = b.step(None, nsteps=3)
    bb, kb = b.get_psi()
    sb = b.stats()
    b.close()
    assert (sa.phases, sa.emin, sa.emax) == (sb.phases, sb.emin, sb.emax)
    assert np.array_equal(pa, pb)
    assert np.array_equal(ka, kb) and np.array_equal(ba, bb)
