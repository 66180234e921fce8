"""The tensor-core propagation over sizes around its tiles of 128 rows and the smallest it
takes, against the FP64 path."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_atoms,ncols", [(186, 4), (188, 2), (206, 4), (207, 2), (227, 4), (289, 4), (372, 2)])
def test_moving_step_matches_fp64(elhl, n_atoms, ncols):
    """Three moving steps, populations at the FP64 bar of the other propagation tests, 1e-10."""
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=3, frag_atoms=20)
    geo = [systems.perturbed_coords(sysm.coords, i, sigma=0.02, seed=5) for i in range(4)]
    out = {}
    for prec in (elhl.PREC_FP64, elhl.PREC_OZ64):
        tr = elhl.Trajectory(sysm, coords=geo[0], dt=5e-4, method=elhl.METHOD_CHEBYSHEV, precision=prec, ncols=ncols,
                             cheb_tol=1e-12)
        tr.init_fmo(12, 11)
        out[prec] = np.stack([tr.step(g, nsteps=1) for g in geo[1:]])
        tr.close()
    assert np.abs(out[elhl.PREC_OZ64] - out[elhl.PREC_FP64]).max() < 1e-10
