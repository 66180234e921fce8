"""Moving nuclei form H~ or apply its factors by the size and the orders of a step: the same
basis takes the factors in short steps and H~ in long ones, a run whose step lengthens
changes over, and both agree with the tensor-core path, which always forms H~."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,phases", [(2e-5, 3), (5e-4, 1)])
def test_form_follows_the_orders(elhl, dt, phases):
    sysm = systems.cubic_cluster(n_atoms=450, seed=7)  # N = 1395: H~ pays from about 45 orders
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    geo = np.stack([systems.perturbed_coords(sysm.coords, i, seed=3) for i in range(3)])
    out = {}
    for prec in ("PREC_FP64", "PREC_OZ64"):
        tr = elhl.Trajectory(sysm, coords=geo[0], dt=dt, method=elhl.METHOD_CHEBYSHEV,
                             precision=getattr(elhl, prec), ncols=2, cheb_tol=1e-14)
        tr.init_fmo(homo + 1, homo)
        pops = tr.step(geo[1:], nsteps=2)
        out[prec] = (pops, *tr.get_psi())
        assert tr.stats().phases == (phases if prec == "PREC_FP64" else 1)
        tr.close()
    p0, b0, k0 = out["PREC_FP64"]
    p1, b1, k1 = out["PREC_OZ64"]
    assert np.abs(p0 - p1).max() < 1e-12
    assert np.abs(k0 - k1).max() < 1e-10 and np.abs(b0 - b1).max() < 1e-10
