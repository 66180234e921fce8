"""A call of several steps enqueues them without a host round trip and looks at the
kernels' error word once at its end: a launch that gave up in any of the steps must
be reported, not only one in the last.  The failure is the test hook's (one CTA leaves
one launch at once, so the others' bounded waits run out); only the first launch after
the hook is set is affected, and the steps after it run on what it left."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


def _stalled(elhl, call):
    elhl.debug_barrier(0.2, 0)
    try:
        with pytest.raises(elhl.ElhlError) as e:
            call()
    finally:
        elhl.debug_barrier(0.0, -1)
    assert e.value.status == elhl.ERR_TIMEOUT


# the row kernel (FP64, N = 450), the tensor-core kernel (OZ64 beyond the row kernel's sizes), the
# general kernel (columns beyond the row kernel's: 4 x 1302)
@pytest.mark.parametrize("prec,n_atoms,ncols", [("PREC_FP64", 0, 2), ("PREC_OZ64", 300, 2), ("PREC_FP64", 420, 4)])
def test_first_of_three_steps(elhl, flake, prec, n_atoms, ncols):
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=11) if n_atoms else flake
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    kw = dict(dt=1e-4, method=elhl.METHOD_CHEBYSHEV, precision=getattr(elhl, prec), ncols=ncols, cheb_tol=1e-14)
    tr = elhl.Trajectory(sysm, **kw)
    tr.init_fmo(homo + 1, homo)
    tr.step(None, nsteps=1)
    _stalled(elhl, lambda: tr.step(None, nsteps=3))
    tr.close()
    tr = elhl.Trajectory(sysm, **kw)  # the next call on the same context is clean
    tr.init_fmo(homo + 1, homo)
    pops = tr.step(None, nsteps=3)
    tr.close()
    assert np.abs(pops[:, :, -1] - 1.0).max() < 1e-10


def test_first_of_three_batch_steps(elhl):
    mix = [systems.cubic_cluster(n_atoms=40, seed=31), systems.cubic_cluster(n_atoms=56, seed=32)]
    b = elhl.Batch(mix, dt=1e-4, precision=elhl.PREC_FP32, ncols=2, cheb_tol=1e-12)
    b.init_fmo()
    b.step(1)
    _stalled(elhl, lambda: b.step(3))
    b.close()
    b = elhl.Batch(mix, dt=1e-4, precision=elhl.PREC_FP32, ncols=2, cheb_tol=1e-12)
    b.init_fmo()
    pops = b.step(3)
    b.close()
    assert np.abs(np.asarray(pops)[..., -1] - 1.0).max() < 1e-5
