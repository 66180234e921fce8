"""The Taylor propagator compares |delta|^2 with tol^2 where the reference compares |delta|
with tol (isConverged, Taylor.f:290-303): a negative tolerance, which no |delta| meets,
still ends in the no-convergence error."""
import pytest

pytestmark = pytest.mark.gpu


def test_negative_tolerance_never_converges(elhl, flake):
    tr = elhl.Trajectory(flake, dt=1e-4, tol=-1e-6, max_conv_calls=20)
    tr.init_fmo(41, 40)
    with pytest.raises(elhl.ElhlError) as e:
        tr.step(None, nsteps=1)
    tr.close()
    assert e.value.status == elhl.ERR_NO_CONVERGENCE
