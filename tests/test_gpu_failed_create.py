"""A trajectory whose creation fails (two atoms at one place) gives back all it took."""
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_OZ64", "PREC_DF64", "PREC_FP32", "taylor"])
def test_no_device_memory_is_kept(elhl, prec):
    torch = pytest.importorskip("torch")
    sysm = systems.cubic_cluster(n_atoms=300, seed=7)
    bad = sysm.coords.copy()
    bad[1] = bad[0]
    kw = dict(dt=1e-4) if prec == "taylor" else dict(dt=1e-4, method=elhl.METHOD_CHEBYSHEV,
                                                     precision=getattr(elhl, prec), ncols=4)
    free = []
    for _ in range(4):
        with pytest.raises(elhl.ElhlError) as e:
            elhl.Trajectory(sysm, coords=bad, **kw)
        assert e.value.status == elhl.ERR_NOT_PD
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[3] == free[1]  # the first call loads modules and makes shared workspaces
