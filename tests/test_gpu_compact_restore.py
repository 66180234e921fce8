"""A member of a compacted batch has given up H~, so a checkpoint on another spectral
interval cannot be restored into it: it is refused, and the batch steps on."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


def test_restore_on_another_interval_is_refused(elhl, tmp_path):
    mix = [systems.cubic_cluster(n_atoms=40, seed=31), systems.cubic_cluster(n_atoms=56, seed=32)]
    path = str(tmp_path / "member.dat")
    for guard, compact in ((0.02, False), (0.01, True)):
        b = elhl.Batch(mix, dt=1e-4, precision=elhl.PREC_FP32, ncols=2, cheb_tol=1e-12, lanczos_guard=guard)
        b.init_fmo()
        b.step(1)
        if not compact:
            b.members[0].snapshot(path)
        else:
            b.compact()
            with pytest.raises(elhl.ElhlError) as e:
                b.members[0].restore(path)
            assert e.value.status == elhl.ERR_BAD_ARG
            pops = b.step(1)
            assert np.isfinite(pops).all()
        b.close()
