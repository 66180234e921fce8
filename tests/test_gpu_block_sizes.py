"""The tensor-core block propagation (BF16X3) over column counts and basis sizes around its
tiles of 128 rows and 64 K, against the FP64 path."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_atoms,ncols", [(661, 16), (681, 32), (702, 64), (703, 32), (1240, 64)])
def test_block_propagation_matches_fp64(elhl, n_atoms, ncols):
    """Populations after two steps within 1e-6 of FP64, the single-precision bar of the
    other block tests (2^-24 per order and row, about 45 orders, N about 2000 to 4000)."""
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=9)
    assert sysm.nao >= 2048
    nao = int(sysm.atom_nao[sysm.fragment_atoms("E")].sum())
    out = {}
    for prec in (elhl.PREC_FP64, elhl.PREC_BF16X3):
        tr = elhl.Trajectory(sysm, dt=1e-4, method=elhl.METHOD_CHEBYSHEV, precision=prec, ncols=ncols,
                             nparticles=ncols, cheb_tol=1e-12)
        tr.init_fmo_states([1 + q % nao for q in range(ncols)])
        out[prec] = tr.step(None, nsteps=2)
        tr.close()
    err = np.abs(out[elhl.PREC_BF16X3] - out[elhl.PREC_FP64])
    assert err[:, :, :-1].max() < 1e-6
    assert err[:, :, -1].max() < 2e-6
