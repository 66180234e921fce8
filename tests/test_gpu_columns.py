"""Psi in and out of the particle-interleaved arrays, over particle counts and sizes
around the 32 x 32 tiles of the transposition."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_atoms,P", [(2, 1), (10, 2), (10, 3), (11, 32), (21, 33), (21, 64)])
def test_set_psi_get_psi_round_trip(elhl, n_atoms, P):
    """What goes in comes out, bit for bit."""
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=4, frag_atoms=2)
    tr = elhl.Trajectory(sysm, dt=1e-4, method=elhl.METHOD_CHEBYSHEV, precision=elhl.PREC_FP64, ncols=P, nparticles=P)
    rng = np.random.default_rng(P)
    bra, ket = (rng.standard_normal((sysm.nao, P)) + 1j * rng.standard_normal((sysm.nao, P)) for _ in range(2))
    tr.set_psi(bra, ket)
    b, k = tr.get_psi()
    tr.close()
    assert np.array_equal(b, bra) and np.array_equal(k, ket)
