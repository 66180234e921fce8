"""Reading a state back takes no device memory: elhl_traj_get_psi never fails for it, and
the server, which reads a request's Psi as it retires it, stays within what the request was
admitted with."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols_per_particle", [1, 2])
def test_get_psi_takes_no_device_memory(elhl, cols_per_particle):
    torch = pytest.importorskip("torch")
    sysm = systems.cubic_cluster(n_atoms=300, seed=11)
    P = 32  # Psi: 32 columns of N = 930, 0.5 MB a state (an allocation shows in 2 MB steps)
    states = list(range(1, P + 1))
    trs = []
    for _ in range(6):
        tr = elhl.Trajectory(sysm, dt=1e-4, method=elhl.METHOD_CHEBYSHEV, precision=elhl.PREC_FP64,
                             ncols=P * cols_per_particle, nparticles=P, cheb_tol=1e-12)
        tr.init_fmo_states(states)
        tr.step(None, nsteps=1)
        trs.append(tr)
    trs[0].get_psi()  # first launch of the transposition: the module is resident
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    psi = [tr.get_psi() for tr in trs]
    assert torch.cuda.mem_get_info()[0] == free
    for b, k in psi[1:]:
        assert np.array_equal(b, psi[0][0]) and np.array_equal(k, psi[0][1])
    dual = np.abs(np.sum(np.conj(psi[0][0]) * psi[0][1], axis=0))  # <bra|ket> of every particle
    assert np.abs(dual - 1.0).max() < 1e-10
    for tr in trs:
        tr.close()
