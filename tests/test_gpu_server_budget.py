"""The server's budget covers what a request's propagation holds besides its matrices and
vectors: the packed operands and the partial products of the tensor-core block product."""
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


def test_packed_operands_count(elhl):
    """Two BF16X3 requests of N = 2,077 whose matrices and vectors alone would fit the budget
    together: the second waits until the first is done; each alone is accepted."""
    sysm = systems.cubic_cluster(n_atoms=670, seed=5)
    n, P = sysm.nao, 16
    assert n >= 2048
    ld = (n + 31) // 32 * 32
    # matrices in FP64 (5) and FP32 (1), two FP64 read-out matrices, vectors, the sliced set-up products
    matrices = ld * n * (5 * 8 + 4 + 2 * 8) + ld * P * (3 * 2 * 4 + 2 * 16) + 28 * n * n + 1e6
    packed = -(-n // 128) * 128 * -(-n // 64) * 64 * 6
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    states = list(range(homo - 7, homo + 9))
    sv = elhl.Server(2 * matrices + packed, dt=1e-4, precision=elhl.PREC_BF16X3, cheb_tol=1e-8)
    ids = [sv.submit(sysm, 2, states) for _ in range(2)]
    assert sv.step() == (1, 1)
    done = []
    for _ in range(8):
        sv.step()
        done += sv.poll()
    assert done == ids
    for rid in ids:
        pops, psi, times = sv.result(rid)
        assert abs(pops[:, -1] - 1.0).max() < 1e-5
    sv.close()
    sv = elhl.Server(matrices + 1.0, dt=1e-4, precision=elhl.PREC_BF16X3, cheb_tol=1e-8)
    rid = sv.submit(sysm, 1, states)  # over the budget by the packed operands alone
    sv.step()
    assert sv.poll() == [rid]
    sv.result(rid)
    sv.close()
