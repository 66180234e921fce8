"""Column counts that are not a power of two, alone and side by side in one server: groups of
four, two and one columns, against the exact propagator."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu

STEPS, DT = 3, 1.0e-4


def _exact(oracle_mod, sysm, states, steps):
    S = oracle_mod.overlap(sysm)
    ex = oracle_mod.ExactPropagator(S, oracle_mod.huckel(sysm, S))
    kets = [oracle_mod.fragment_mo(sysm, "E", s)[0].astype(complex) for s in states]
    return np.stack([oracle_mod.exact_populations(sysm, S, ex.ket(k, steps * DT)) for k in kets])


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 1e-6)])
@pytest.mark.parametrize("P", [3, 5, 6, 7])
def test_odd_column_counts(elhl, oracle_mod, P, prec, tol):
    """One trajectory of P columns: populations at the bars of the other propagation tests."""
    sysm = systems.cubic_cluster(n_atoms=41, seed=6, frag_atoms=8)
    states = list(range(2, 2 + P))
    tr = elhl.Trajectory(sysm, dt=DT, method=elhl.METHOD_CHEBYSHEV, precision=getattr(elhl, "PREC_" + prec.upper()),
                         ncols=P, nparticles=P, cheb_tol=1e-12)
    tr.init_fmo_states(states)
    pops = tr.step(None, nsteps=STEPS)[-1]
    tr.close()
    assert np.abs(pops[:, :-1] - _exact(oracle_mod, sysm, states, STEPS)[:, :-1]).max() < tol


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 1e-6)])
def test_mixed_column_counts_in_one_server(elhl, oracle_mod, prec, tol):
    """Requests of 1, 2, 3, 5 and 8 columns and uneven sizes propagated in one launch per step."""
    counts, atoms = [1, 8, 3, 5, 2], [24, 31, 37, 45, 52]
    sv = elhl.Server(4e9, dt=DT, precision=getattr(elhl, "PREC_" + prec.upper()), cheb_tol=1e-12)
    mix = [(systems.cubic_cluster(n_atoms=a, seed=q, frag_atoms=8), list(range(1, 1 + c)))
           for q, (a, c) in enumerate(zip(atoms, counts))]
    ids = [sv.submit(sysm, STEPS, states) for sysm, states in mix]
    while sum(sv.step()) > 0:
        pass
    sv.poll()
    for i, (sysm, states) in zip(ids, mix):
        pops = sv.result(i)[0]
        assert np.abs(pops[:, :-1] - _exact(oracle_mod, sysm, states, STEPS)[:, :-1]).max() < tol
    sv.close()


def test_uneven_batch_with_more_rows_per_cta_than_a_tile(elhl):
    """Forty FP32 members of N about 310 to 680: row ranges of more than 128 rows with every
    kind of remainder, within 1e-6 of the same batch in FP64."""
    systems_ = [systems.cubic_cluster(n_atoms=100 + 3 * q, seed=q, frag_atoms=16) for q in range(40)]
    out = {}
    for prec in (elhl.PREC_FP64, elhl.PREC_FP32):
        b = elhl.Batch(systems_, dt=DT, precision=prec, ncols=2, cheb_tol=1e-12)
        b.init_fmo()
        b.compact()
        out[prec] = b.step(nsteps=2)
        b.close()
    assert np.abs(out[elhl.PREC_FP32] - out[elhl.PREC_FP64])[..., :-1].max() < 1e-6
