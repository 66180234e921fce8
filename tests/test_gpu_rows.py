"""The shared-memory row kernel (cheb_rows.cuh) over its sizes, against the exact
propagator: one to nine rows per CTA, last CTAs with fewer rows, lane groups with
padding columns, two and four columns, and the sizes on either side of its limit
(N m = 5000 in FP64 and DF64)."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu

CASES = ([("fp64", a, 4) for a in (2, 16, 49, 50, 98, 99, 390, 403, 404)] + [("fp64", a, 2) for a in (2, 49, 150, 404)]
         + [("df64", a, 4) for a in (2, 50, 99, 390)] + [("oz64", a, 4) for a in (2, 50, 225, 226)]
         + [("fp32", a, m) for a, m in ((2, 4), (50, 4), (99, 2), (390, 4), (786, 4))])


@pytest.mark.parametrize("prec_name,n_atoms,m", CASES)
def test_rows_vs_exact(elhl, oracle_mod, prec_name, n_atoms, m):
    """Two steps of 0.1 fs at one geometry (four columns: through the moving-nuclei
    path), Psi against the exact propagator.  FP64 and OZ64 truncate at 1e-14 and
    round about 60 orders of vectors of norm 1: 1e-11; DF64's pairs carry 4e-15 per
    element and order: 1e-10; FP32 as its other operator tests: 5e-6 (the sign of
    single roundings over 60 orders)."""
    prec = {"fp64": elhl.PREC_FP64, "df64": elhl.PREC_DF64, "oz64": elhl.PREC_OZ64, "fp32": elhl.PREC_FP32}[prec_name]
    tol = {"fp64": 1e-11, "oz64": 1e-11, "df64": 1e-10, "fp32": 5e-6}[prec_name]
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=3, frag_atoms=min(20, n_atoms))
    S = oracle_mod.overlap(sysm)
    rng = np.random.default_rng(n_atoms)
    ket = rng.standard_normal((sysm.nao, 2)) + 1j * rng.standard_normal((sysm.nao, 2))
    ket /= np.sqrt(np.einsum("ip,ij,jp->p", ket.conj(), S, ket).real)
    tr = elhl.Trajectory(sysm, dt=1e-4, method=elhl.METHOD_CHEBYSHEV, precision=prec, ncols=m,
                         cheb_tol=1e-14 if prec_name != "fp32" else 1e-9)
    tr.set_psi(S @ ket, ket)
    if m == 4:
        tr.step(np.stack([sysm.coords] * 2), nsteps=2)
    else:
        tr.step(None, nsteps=2)
    bra, out = tr.get_psi()
    tr.close()
    ref = oracle_mod.ExactPropagator(S, oracle_mod.huckel(sysm, S)).ket(ket, 2e-4)
    assert np.abs(out - ref).max() < tol
    assert np.abs(bra - S @ ref).max() < 10 * tol
