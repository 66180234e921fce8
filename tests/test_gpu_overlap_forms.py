"""S, h and the Ehrenfest force pieces over the forms their kernels distinguish:
third-row and two-exponent shells, shells of one atom with different exponents,
different on-site parameters within a shell, few atoms (pairs that do not fill a
warp) and sizes around the force kernels' tiles."""
import copy

import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


def _basis(kind, n_atoms=24):
    sysm = copy.deepcopy(systems.cubic_cluster(n_atoms=n_atoms, seed=9, frag_atoms=4))
    rng = np.random.default_rng(5)
    heavy = np.isin(sysm.ao_atom, [a for a in range(sysm.natoms) if sysm.symbols[a] != "H"])
    if kind == "third_row":  # every second heavy atom carries 3s, 3p
        sysm.ao_n[heavy & (sysm.ao_atom % 2 == 0)] = 3
    elif kind == "two_zetas":  # p shells contracted from two exponents
        p = sysm.ao_l == 1
        sysm.ao_nzeta[p] = 2
        sysm.ao_zeta[p, 1] = sysm.ao_zeta[p, 0] * 0.55
        sysm.ao_coef[p, 0], sysm.ao_coef[p, 1] = 0.7, 0.4
    elif kind == "split_zetas":  # s and p of one atom with different exponents
        sysm.ao_zeta[sysm.ao_l == 1, 0] *= 0.83
    elif kind == "site_parameters":
        sysm.ao_ip[:] = sysm.ao_ip * (1.0 + 0.01 * rng.standard_normal(sysm.nao))
        sysm.ao_vshift[:] = 0.05 * rng.standard_normal(sysm.nao)
        sysm.ao_kwh[:] = 1.75 + 0.1 * rng.random(sysm.nao)
    return sysm


@pytest.mark.parametrize("kind", ["eht", "third_row", "two_zetas", "split_zetas", "site_parameters"])
def test_overlap_and_huckel_forms(elhl, oracle_mod, kind):
    """S to 1e-13 and h to 1e-11, the bars of the plain basis (both sides FP64 with a
    few hundred operations per element; |h| <= 60 |S|)."""
    sysm = _basis(kind)
    S = oracle_mod.overlap(sysm)
    h = oracle_mod.huckel(sysm, S)
    assert np.linalg.eigvalsh(S)[0] > 1e-6
    tr = elhl.Trajectory(sysm, dt=1e-4)
    gS, gh, _ = tr.matrices()
    tr.close()
    assert np.abs(gS - S).max() < 1e-13
    assert np.abs(gh - h).max() < 1e-11


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 128, 129, 200])
def test_ehrenfest_kernel_from_states(elhl, oracle_mod, n):
    """K = X o A - H A from bra and ket against the matrix product, to 1e-10 of its largest entry
    (n products of FP64 roundings)."""
    rng = np.random.default_rng(n)
    H, X = (np.asfortranarray(rng.standard_normal((n, n))) for _ in range(2))
    bra, ket = (np.asfortranarray(rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))) for _ in range(2))
    K = elhl.ehrenfest_kernel(H, X, bra=bra, ket=ket)
    ref = oracle_mod.ehrenfest_kernel(H, X, bra=bra, ket=ket)
    assert np.abs(K - ref).max() <= 1e-10 * np.abs(ref).max()


@pytest.mark.parametrize("kind,n_atoms", [("eht", 1), ("eht", 2), ("eht", 3), ("eht", 4), ("eht", 7),
                                          ("two_zetas", 12), ("third_row", 12)])
def test_pulay_forces_forms(elhl, oracle_mod, kind, n_atoms):
    """Forces to 1e-9 of the largest at delta = 1e-5 (S round-off 1e-15 over 2 delta)."""
    sysm = _basis(kind, n_atoms) if n_atoms > 4 else systems.cubic_cluster(n_atoms=n_atoms, seed=9, frag_atoms=1)
    K = np.asfortranarray(np.random.default_rng(n_atoms).standard_normal((sysm.nao, sysm.nao)))
    F = elhl.ehrenfest_forces(sysm, K, delta=1e-5)
    ref = oracle_mod.pulay_forces(sysm, K, delta=1e-5)
    assert np.abs(F - ref).max() <= 1e-9 * max(np.abs(ref).max(), 1e-12)
