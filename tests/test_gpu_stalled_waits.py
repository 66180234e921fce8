"""Every bounded wait of the cooperative kernels that can run out is made to, once, by the
test hooks: a CTA that leaves or withholds what the others wait for.  The call returns
ELHL_ERR_TIMEOUT after the hook's limit (0.2 s; the Taylor kernel after its
own, 5 s), and the next call on the same context succeeds.  (The Chebyshev row kernels
and the tensor-core kernel's grid barrier: test_gpu_stalled_step.py.)"""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


def _expect_timeout(elhl, call, exit_cta=-1, stall=0):
    elhl.debug_barrier(0.2, exit_cta)
    elhl.debug_stall(stall)
    try:
        with pytest.raises(elhl.ElhlError) as e:
            call()
    finally:
        elhl.debug_barrier(0.0, -1)
        elhl.debug_stall(0)
    assert e.value.status == elhl.ERR_TIMEOUT


# H' rows in shared memory, vectors as tagged words (N = 450); read from L2, a barrier per round (N = 1302)
@pytest.mark.parametrize("n_atoms", [0, 420])
def test_taylor_round(elhl, flake, n_atoms):
    sysm = systems.cubic_cluster(n_atoms=n_atoms, seed=11) if n_atoms else flake
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))

    def run(stalled):
        tr = elhl.Trajectory(sysm, dt=1e-5)
        tr.init_fmo(homo + 1, homo)
        if stalled:
            _expect_timeout(elhl, lambda: tr.step(None, nsteps=1), exit_cta=1)
        else:
            pops = tr.step(None, nsteps=1)
            assert np.abs(pops[:, :, -1] - 1.0).max() < 1e-6
        tr.close()

    run(True)
    run(False)


def test_taylor_dropin(elhl, oracle_mod, flake):
    S = oracle_mod.overlap(flake)
    Hp = oracle_mod.h_prime(oracle_mod.sy_invert(S), oracle_mod.huckel(flake, S))
    bra, ket = oracle_mod.initial_states(flake, S, 41, 40)
    args = (np.ascontiguousarray(bra[:, 0]), np.ascontiguousarray(ket[:, 0]), 0.0, 1e-5, 1e-5 / oracle_mod.H_BAR)
    _expect_timeout(elhl, lambda: elhl.propagation_gpucaller(Hp, *args), exit_cta=2)
    b, k, _ = elhl.propagation_gpucaller(Hp, *args)
    assert abs(abs(np.vdot(b, k)) - 1.0) < 1e-6


@pytest.mark.parametrize("where", [1, 2])
@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_FP32"])
def test_rebuild(elhl, where, prec):
    """The Lanczos words (1) and the flags between the CTAs of a leaf (2) of a moving step."""
    sysm = systems.cubic_cluster(n_atoms=64, seed=7)
    coords = np.stack([systems.perturbed_coords(sysm.coords, i, seed=3) for i in range(2)])
    tr = elhl.Trajectory(sysm, coords=coords[0], dt=1e-4, method=elhl.METHOD_CHEBYSHEV,
                         precision=getattr(elhl, prec), ncols=4, cheb_tol=1e-12)
    tr.init_fmo(41, 40)
    b0, k0 = tr.get_psi()
    _expect_timeout(elhl, lambda: tr.step(coords[1:], nsteps=1), stall=where)
    tr.set_psi(b0, k0)
    pops = tr.step(coords[1:], nsteps=1)
    tr.close()
    tr = elhl.Trajectory(sysm, coords=coords[0], dt=1e-4, method=elhl.METHOD_CHEBYSHEV,
                         precision=getattr(elhl, prec), ncols=4, cheb_tol=1e-12)
    tr.set_psi(b0, k0)
    ref = tr.step(coords[1:], nsteps=1)
    tr.close()
    assert np.array_equal(pops, ref)


def test_partial_sums_of_the_tensor_core_kernel(elhl):
    sysm = systems.cubic_cluster(n_atoms=300, seed=11)
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    kw = dict(dt=1e-4, method=elhl.METHOD_CHEBYSHEV, precision=elhl.PREC_OZ64, ncols=2, cheb_tol=1e-14)
    tr = elhl.Trajectory(sysm, **kw)
    tr.init_fmo(homo + 1, homo)
    _expect_timeout(elhl, lambda: tr.step(None, nsteps=1), stall=3)
    tr.close()
    tr = elhl.Trajectory(sysm, **kw)
    tr.init_fmo(homo + 1, homo)
    pops = tr.step(None, nsteps=2)
    tr.close()
    assert np.abs(pops[:, :, -1] - 1.0).max() < 1e-10


def test_df64_grid_barrier(elhl, flake):
    """cheb_df_kernel's barrier (a DF64 trajectory is created on the factors G h G^T)."""
    kw = dict(dt=1e-4, method=elhl.METHOD_CHEBYSHEV, precision=elhl.PREC_DF64, ncols=2, cheb_tol=1e-14)
    tr = elhl.Trajectory(flake, **kw)
    tr.init_fmo(41, 40)
    tr.step(None, nsteps=1)
    _expect_timeout(elhl, lambda: tr.step(None, nsteps=2), exit_cta=5)
    tr.close()
    tr = elhl.Trajectory(flake, **kw)
    tr.init_fmo(41, 40)
    pops = tr.step(None, nsteps=2)
    tr.close()
    assert np.abs(pops[:, :, -1] - 1.0).max() < 1e-10
