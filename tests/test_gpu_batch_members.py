"""A batch follows what its members do by themselves between its steps: an odd number of
steps of their own, moving steps (on the factors too), and checkpoints of another run.  Each
member agrees with a trajectory of its own that does the same."""
import numpy as np
import pytest

from dynemol_gb300 import systems

pytestmark = pytest.mark.gpu


def _mix():
    return [systems.cubic_cluster(n_atoms=40, seed=31), systems.cubic_cluster(n_atoms=56, seed=32),
            systems.cubic_cluster(n_atoms=450, seed=7)]


@pytest.mark.parametrize("prec,tol", [("PREC_FP64", 1e-11), ("PREC_FP32", 2e-6)])
def test_members_that_stepped_alone(elhl, prec, tol):
    mix = _mix()
    kw = dict(dt=2e-5, precision=getattr(elhl, prec), ncols=2, cheb_tol=1e-12)  # N = 1395 moves on the factors (FP64)
    geo = [systems.perturbed_coords(s.coords, 1, seed=3) for s in mix]
    homo = [systems.fermi_state(s, s.fragment_atoms("E")) for s in mix]
    b = elhl.Batch(mix, **kw)
    b.init_fmo()
    got = [b.step(1)]
    b.members[0].step(None, nsteps=1)
    b.members[2].step(geo[2], nsteps=1)
    got.append(b.step(2)[-1:])
    b.members[1].step(geo[1], nsteps=1)
    b.members[1].step(None, nsteps=2)
    got.append(b.step(1))
    psi = [m.get_psi()[1] for m in b.members]
    b.close()
    for i, s in enumerate(mix):
        tr = elhl.Trajectory(s, method=elhl.METHOD_CHEBYSHEV, **kw)
        tr.init_fmo(homo[i] + 1, homo[i])
        ref = [tr.step(None, nsteps=1)[-1]]
        if i == 0:
            tr.step(None, nsteps=1)
        if i == 2:
            tr.step(geo[2], nsteps=1)
        ref.append(tr.step(None, nsteps=2)[-1])
        if i == 1:
            tr.step(geo[1], nsteps=1)
            tr.step(None, nsteps=2)
        ref.append(tr.step(None, nsteps=1)[-1])
        k = tr.get_psi()[1]
        tr.close()
        for q in range(3):
            assert np.abs(got[q][-1, i] - ref[q]).max() < tol
        assert np.abs(psi[i] - k).max() < 10 * tol


def test_member_restored_from_a_run_on_the_factors(elhl, tmp_path):
    """The member keeps an explicit operator; its columns are the checkpoint's."""
    mix = _mix()[1:]
    kw = dict(dt=2e-5, precision=elhl.PREC_FP64, ncols=2, cheb_tol=1e-12)
    s = mix[1]
    homo = systems.fermi_state(s, s.fragment_atoms("E"))
    path = str(tmp_path / "run.dat")
    tr = elhl.Trajectory(s, method=elhl.METHOD_CHEBYSHEV, **kw)
    tr.init_fmo(homo + 1, homo)
    tr.step(s.coords, nsteps=1)
    assert tr.stats().phases == 3
    tr.snapshot(path)
    ref = tr.step(None, nsteps=3)
    tr.close()
    b = elhl.Batch(mix, **kw)
    b.init_fmo()
    b.step(1)
    b.members[1].restore(path)
    got = b.step(3)
    b.close()
    assert np.abs(got[:, 1] - ref).max() < 1e-11


def test_server_request_restored_from_a_run_on_the_factors(elhl, tmp_path):
    mix = _mix()
    s = mix[2]
    homo = systems.fermi_state(s, s.fragment_atoms("E"))
    path = str(tmp_path / "run.dat")
    tr = elhl.Trajectory(s, dt=2e-5, method=elhl.METHOD_CHEBYSHEV, precision=elhl.PREC_FP64, ncols=2, cheb_tol=1e-12)
    tr.init_fmo(homo + 1, homo)
    tr.step(s.coords, nsteps=1)
    tr.snapshot(path)
    ref = tr.step(None, nsteps=2)[-1]
    tr.close()
    sv = elhl.Server(4e9, dt=2e-5, precision=elhl.PREC_FP64, cheb_tol=1e-12)
    h0 = systems.fermi_state(mix[0], mix[0].fragment_atoms("E"))
    other = sv.submit(mix[0], 2, [h0 + 1, h0])
    rid = sv.submit(s, 2, [homo + 1, homo], restart=path)
    done = []
    for _ in range(4):
        sv.step()
        done += sv.poll()
    assert sorted(done) == sorted([other, rid])
    pops, _, _ = sv.result(rid)
    sv.result(other)
    sv.close()
    assert np.abs(pops - ref).max() < 1e-11
