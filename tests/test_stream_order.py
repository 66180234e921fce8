"""The library's streams are created non-blocking, so work on the legacy default stream
(plain cudaMemset, cudaMemcpy, a launch without a stream) is ordered with theirs by
nothing: where another library keeps that stream busy, a late clear erases what kernels
have written since."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dynemol_gb300", "csrc")


def test_no_legacy_stream_copies_or_clears():
    found = []
    for name in sorted(os.listdir(CSRC)):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        found += [f"{name}: {m.group(0)}" for m in re.finditer(r"\bcuda(?:Memset|Memcpy)(?:2D|ToSymbol)?\(", text)]
    assert not found, found


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_DF64", "PREC_FP32"])
def test_created_beside_a_busy_default_stream(elhl, prec):
    """Set-up, a moving and two fixed steps while the legacy default stream works through
    half a second of another library's kernel: the same bits as with that stream idle."""
    torch = pytest.importorskip("torch")
    from dynemol_gb300 import systems
    sysm = systems.cubic_cluster(n_atoms=64, seed=7)
    homo = systems.fermi_state(sysm, sysm.fragment_atoms("E"))
    coords = np.stack([systems.perturbed_coords(sysm.coords, i, seed=3) for i in range(2)])

    def run(busy):
        if busy:
            torch.cuda._sleep(1_000_000_000)
        tr = elhl.Trajectory(sysm, coords=coords[0], dt=1e-4, method=elhl.METHOD_CHEBYSHEV,
                             precision=getattr(elhl, prec), ncols=4, cheb_tol=1e-14)
        tr.init_fmo(homo + 1, homo)
        b, k = tr.get_psi()
        tr.set_psi(b, k)
        pops = [tr.step(coords[1:], nsteps=1), tr.step(None, nsteps=2)]
        torch.cuda.synchronize()
        pops.append(tr.step(None, nsteps=1))
        psi = tr.get_psi()
        tr.close()
        return pops + list(psi)

    torch.cuda.synchronize()
    ref = run(False)
    for a, b in zip(ref, run(True)):
        assert np.array_equal(a, b)
