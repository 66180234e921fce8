"""Performance cases of the electron-hole propagator: the work its users have it do, through the Python
mirror of the C ABI (``dynemol_gb300.api``).

Kinds (``case["kind"]``):

* ``moving``  one nuclear step of a trajectory whose geometry changes: new coordinates in, populations and
              the propagated Psi (bra and ket) out; S, h, the Cholesky factor and the operator rebuilt.  The
              Ehrenfest run of the benchmark (1,200 atoms) and its smaller siblings, in every precision;
* ``fixed``   a block of steps at fixed nuclei (the C100H50 flake of the benchmark, dt 0.1 fs);
* ``batch``   many fixed-nuclei trajectories of uneven size advanced together;
* ``block``   an ensemble of 16 to 64 wavepackets on one basis (the precision study's GEMM regime);
* ``dropin``  the reference's entry point: one particle, one step, S, h, H' and Psi in host memory;
* ``forces``  the Ehrenfest force call of one step: the force kernel, then the overlap-derivative forces;
* ``serve``   a few requests through the continuous-batching server, submission to results.

Results of a trajectory propagated in FP32 or BF16X3 are kept in single precision, all others in double.

``exact`` restates the physics independently in 64 bits: Slater overlaps by quadrature in prolate
spheroidal coordinates, Wolfsberg-Helmholz h, fragment orbitals and propagation by eigendecomposition.
"""
import math

import numpy as np
import torch

from dynemol_gb300 import api, systems

HBAR = 6.58264e-4  # eV ps
PRECISIONS = {"fp64": api.PREC_FP64, "fp32": api.PREC_FP32, "bf16x3": api.PREC_BF16X3, "df64": api.PREC_DF64,
              "oz64": api.PREC_OZ64}
SINGLE = ("fp32", "bf16x3")
GEOMETRIES = 6  # coordinate sets a moving trajectory's host program walks through


def listed():
    return [
        # a 20-atom molecule with moving nuclei: latency and launches
        {"name": "moving_oz64_20", "kind": "moving", "atoms": 20, "precision": "oz64"},
        # the benchmark's small workload, an odd atom count
        {"name": "moving_oz64_301", "kind": "moving", "atoms": 301, "precision": "oz64"},
        # the headline run: 1,200 atoms, N = 3720, default precision
        {"name": "moving_oz64_1200", "kind": "moving", "atoms": 1200, "precision": "oz64"},
        # the plain FP64 path (the reference's arithmetic) on a mid-size cluster
        {"name": "moving_fp64_333", "kind": "moving", "atoms": 333, "precision": "fp64"},
        # FP64-level results from FP32 pairs
        {"name": "moving_df64_600", "kind": "moving", "atoms": 600, "precision": "df64"},
        # single precision with a geometry that changes
        {"name": "moving_fp32_240", "kind": "moving", "atoms": 240, "precision": "fp32"},
        # the benchmark's flake, fixed nuclei, a block of steps per call
        {"name": "fixed_fp64_flake", "kind": "fixed", "atoms": 150, "precision": "fp64", "steps": 20},
        # a trajectory mix, 24 members of N about 200 to 3000
        {"name": "batch_fp32_24", "kind": "batch", "members": 24, "max_atoms": 960, "precision": "fp32", "steps": 4},
        # an ensemble on the tensor cores
        {"name": "block_bf16x3_64", "kind": "block", "atoms": 1320, "columns": 64, "precision": "bf16x3", "steps": 4},
        # the drop-in call of the Fortran host
        {"name": "dropin_150", "kind": "dropin", "atoms": 150},
        # forces of one Ehrenfest step
        {"name": "forces_200", "kind": "forces", "atoms": 200},
        # a handful of served requests, set-up included
        {"name": "serve_fp32_6", "kind": "serve", "requests": 6, "max_atoms": 320, "precision": "fp32", "steps": 12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges, none of the listed cases themselves."""
    shapes = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _drawn(rng)
        if case not in shapes:
            return case


def _drawn(rng):
    kind = rng.choice(["moving", "moving", "moving", "fixed", "batch", "block", "dropin", "forces", "serve"])
    if kind == "moving":
        p = rng.choice(["oz64", "oz64", "fp64", "df64", "fp32"])
        return {"kind": kind, "atoms": _log_int(rng, 16, {"oz64": 1200, "fp64": 400}.get(p, 700)), "precision": p}
    if kind == "fixed":
        return {"kind": kind, "atoms": _log_int(rng, 24, 400), "precision": rng.choice(["fp64", "fp32"]),
                "steps": rng.randint(1, 24)}
    if kind == "batch":
        return {"kind": kind, "members": rng.randint(4, 24), "max_atoms": _log_int(rng, 120, 960),
                "precision": rng.choice(["fp32", "fp32", "fp64"]), "steps": rng.randint(1, 4)}
    if kind == "block":
        return {"kind": kind, "atoms": rng.randint(670, 1320), "columns": rng.choice([16, 24, 32, 64]),
                "precision": rng.choice(["fp32", "bf16x3", "bf16x3"]), "steps": rng.randint(1, 4)}
    if kind == "dropin":
        return {"kind": kind, "atoms": _log_int(rng, 20, 260)}
    if kind == "forces":
        return {"kind": kind, "atoms": _log_int(rng, 20, 400)}
    return {"kind": kind, "requests": rng.randint(2, 6), "max_atoms": _log_int(rng, 60, 320),
            "precision": rng.choice(["fp32", "fp64"]), "steps": rng.randint(3, 12)}


# ---------------------------------------------------------------- inputs
def _cluster(atoms, seed):
    return systems.cubic_cluster(n_atoms=atoms, seed=1 + seed, frag_atoms=min(20, max(4, atoms // 4)))


def _system(case, seed):
    if case["kind"] == "fixed" and case["atoms"] == 150:
        return systems.honeycomb_flake(seed=1 + seed)
    return _cluster(case["atoms"], seed)


def _mix(case, seed, count):
    """`count` clusters spread over the case's sizes (from about an eighth of the largest up)."""
    top = case["max_atoms"]
    lo = max(24, top // 14)
    return [_cluster(int(round(lo + (top - lo) * (q + 0.5) / count)), 1000 * (seed + 1) + q) for q in range(count)]


def _steps_dt(case):
    return 5.0e-4 if case["kind"] in ("moving", "dropin", "forces") else 1.0e-4


def _geometries(sysm, seed):
    return [systems.perturbed_coords(sysm.coords, i, sigma=0.02, seed=7 + seed) for i in range(GEOMETRIES)]


def _homo(sysm):
    return systems.fermi_state(sysm, sysm.fragment_atoms("E"))


def _frag_states(sysm, count):
    nao = int(sysm.atom_nao[sysm.fragment_atoms("E")].sum())
    return [1 + (q % nao) for q in range(count)]


def _columns(case, q):
    """Columns and steps of request q of a served mix."""
    return 1 + (3 * q) % 8, 1 + (case["steps"] * (q + 1)) // case["requests"]


def prepare(case, seed):
    kind = case["kind"]
    dt = _steps_dt(case)
    if kind in ("moving", "fixed"):
        sysm = _system(case, seed)
        geo = _geometries(sysm, seed) if kind == "moving" else None
        tr = api.Trajectory(sysm, coords=None if geo is None else geo[0], dt=dt, method=api.METHOD_CHEBYSHEV,
                            precision=PRECISIONS[case["precision"]], ncols=4 if geo else 2, cheb_tol=1e-12)
        tr.init_fmo(_homo(sysm) + 1, _homo(sysm))
        return {"kind": kind, "tr": tr, "geo": geo, "at": 0, "steps": case.get("steps", 1),
                "single": case["precision"] in SINGLE}
    if kind == "block":
        sysm = _system(case, seed)
        m = case["columns"]
        tr = api.Trajectory(sysm, dt=dt, method=api.METHOD_CHEBYSHEV, precision=PRECISIONS[case["precision"]],
                            ncols=m, nparticles=m, cheb_tol=1e-9)
        tr.init_fmo_states(_frag_states(sysm, m))
        return {"kind": kind, "tr": tr, "steps": case["steps"], "single": True}
    if kind == "batch":
        b = api.Batch(_mix(case, seed, case["members"]), dt=dt, precision=PRECISIONS[case["precision"]], ncols=2,
                      cheb_tol=1e-12 if case["precision"] == "fp64" else 1e-9)
        b.init_fmo()
        b.compact()
        return {"kind": kind, "batch": b, "steps": case["steps"], "single": case["precision"] in SINGLE}
    if kind == "serve":
        sv = api.Server(32e9, dt=dt, precision=PRECISIONS[case["precision"]],
                        cheb_tol=1e-12 if case["precision"] == "fp64" else 1e-9)
        reqs = []
        for q, sysm in enumerate(_mix(case, seed, case["requests"])):
            cols, steps = _columns(case, q)
            reqs.append((sysm, steps, _frag_states(sysm, cols)))
        return {"kind": kind, "server": sv, "requests": reqs, "single": case["precision"] in SINGLE}
    sysm = _system(case, seed)
    S, h = _matrices(sysm, sysm.coords)
    ket = np.stack([_fmo(sysm, S, h, s) for s in (_homo(sysm) + 1, _homo(sysm))], 1)
    Sn, hn = S.cpu().numpy(), h.cpu().numpy()
    if kind == "dropin":
        k = ket[:, 0].astype(np.complex128)
        return {"kind": kind, "S": np.asfortranarray(Sn), "h": np.asfortranarray(hn), "bra": (Sn @ k), "ket": k,
                "dt": dt}
    Hp = torch.cholesky_solve(h, torch.linalg.cholesky(S)).cpu().numpy()
    kets = (ket * np.exp(1j * np.arange(len(ket)))[:, None]).astype(np.complex128)
    return {"kind": kind, "sys": sysm, "H": np.asfortranarray(Hp), "X": np.asfortranarray(_x_matrix(sysm)),
            "bra": np.asfortranarray((Sn @ kets).conj()), "ket": np.asfortranarray(kets)}


# ---------------------------------------------------------------- one pass
def _held(single, pops, *psis):
    if single:
        return [pops.astype(np.float32)] + [p.astype(np.complex64) for p in psis]
    return [pops, *psis]


def run(state):
    kind = state["kind"]
    if kind == "moving":
        state["at"] = state["at"] % (GEOMETRIES - 1) + 1
        pops = state["tr"].step(state["geo"][state["at"]], nsteps=1)
        bra, ket = state["tr"].get_psi()
        return _held(state["single"], pops, bra, ket)
    if kind in ("fixed", "block"):
        pops = state["tr"].step(None, nsteps=state["steps"])
        bra, ket = state["tr"].get_psi()
        return _held(state["single"], pops, bra, ket)
    if kind == "batch":
        pops = state["batch"].step(nsteps=state["steps"])
        psi = [tr.get_psi()[1].ravel(order="F") for tr in state["batch"].members]
        return _held(state["single"], pops, np.concatenate(psi))
    if kind == "serve":
        sv = state["server"]
        ids = [sv.submit(sysm, steps, states) for sysm, steps, states in state["requests"]]
        while sum(sv.step()) > 0:
            pass
        sv.poll()
        got = [sv.result(i) for i in ids]
        return _held(state["single"], np.concatenate([p.ravel() for p, _, _ in got]),
                     np.concatenate([k.ravel(order="F") for _, k, _ in got]))
    if kind == "dropin":
        bra, ket = state["bra"].copy(), state["ket"].copy()
        Hp, ao_bra, bra, ket, tau = api.propagationelhl_gpucaller(state["S"], state["h"], bra, ket, 0.0, state["dt"],
                                                                  state["dt"] / HBAR)
        return [Hp, ao_bra, bra, ket, tau]
    K = api.ehrenfest_kernel(state["H"], state["X"], bra=state["bra"], ket=state["ket"])
    return [K, api.ehrenfest_forces(state["sys"], K, delta=1e-5)]


# ---------------------------------------------------------------- what a pass cannot do without
def _orders(dt):
    """Chebyshev orders of one step on these systems (spectral half width about 130 eV)."""
    return 143.0 if dt > 3e-4 else 45.0


def _nao(atoms):
    return round(0.6 * atoms) * 4 + round(0.3 * atoms) + (atoms - round(0.6 * atoms) - round(0.3 * atoms)) * 4


def work(case):
    kind, dt = case["kind"], _steps_dt(case)
    if kind in ("batch", "serve"):
        count = case["members"] if kind == "batch" else case["requests"]
        top = case["max_atoms"]
        lo = max(24, top // 14)
        ns = [_nao(int(round(lo + (top - lo) * (q + 0.5) / count))) for q in range(count)]
        cols = [2 if kind == "batch" else _columns(case, q)[0] for q in range(count)]
        steps = [case["steps"] if kind == "batch" else _columns(case, q)[1] for q in range(count)]
        size = 4 if case["precision"] in SINGLE else 8
        flops = sum(s * (_orders(dt) + 1) * 4.0 * n * n * m for n, m, s in zip(ns, cols, steps))
        if kind == "serve":  # overlap to operator: Cholesky, inverse and two triangular products
            flops += sum(3.0 * n ** 3 for n in ns)
            return {"bytes": sum(24.0 * n + 16.0 * n * m for n, m in zip(ns, cols)), "flops": flops}
        return {"bytes": sum(size * float(n) * n + 32.0 * n * m for n, m in zip(ns, cols)), "flops": flops}
    n = 450 if kind == "fixed" and case["atoms"] == 150 else _nao(case["atoms"])
    if kind == "moving":  # Cholesky and inverse, then the series on four columns with the factors applied
        return {"bytes": 24.0 * case["atoms"] + 128.0 * n, "flops": 2 / 3 * n ** 3 + _orders(dt) * 4.0 * n * n * 4}
    if kind in ("fixed", "block"):
        m = case.get("columns", 2)
        size = 4 if case["precision"] in SINGLE else 8
        return {"bytes": size * float(n) * n + 48.0 * n * m, "flops": case["steps"] * (_orders(dt) + 1) * 4.0 * n * n * m}
    if kind == "dropin":  # S and h in, H' out; S^-1 h and the Taylor series of bra and ket
        return {"bytes": 24.0 * n * n + 80.0 * n, "flops": 2.0 * n ** 3 + 300 * 8.0 * n * n}
    return {"bytes": 24.0 * n * n + 64.0 * n, "flops": 2.0 * n ** 3 + 6 * 400.0 * n * n}


# ---------------------------------------------------------------- the same in 64 bits, independently
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


_LAG = np.polynomial.laguerre.laggauss(10)
_LEG = np.polynomial.legendre.leggauss(56)
_AXIS = {-1: 1, 0: 2, 1: 0}  # m -> Cartesian axis of a p orbital


def _radials(shells_a, shells_b, R):
    """{(p, q): (sigma, pi)} of the shells (n, l, zeta) of two atoms at the distances R."""
    dev = R.device
    t, wt = (torch.as_tensor(x, device=dev) for x in _LAG)
    nu, wn = (torch.as_tensor(x, device=dev) for x in _LEG)
    out = {}
    for p, (na, la, za) in enumerate(shells_a):
        for q, (nb, lb, zb) in enumerate(shells_b):
            sg, pi = torch.empty_like(R), torch.zeros_like(R)
            for c0 in range(0, len(R), 40000):
                r = R[c0:c0 + 40000, None, None]
                pp, qq = r * (za + zb) / 2, r * (za - zb) / 2
                mu, v = 1 + t[None, :, None] / pp, nu[None, None, :]
                w = wt[None, :, None] * wn[None, None, :] * torch.exp(-pp - qq * v) / pp
                half = r / 2
                ra, rb = half * (mu + v), half * (mu - v)
                f = w * half * ra ** (na - la) * rb ** (nb - lb)  # r_a r_b of the volume element included
                if la:
                    f = f * half * (1 + mu * v) * math.sqrt(3)
                if lb:
                    f = f * half * (mu * v - 1) * math.sqrt(3)
                norm = ((2 * za) ** (na + 0.5) * (2 * zb) ** (nb + 0.5)
                        / math.sqrt(math.factorial(2 * na) * math.factorial(2 * nb)))
                sg[c0:c0 + 40000] = norm * f.sum((1, 2)) / 2
                if la and lb:
                    g = w * half ** 3 * 3 * ra ** (na - 1) * rb ** (nb - 1) * (mu * mu - 1) * (1 - v * v)
                    pi[c0:c0 + 40000] = norm * g.sum((1, 2)) / 4
            out[p, q] = (sg, pi)
    return out


def _kinds(sysm):
    kinds = {}
    for a in range(sysm.natoms):
        s = slice(int(sysm.atom_ao0[a]), int(sysm.atom_ao0[a] + sysm.atom_nao[a]))
        kinds.setdefault(tuple((int(n), int(l), int(m), float(z[0]), float(c[0])) for n, l, m, z, c in zip(
            sysm.ao_n[s], sysm.ao_l[s], sysm.ao_m[s], sysm.ao_zeta[s], sysm.ao_coef[s])), []).append(a)
    return list(kinds.items())


def _blocks(aos_a, aos_b, d):
    """Overlap blocks (pairs, nao_a, nao_b) of atoms displaced by d (A to B)."""
    sha, shb = (sorted({(n, l, z) for n, l, _, z, _ in aos}) for aos in (aos_a, aos_b))
    R = d.norm(dim=1)
    u = d / R[:, None]
    rad = _radials(sha, shb, R)
    out = torch.zeros((len(R), len(aos_a), len(aos_b)), dtype=torch.float64, device=d.device)
    for i, (na, la, ma, za, ca) in enumerate(aos_a):
        for j, (nb, lb, mb, zb, cb) in enumerate(aos_b):
            sg, pi = rad[sha.index((na, la, za)), shb.index((nb, lb, zb))]
            x = u[:, _AXIS[ma]] if la else 1.0
            y = u[:, _AXIS[mb]] if lb else 1.0
            v = sg * x * y
            if la and lb:
                v = v + pi * ((1.0 if ma == mb else 0.0) - x * y)
            out[:, i, j] = ca * cb * v
    out[R > 12.0] = 0.0
    return out


def _overlap(sysm, coords):
    dev = _dev()
    xyz = torch.as_tensor(np.ascontiguousarray(coords), device=dev)
    S = torch.eye(sysm.nao, dtype=torch.float64, device=dev)
    ao0 = torch.as_tensor(sysm.atom_ao0.astype(np.int64), device=dev)
    kinds = _kinds(sysm)
    for x, (aos_a, at_a) in enumerate(kinds):
        for aos_b, at_b in kinds[x:]:
            a = torch.as_tensor(at_a, device=dev).repeat_interleave(len(at_b))
            b = torch.as_tensor(at_b, device=dev).repeat(len(at_a))
            a, b = a[a != b], b[a != b]
            if not len(a):
                continue
            blk = _blocks(aos_a, aos_b, xyz[b] - xyz[a])
            r = (ao0[a][:, None, None] + torch.arange(len(aos_a), device=dev)[None, :, None]).expand_as(blk)
            c = (ao0[b][:, None, None] + torch.arange(len(aos_b), device=dev)[None, None, :]).expand_as(blk)
            S[r, c] = blk
            S[c, r] = blk
    return S


def _x_matrix(sysm):
    ip, k = sysm.ao_ip, sysm.ao_kwh
    c1, c2 = ip[:, None] - ip[None, :], ip[:, None] + ip[None, :]
    c3 = (c1 / c2) ** 2
    kk = (k[:, None] + k[None, :]) / 2
    return (kk + c3 + c3 ** 2 * (1 - kk)) * c2 / 2 + (sysm.ao_vshift[:, None] + sysm.ao_vshift[None, :]) / 2


def _matrices(sysm, coords):
    S = _overlap(sysm, coords)
    h = torch.as_tensor(_x_matrix(sysm), device=S.device) * S
    h.fill_diagonal_(0.0)
    return S, h + torch.diag(torch.as_tensor(sysm.ao_ip + sysm.ao_vshift, device=S.device))


def _fmo(sysm, S, h, state):
    """Fragment orbital `state` (1-based, ascending energy), largest component positive, in the full basis."""
    aos = np.concatenate([np.arange(sysm.atom_ao0[a], sysm.atom_ao0[a] + sysm.atom_nao[a])
                          for a in sysm.fragment_atoms("E")])
    sf, hf = S.cpu().numpy()[np.ix_(aos, aos)], h.cpu().numpy()[np.ix_(aos, aos)]
    li = np.linalg.inv(np.linalg.cholesky(sf))
    c = li.T @ np.linalg.eigh(li @ hf @ li.T)[1][:, state - 1]
    full = np.zeros(sysm.nao)
    full[aos] = c * np.sign(c[np.argmax(np.abs(c))])
    return full


class _Exact:
    """exp(-i S^-1 h t / hbar) by the generalised eigenvectors."""

    def __init__(self, sysm, coords, S=None, h=None):
        self.sys = sysm
        self.S, self.h = _matrices(sysm, coords) if S is None else (S, h)
        L = torch.linalg.cholesky(self.S)
        w = torch.linalg.solve_triangular(L, self.h, upper=False)
        w = torch.linalg.solve_triangular(L, w.T.contiguous(), upper=False)
        self.E, U = torch.linalg.eigh((w + w.T) / 2)
        self.C = torch.linalg.solve_triangular(L.T, U, upper=True)  # C^T S C = 1
        self.SC = self.S @ self.C

    def ket(self, psi, t):
        """Psi(t) of AO columns psi (complex tensor)."""
        return self._apply(self.C, self.SC, psi, t)

    def bra(self, psi, t):
        """The dual state S Psi: S exp(-i S^-1 h t / hbar) S^-1."""
        return self._apply(self.SC, self.C, psi, t)

    def _apply(self, out, into, psi, t):
        ph = torch.exp(-1j * self.E * (t / HBAR))[:, None]
        c = ph * torch.complex(into.T @ psi.real.contiguous(), into.T @ psi.imag.contiguous())
        return torch.complex(out @ c.real.contiguous(), out @ c.imag.contiguous())

    def pops(self, bra, ket):
        v = (bra.conj() * ket).real.T.cpu().numpy()  # (P, N)
        frag = self.sys.ao_frag
        return np.stack([v[:, frag == f].sum(1) for f in range(self.sys.nfrag)] + [v.sum(1)], 1)


def _c(x, like):
    return torch.as_tensor(np.asarray(x, np.complex128), device=like.device)


def _run_fixed(sysm, states, steps, dt):
    """Populations after each step and the final bra and ket of fragment orbitals `states`."""
    e = _Exact(sysm, sysm.coords)
    ket0 = _c(np.stack([_fmo(sysm, e.S, e.h, s) for s in states], 1), e.S)
    pops = []
    for k in range(1, steps + 1):
        ket = e.ket(ket0, k * dt)
        bra = torch.complex(e.S @ ket.real.contiguous(), e.S @ ket.imag.contiguous())
        pops.append(e.pops(bra, ket))
    return np.stack(pops), bra.cpu().numpy(), ket.cpu().numpy()


def exact(case, seed):
    kind, dt = case["kind"], _steps_dt(case)
    if kind == "moving":
        sysm = _system(case, seed)
        geo = _geometries(sysm, seed)
        S0, h0 = _matrices(sysm, geo[0])
        ket = np.stack([_fmo(sysm, S0, h0, s) for s in (_homo(sysm) + 1, _homo(sysm))], 1)
        bra = S0.cpu().numpy() @ ket
        e = _Exact(sysm, geo[1])
        ket, bra = e.ket(_c(ket, e.S), dt), e.bra(_c(bra, e.S), dt)
        return [e.pops(bra, ket)[None], bra.cpu().numpy(), ket.cpu().numpy()]
    if kind == "fixed":
        sysm = _system(case, seed)
        return list(_run_fixed(sysm, (_homo(sysm) + 1, _homo(sysm)), case["steps"], dt))
    if kind == "block":
        sysm = _system(case, seed)
        return list(_run_fixed(sysm, _frag_states(sysm, case["columns"]), case["steps"], dt))
    if kind == "batch":
        pops, kets = [], []
        for sysm in _mix(case, seed, case["members"]):
            p, _, k = _run_fixed(sysm, (_homo(sysm) + 1, _homo(sysm)), case["steps"], dt)
            pops.append(p)
            kets.append(k.ravel(order="F"))
        return [np.stack(pops, 1), np.concatenate(kets)]
    if kind == "serve":
        pops, kets = [], []
        for q, sysm in enumerate(_mix(case, seed, case["requests"])):
            cols, steps = _columns(case, q)
            p, _, k = _run_fixed(sysm, _frag_states(sysm, cols), steps, dt)
            pops.append(p[-1].ravel())
            kets.append(k.ravel(order="F"))
        return [np.concatenate(pops), np.concatenate(kets)]
    st = prepare(case, seed)  # host inputs only, made by the functions above
    if kind == "dropin":
        S, h = (torch.as_tensor(np.ascontiguousarray(st[k]), device=_dev()) for k in ("S", "h"))
        e = _Exact(None, None, S, h)
        bra, ket = (x(_c(st[k][:, None], S), dt) for x, k in ((e.bra, "bra"), (e.ket, "ket")))
        inv = e.C @ e.C.T
        ao = torch.complex(inv @ bra.real.contiguous(), inv @ bra.imag.contiguous())
        # the accepted sub-step is a control decision, not a computed number of the physics: no value
        return [torch.linalg.solve(S, h).cpu().numpy()] + [x[:, 0].cpu().numpy() for x in (ao, bra, ket)] + [None]
    sysm = st["sys"]
    b, k = st["bra"], st["ket"]
    rho = sum(s * (b[:, None, c] * k[None, :, c]).real for c, s in ((0, 1.0), (1, -1.0)))
    A = (rho + rho.T) / 2
    K = st["X"] * A - st["H"] @ A
    return [K, _pulay(sysm, K, 1e-5)]


def _pulay(sysm, K, delta):
    """Forces 2 sum_L (-dS/dR . K), central differences of the quadrature overlaps."""
    dev = _dev()
    xyz = torch.as_tensor(np.ascontiguousarray(sysm.coords), device=dev)
    Kt = torch.as_tensor(K, device=dev)
    ao0 = torch.as_tensor(sysm.atom_ao0.astype(np.int64), device=dev)
    F = torch.zeros((sysm.natoms, sysm.natoms, 3), dtype=torch.float64, device=dev)
    kinds = _kinds(sysm)
    for aos_l, at_l in kinds:
        for aos_k, at_k in kinds:
            lo = torch.as_tensor(at_l, device=dev).repeat_interleave(len(at_k))
            kk = torch.as_tensor(at_k, device=dev).repeat(len(at_l))
            lo, kk = lo[kk < lo], kk[kk < lo]
            if not len(lo):
                continue
            d = xyz[kk] - xyz[lo]
            near = d.norm(dim=1) < 12.0
            i = (ao0[kk][:, None, None] + torch.arange(len(aos_k), device=dev)[None, None, :])
            j = (ao0[lo][:, None, None] + torch.arange(len(aos_l), device=dev)[None, :, None])
            kern = Kt[i.expand(-1, len(aos_l), -1), j.expand(-1, -1, len(aos_k))]
            for c in range(3):
                e = torch.zeros(3, dtype=torch.float64, device=dev)
                e[c] = delta
                g = (_blocks(aos_l, aos_k, d + e) - _blocks(aos_l, aos_k, d - e)) / (2 * delta)
                F[kk, lo, c] = -(g * kern).sum((1, 2)) * near
    return (2.0 * 1.602176565e-9 * (F.sum(1) - F.sum(0))).cpu().numpy()
