"""Performance cases of the sweep engine: block SVDs, DMRG runs and sweeps, bond updates, TDVP
sweeps and tree-tensor-network sweeps, through the public Python API.

Inputs are made from the seed alone in 64-bit torch / numpy: Hamiltonians with seeded random
couplings, and states that a run meets in the middle of its sweeps (low-lying or time-evolved
states of a small lattice held as a dense vector, cut into a canonical MPS by charge sector),
so that Schmidt spectra are graded as in real use.  Outputs are gauge-independent: energies,
spectra, bond dimensions, expectation values, dense amplitudes of small chains.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

tn = load_package()
DEV = "cuda"
SPINS = (1, -1)  # charges of the two site states
F64 = torch.float64
_contexts = {}


def _ctx(precision):
    """One context per precision, as a program keeps it."""
    if precision not in _contexts:
        _contexts[precision] = tn.Context(0, precision=precision)
    return _contexts[precision]


# ------------------------------------------------------------------------------------
# cases
# ------------------------------------------------------------------------------------

def listed():
    return [
        # the block SVD of one bond by itself, host blocks in, spectrum out: the small bonds of
        # the first sweeps and chain ends (a few dozen states), a bond of the N = 100
        # Heisenberg workload (chi ~ 180, blocks of about 100 columns), and the largest bond
        # of the chi = 2048 cylinder (blocks up to 1200 x 1100)
        {"name": "svd_chi32", "kind": "svd", "chi": 32, "precision": "fp64"},
        {"name": "svd_chi180", "kind": "svd", "chi": 180, "precision": "fp64"},
        {"name": "svd_chi2048", "kind": "svd", "chi": 2048, "precision": "split"},
        # a whole two-site DMRG run from a Neel state on a chain small enough to be exact
        # (first runs, tests), in the default FP64 context
        {"name": "dmrg_N12_fp64", "kind": "dmrg", "N": 12, "maxdim": 64, "sweeps": 4,
         "precision": "fp64"},
        # the ordinary run: a Heisenberg chain from a Neel state, bond dimension ramped up
        {"name": "dmrg_N64_split", "kind": "dmrg", "N": 64, "maxdim": 128, "sweeps": 3,
         "precision": "split"},
        # one full sweep from the middle of a run in FP64: J1-J2 cylinder of 4 x 5 sites
        # (long-range MPO), two-site updates
        {"name": "sweep_j1j2_20_fp64", "kind": "sweep", "lx": 5, "chi": 160, "nsite": 2,
         "precision": "fp64"},
        # the bond update in the middle of the 6 x 4 J1-J2 cylinder, where a large run spends
        # its time: Lanczos on tensor cores, block SVD, truncation
        {"name": "bond_j1j2_24_chi384", "kind": "bond", "lx": 6, "chi": 384,
         "precision": "split"},
        {"name": "bond_j1j2_24_chi1024", "kind": "bond", "lx": 6, "chi": 1024,
         "precision": "split"},
        # real-time two-site TDVP from a Neel state: the first steps of a quench (tiny bonds),
        # complex FP64
        {"name": "tdvp_N12_fp64", "kind": "tdvp", "N": 12, "t0": 0.0, "maxdim": 64, "sweeps": 3,
         "imaginary": False, "precision": "fp64"},
        # one step in the middle of a quench, bonds grown, split precision
        {"name": "tdvp_N18_split", "kind": "tdvp", "N": 18, "t0": 4.0, "maxdim": 112, "sweeps": 1,
         "imaginary": False, "precision": "split"},
        # tree tensor networks: a small tree in FP64, and several instances of the 64-site tree
        # in lockstep on the tensor cores
        {"name": "ttn_N16_chi16_fp64", "kind": "ttn", "N": 16, "chi": 16, "instances": 1,
         "precision": "fp64"},
        {"name": "ttn_N64_chi64_x4", "kind": "ttn", "N": 64, "chi": 64, "instances": 4,
         "precision": "split"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["svd", "svd", "dmrg", "sweep", "bond", "tdvp", "ttn"])
    prec = rng.choice(["fp64", "split"])
    if kind == "svd":
        return {"kind": "svd", "chi": _log_int(rng, 32, 2000), "precision": prec}
    if kind == "dmrg":
        return {"kind": "dmrg", "N": _log_int(rng, 12, 60), "maxdim": _log_int(rng, 48, 120),
                "sweeps": rng.choice([2, 3]), "precision": prec}
    if kind == "sweep":
        return {"kind": "sweep", "lx": rng.choice([3, 4, 5]), "chi": _log_int(rng, 24, 160),
                "nsite": rng.choice([1, 2, 2]), "precision": prec}
    if kind == "bond":
        if prec == "fp64":
            return {"kind": "bond", "lx": 5, "chi": _log_int(rng, 64, 256), "precision": prec}
        lx = rng.choice([5, 6])
        return {"kind": "bond", "lx": lx, "chi": _log_int(rng, 64, 1000 if lx == 6 else 300),
                "precision": prec}
    if kind == "tdvp":
        return {"kind": "tdvp", "N": rng.choice([9, 10, 11, 12, 13, 14, 15, 16]),
                "t0": rng.choice([0.0, 1.5, 3.0]), "maxdim": _log_int(rng, 32, 100), "sweeps": 1,
                "imaginary": rng.random() < 0.3, "precision": prec}
    return {"kind": "ttn", "N": rng.choice([12, 16, 20, 27, 32]), "chi": _log_int(rng, 10, 48),
            "instances": rng.choice([1, 2, 3]), "precision": prec}


# ------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------

def _sector_dims(chi):
    """Charge-sector dimensions of a bond of dimension ~chi (charges 0, +-2, ...): Gaussian in
    the charge, the largest sector about 0.3 chi as on the benchmark chains."""
    qs = range(-12, 13, 2)
    w = [math.exp(-0.5 * (q / 2.66) ** 2) for q in qs]
    return {q: int(round(chi * x / sum(w))) for q, x in zip(qs, w)}


def _svd_shapes(chi):
    """Two-site blocks (middle charges +-1, +-3, ...) between two such bonds, of odd sizes too."""
    left, right = _sector_dims(chi), _sector_dims(0.92 * chi)
    out = []
    for m in range(-9, 10, 2):
        r = left.get(m - 1, 0) + left.get(m + 1, 0) + (m + chi) % 4
        c = right.get(m - 1, 0) + right.get(m + 1, 0) + (m * m + chi) % 3
        if min(r, c) > 0:
            out.append((r, c))
    return out


def _svd_blocks(case, seed):
    """Graded blocks (8 decades on both sides), as a two-site tensor between Schmidt bases."""
    rng = np.random.default_rng(seed)
    blocks = []
    for r, c in _svd_shapes(case["chi"]):
        dl = 10.0 ** (-8.0 * (np.arange(r) / r) ** 0.8) * rng.uniform(0.7, 1.3, r)
        dr = 10.0 ** (-8.0 * (np.arange(c) / c) ** 0.8) * rng.uniform(0.7, 1.3, c)
        blocks.append(np.asfortranarray(dl[:, None] * rng.standard_normal((r, c)) * dr[None, :]))
    return blocks


SVD_CUTOFF = 1e-12


def _bonds(case, seed):
    """(N, [(i, j, J)]): a chain or a J1-J2 cylinder of circumference 4 (J2 = J1 / 2), every
    coupling scaled by a seeded factor in [0.9, 1.1]."""
    rng = np.random.default_rng(seed)
    if "lx" in case:
        N = 4 * case["lx"]
        terms = [(i, j, J) for J, o, i, _, j in tn.models.j1j2_cylinder_terms(case["lx"], 4)
                 if o == "Sz"]
    else:
        N = case["N"]
        terms = [(i, i + 1, 1.0) for i in range(N - 1)]
    return N, [(i, j, J * f) for (i, j, J), f in zip(terms, rng.uniform(0.9, 1.1, len(terms)))]


def _mpo(N, bonds, ctx):
    terms = []
    for i, j, J in bonds:
        terms += [(J, "Sz", i, "Sz", j), (0.5 * J, "S+", i, "S-", j), (0.5 * J, "S-", i, "S+", j)]
    return tn.MPO(*tn.models.mpo_from_terms(N, terms), ctx)


def _neel_bits(N):
    return tn.models.neel_states(N)


def _apply(v, N, bonds):
    """H v on the dense vector of N spins (site 0 slowest): S_i.S_j = swap(i, j) / 2 - 1/4."""
    out = v * (-0.25 * sum(J for _, _, J in bonds))
    for i, j, J in bonds:
        x = v.view(2 ** i, 2, 2 ** (j - i - 1), 2, 2 ** (N - j - 1))
        out.view_as(x).add_(x.transpose(1, 3), alpha=0.5 * J)
    return out


def _neel_vector(N, dtype):
    v = torch.zeros(2 ** N, dtype=dtype, device=DEV)
    v[int("".join(map(str, _neel_bits(N))), 2)] = 1.0
    return v


def _low_state(N, bonds, steps):
    """Lowest Ritz pair of `steps` Lanczos iterations from the Neel state."""
    v = _neel_vector(N, F64)
    V, a, b, prev = [v], [], [], None
    for _ in range(steps):
        w = _apply(V[-1], N, bonds)
        a.append(float(w @ V[-1]))
        w.sub_(V[-1], alpha=a[-1])
        if prev is not None:
            w.sub_(prev, alpha=b[-1])
        prev = V[-1]
        b.append(float(w.norm()))
        if b[-1] < 1e-9:
            break
        V.append(w / b[-1])
    k = len(a)
    e, u = np.linalg.eigh(np.diag(a) + np.diag(b[: k - 1], 1) + np.diag(b[: k - 1], -1))
    out = torch.zeros_like(v)
    for x, c in zip(V, u[:, 0]):
        out.add_(x, alpha=float(c))
    return float(e[0]), out / out.norm()


def _evolve(v, N, bonds, tau):
    """exp(tau H) v by Taylor steps of length <= 0.1 in the norm-bounded exponent."""
    n = max(1, int(math.ceil(abs(tau) / 0.1)))
    for _ in range(n):
        term, out = v, v.clone()
        for k in range(1, 26):
            term = _apply(term, N, bonds) * (tau / n / k)
            out += term
        v = out
    return v


def _split_rows(C, q_rows, keep_max, cutoff):
    """Orthonormal basis (rows x k) of the row space of C, block by charge: eigenvectors of the
    reduced density matrix, the keep_max largest weights above cutoff.  Returns (U, charges)."""
    rho = (C @ C.mH).cpu()
    q = np.asarray(q_rows)
    found = []
    for s in np.unique(q):
        idx = np.nonzero(q == s)[0]
        w, U = torch.linalg.eigh(rho[idx][:, idx])
        found += [(float(x), int(s), idx, U[:, n]) for n, x in enumerate(w)]
    total = sum(f[0] for f in found)
    found = [f for f in sorted(found, key=lambda f: -f[0])[:keep_max] if f[0] > cutoff * total]
    found.sort(key=lambda f: (f[1], -f[0]))
    U = torch.zeros((len(q), len(found)), dtype=rho.dtype)
    for n, (_, _, idx, u) in enumerate(found):
        U[torch.from_numpy(idx), n] = u
    return U.to(C.device), np.array([f[1] for f in found], dtype=np.int32)


def _to_mps(v, N, center, chi, cutoff=1e-13):
    """Canonical MPS tensors and link charges of a dense vector, orthogonality centre at
    `center`, bonds cut at chi states."""
    pq = np.array(SPINS)
    tensors, links = [None] * N, [None] * (N + 1)
    links[0] = np.array([0], dtype=np.int32)
    links[N] = np.array([N % 2], dtype=np.int32)  # the charge of the Neel state
    C = v.reshape(1, -1)
    for i in range(center):
        C = C.reshape(2 * len(links[i]), -1)
        U, links[i + 1] = _split_rows(C, (links[i][:, None] + pq[None, :]).ravel(), chi, cutoff)
        tensors[i] = U.reshape(len(links[i]), 2, -1)
        C = U.mH @ C
    C = C.reshape(-1, 1)
    for i in range(N - 1, center, -1):
        R = C.reshape(-1, 2 * len(links[i + 1])).mT
        U, ql = _split_rows(R, (links[i + 1][None, :] - pq[:, None]).ravel(), chi, cutoff)
        links[i] = ql
        tensors[i] = U.mT.reshape(-1, 2, len(links[i + 1]))
        C = (U.mH @ R).mT
    tensors[center] = (C / C.norm()).reshape(len(links[center]), 2, len(links[center + 1]))
    return [t.cpu().numpy() for t in tensors], links


def _lattice_state(case, seed):
    """(N, bonds, tensors, links): a low-lying state (sweep, bond) or a quenched one (tdvp)."""
    N, bonds = _bonds(case, seed)
    if case["kind"] == "tdvp":
        v = _neel_vector(N, F64 if case["imaginary"] else torch.complex128)
        if case["t0"]:
            v = _evolve(v, N, bonds, -0.3 * case["t0"] if case["imaginary"] else -1j * case["t0"])
        v = v / v.norm()
        return N, bonds, *_to_mps(v, N, 0, case["maxdim"], 1e-11)
    _, v = _low_state(N, bonds, 24)
    center = N // 2 - 1 if case["kind"] == "bond" else 0
    return N, bonds, *_to_mps(v, N, center, case["chi"])


def _ttn_inputs(case, seed):
    """Isometric random trees (QR toward the centre, positive diagonals) and TFIM couplings."""
    out = []
    for k in range(case["instances"]):
        g, sn, ts, center = tn.ttn.random_ttn_tensors(case["N"], case["chi"], 1000 * seed + k)
        dist = tn.ttn._bfs(g, center)
        legs = {v: [("s", n) for n, x in enumerate(sn) if x == v] + [("n", u) for u in g[v]]
                for v in g}
        for v in sorted(g, key=lambda x: (-dist[x], x)):
            if v == center:
                continue
            par = next(u for u in g[v] if dist[u] == dist[v] - 1)
            ax = legs[v].index(("n", par))
            t = np.moveaxis(ts[v], ax, -1)
            q, r = np.linalg.qr(t.reshape(-1, t.shape[-1]))
            s = np.where(np.diag(r) < 0, -1.0, 1.0)
            ts[v] = np.moveaxis((q * s).reshape(t.shape), -1, ax)
            pax = legs[par].index(("n", v))
            ts[par] = np.moveaxis(np.tensordot(s[:, None] * r, ts[par], axes=([1], [pax])), 0, pax)
        ts[center] = ts[center] / np.linalg.norm(ts[center])
        out.append((g, sn, ts, center, *tn.ttn.tfim_instance(case["N"], 1000 * seed + 500 + k)))
    return out


def prepare(case, seed):
    kind, ctx = case["kind"], _ctx(case["precision"])
    st = {"case": case, "ctx": ctx}
    if kind == "svd":
        st["blocks"] = _svd_blocks(case, seed)
    elif kind == "dmrg":
        N, bonds = _bonds(case, seed)
        st["H"] = _mpo(N, bonds, ctx)
        st["psi"] = tn.MPS.product(_neel_bits(N), st["H"].phys_q, ctx)
        ramp = [max(16, case["maxdim"] >> (case["sweeps"] - 1 - k)) for k in range(case["sweeps"])]
        st["params"] = tn.DMRGParams(maxdim=ramp, nsweeps=[1] * case["sweeps"], cutoff=1e-10)
    elif kind in ("sweep", "bond", "tdvp"):
        N, bonds, tensors, links = _lattice_state(case, seed)
        st["H"] = _mpo(N, bonds, ctx)
        center = N // 2 - 1 if kind == "bond" else 0
        st["psi"] = tn.MPS(tensors, links, st["H"].phys_q, center, ctx)
        if kind == "bond":  # a run has its environments at the bond that it updates
            st["env"] = tn.StateEnvs(st["psi"], st["H"])
            st["env"].position_(center, 2)
            st["pos"] = center
            x = np.tensordot(tensors[center], tensors[center + 1], axes=([2], [0]))
            st["start"] = _two_site_blocks(x, links[center], links[center + 2])
    else:
        inst = _ttn_inputs(case, seed)
        st["psis"] = [tn.ttn.TTN(g, sn, 2, ts, c, ctx) for g, sn, ts, c, _, _ in inst]
        st["models"] = [tn.ttn.CouplingModel(tn.ttn.tfim_terms(J, h), case["N"])
                        for _, _, _, _, J, h in inst]
        st["path"] = tn.ttn.default_sweeppath(st["psis"][0])
    return st


# ------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------

def _amplitudes(tensors):
    """Dense amplitudes of a small MPS."""
    v = np.ones((1, 1))
    for t in tensors:
        v = np.tensordot(v, t, axes=([1], [0])).reshape(-1, t.shape[2])
    return v.ravel()


def _two_site(psi, p):
    """The updated two-site tensor, block by block (left sector, two spins): its outer bases
    are untouched by the update."""
    links = [dict(zip(*(x.tolist() for x in psi.link(i)))) for i in (p, p + 1, p + 2)]
    sites = []
    for i in (0, 1):
        flat, off, blocks = torch.from_numpy(psi.site_blocks(p + i)).to(DEV), 0, {}
        for q in sorted(links[i]):
            for s in SPINS:
                if q + s in links[i + 1]:
                    a, b = links[i][q], links[i + 1][q + s]
                    blocks[q, s] = flat[off:off + a * b].view(b, a).T
                    off += a * b
        sites.append(blocks)
    out = []
    for q in sorted(links[0]):
        for s in SPINS:
            for t in SPINS:
                if q + s + t in links[2]:
                    if q + s in links[1]:
                        out.append((sites[0][q, s] @ sites[1][q + s, t]).reshape(-1))
                    else:
                        n = links[0][q] * links[2][q + s + t]
                        out.append(torch.zeros(n, dtype=F64, device=DEV))
    return torch.cat(out)


def _two_site_blocks(x, ql, qr):
    """The same blocks of a dense tensor x[(l, s), (t, r)]."""
    x = np.asarray(x).reshape(len(ql), 2, 2, len(qr))
    out = []
    for q in np.unique(ql):
        for i, s in enumerate(SPINS):
            for j, t in enumerate(SPINS):
                cols = np.nonzero(qr == q + s + t)[0]
                if len(cols):
                    out.append(x[np.nonzero(ql == q)[0], i, j][:, cols].ravel())
    return torch.from_numpy(np.concatenate(out)).to(DEV)


def _fixed(x, chi):
    """Block data, whose length goes by the sectors, at a length that goes by chi alone."""
    return torch.nn.functional.pad(x, (0, 2 * chi * chi - len(x)))


def _padded(eigs, n):
    """Spectra of varying length as rows of n values."""
    out = np.zeros((len(eigs), n))
    for row, e in zip(out, eigs):
        row[: len(e)] = e
    return out


def _report(psi, sw, maxdim):
    out = {"energy": np.array(sw.energy[-1:]),
           "table": np.array([sw.energy[-1], sw.entropy[-1], sw.maxtruncerr[-1]]),
           "energies": np.array(sw.energy), "linkdims": np.array(psi.linkdims()),
           "spectra": _padded(sw.lasteigs, maxdim), "sz": np.array(tn.measure(psi, "Sz"))}
    if psi.N <= 14:
        out["state"] = _amplitudes([psi.site(i) for i in range(psi.N)])
    return out


BOND_CUTOFF = 1e-10
KRYLOV = {"solver_krylovdim": 5, "solver_maxiter": 2}


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "svd":
        kept, sv, err = tn.svd_truncate(st["blocks"], maxdim=case["chi"], cutoff=SVD_CUTOFF,
                                        ctx=st["ctx"])
        return {"kept": kept, "values": np.concatenate(sv + [np.array([err])])}
    if kind == "dmrg":
        env = tn.StateEnvs(st["psi"], st["H"])
        sw = tn.dmrg_(env, st["params"], 2, outputlevel=0)
        return _report(env.getpsi(), sw, case.get("chi", case.get("maxdim")))
    if kind == "sweep":
        env, sw = tn.StateEnvs(st["psi"], st["H"]), tn.SweepData()
        tn.fullsweep_(env, tn.eig_solver, case["nsite"], sw, maxdim=case["chi"],
                      cutoff=BOND_CUTOFF, outputlevel=0, **KRYLOV)
        return _report(env.getpsi(), sw, case.get("chi", case.get("maxdim")))
    if kind == "bond":  # the two updates that a full sweep gives a bond
        table, spectra, kw = [], [], dict(maxdim=case["chi"], cutoff=BOND_CUTOFF, **KRYLOV)
        for ortho in ("left", "right"):
            e, err, eigs = tn.update_position_(st["env"], tn.eig_solver, st["pos"], 2, ortho, **kw)
            table.append([e, err])
            spectra.append(eigs)
        x = _two_site(st["env"].getpsi(), st["pos"])  # an eigenvector: its sign is free
        return {"table": np.array(table), "spectra": _padded(spectra, case["chi"]),
                "two_site": _fixed(torch.sign(x @ st["start"]) * x, case["chi"])}
    if kind == "tdvp":
        eng = tn.TDVPEngine(st["psi"], st["H"])
        for _ in range(case["sweeps"]):
            tn.tdvpsweep_(eng, -0.05 if case["imaginary"] else -0.05j, maxdim=case["maxdim"],
                          cutoff=1e-9)
        return _report(eng.getpsi(), eng.swdata, case["maxdim"])
    envs = tn.ttn.StateEnvsTTN.batch(st["psis"], st["models"])
    sws = [tn.ttn.SweepDataTTN() for _ in envs]
    tn.ttn.fullsweep_batch_(envs, st["path"], tn.eig_solver, sws, maxdim=case["chi"],
                            outputlevel=0)
    out = {"energies": np.array([sw.energy[-1] for sw in sws]),
           "linkdims": np.array([sw.maxchi[-1] for sw in sws])}
    if case["instances"] == 1:
        out["x"] = np.array(tn.ttn.measure(envs[0].getpsi(), tn.ttn.PAULI_X))
    return out


# ------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------

def _svd_work(shapes):
    """Factorisation with both sets of singular vectors, as the engine's users need it:
    about 14 r c min(r, c) flops (bidiagonalisation, two factors, their products)."""
    return sum(14.0 * r * c * min(r, c) for r, c in shapes)


def _update_flops(chi_l, chi_m, chi_r, w, matvecs, one_site=False, cplx=False):
    """Flops of one update: H_eff products (both environment contractions over the charge
    blocks of every MPO state) and the block SVD."""
    L, R = _sector_dims(chi_l), _sector_dims(chi_r)
    g = lambda D, q: D.get(q, 0)  # noqa: E731
    heff, shapes = 0.0, []
    for m in range(-11, 12, 2):
        r, c = g(L, m - 1) + g(L, m + 1), g(R, m - 1) + g(R, m + 1)
        if one_site:
            c = min(c, max(1, int(0.3 * chi_m)))
        if min(r, c) < 1:
            continue
        shapes.append((r, c))
        heff += 2.0 * w * (g(L, m - 1) ** 2 + g(L, m + 1) ** 2) * c
        heff += 2.0 * w * r * (c * c if one_site else g(R, m - 1) ** 2 + g(R, m + 1) ** 2)
    return (4.0 if cplx else 1.0) * (heff * matvecs + _svd_work(shapes))


def _mps_bytes(N, chi, planes=1):
    D = [min(2 ** min(i, 30), 2 ** min(N - i, 30), chi) for i in range(N + 1)]
    return 8.0 * planes * sum(0.6 * 2 * 0.3 * a * b + 2 for a, b in zip(D, D[1:]))


def work(case):
    kind = case["kind"]
    if kind == "svd":
        shapes = _svd_shapes(case["chi"])
        n = sum(r * c + min(r, c) for r, c in shapes)
        return {"bytes": 8.0 * n, "flops": _svd_work(shapes)}
    if kind == "ttn":
        flops = values = 0.0
        g, sn, ts, _ = tn.ttn.random_ttn_tensors(case["N"], case["chi"], 0)
        for t in ts.values():  # two visits per sweep: products of 7 matvecs, QR, link moves
            D = max(t.shape)
            flops += 2 * (7 * 2.0 * t.size * sum(2 * d for d in t.shape) + 6.0 * t.size * D)
            values += t.size
        k = case["instances"]
        return {"bytes": 16.0 * values * k, "flops": flops * k}
    N = 4 * case["lx"] if "lx" in case else case["N"]
    chi = case.get("chi", case.get("maxdim"))
    w = 20 if "lx" in case else 5
    D = [min(2 ** min(i, 30), 2 ** min(N - i, 30), chi) for i in range(N + 1)]
    cplx = kind == "tdvp" and not case["imaginary"]
    if kind == "bond":
        p = N // 2 - 1
        # both environments, the two-site tensor in and out
        env = 8.0 * w * 0.2 * (D[p] ** 2 + D[p + 2] ** 2)
        return {"bytes": env + 16.0 * 4 * 0.3 * D[p] * D[p + 2],
                "flops": 2 * _update_flops(D[p], D[p + 1], D[p + 2], w, 7)}
    mv = {"dmrg": 7, "sweep": 7, "tdvp": 14}[kind]
    one = case.get("nsite", 2) == 1
    flops = 0.0
    for k in range(case.get("sweeps", 1)):
        chik = chi if kind != "dmrg" else max(16, chi >> (case["sweeps"] - 1 - k))
        E = [min(d, chik) for d in D]
        flops += sum(2 * _update_flops(E[i], E[i + 1], E[i + 2], w, mv, one, cplx)
                     for i in range(N - 1))
    return {"bytes": 2 * _mps_bytes(N, chi, 2 if cplx else 1), "flops": flops}


# ------------------------------------------------------------------------------------
# 64-bit values
# ------------------------------------------------------------------------------------

def _sz_profile(v, N):
    p = (v.abs() ** 2).reshape([2] * N)
    return np.array([float(p.select(i, 0).sum() - p.select(i, 1).sum()) / 2 for i in range(N)])


def _truncated(P, maxdim, cutoff):
    """(discarded weight, kept values) of ITensors' truncation of descending weights P."""
    n, total, err = len(P), float(P.sum()), 0.0
    while n > maxdim:
        n -= 1
        err += P[n]
    while n > 1 and err + P[n - 1] <= cutoff * total:
        n -= 1
        err += P[n]
    cut = 0.0
    if n < len(P):
        cut = 0.5 * (P[n - 1] + P[n])
        if abs(P[n - 1] - P[n]) < 1e-3 * P[n - 1]:
            cut += 1e-3 * P[n - 1]
    return err / total, P[P > cut]


def _restarted_lanczos(heff, x):
    """Lowest Ritz pair of thick-restart Lanczos with krylovdim 5, two cycles."""
    V = [x.reshape(-1) / x.norm()]
    for cycle in range(2):
        while True:
            w = heff(V[-1])
            Q = torch.stack(V)
            for _ in range(2):
                w = w - Q.T @ (Q @ w)
            if len(V) == 5:
                break
            V.append(w / w.norm())
        Hm = (Q @ torch.stack([heff(y) for y in V]).T).cpu()
        e, u = torch.linalg.eigh(0.5 * (Hm + Hm.T))
        if cycle == 0:
            V = list(u[:, :3].T.to(DEV) @ Q) + [w / w.norm()]
    y = u[:, 0].to(DEV) @ Q
    return float(e[0]), y / y.norm()


def _exact_bond(case, seed):
    """Both updates of the bond: Lanczos on the projected Hamiltonian, applied through the
    dense vector, and the truncation of the two-site tensor's weights."""
    N, bonds, ts, links = _lattice_state(case, seed)
    p = N // 2 - 1
    ts = [torch.from_numpy(np.ascontiguousarray(t)).to(DEV) for t in ts]
    A = torch.ones((1, 1), dtype=F64, device=DEV)
    for t in ts[:p]:
        A = (A @ t.flatten(1)).reshape(-1, t.shape[2])
    B = torch.ones((1, 1), dtype=F64, device=DEV)
    for t in reversed(ts[p + 2:]):
        B = (t.flatten(0, 1) @ B).reshape(t.shape[0], -1)
    a, b = A.shape[1], B.shape[0]

    def heff(x):
        full = (A @ x.reshape(a, -1)).reshape(-1, b) @ B
        y = _apply(full.reshape(-1), N, bonds).reshape(A.shape[0], -1)
        return ((A.T @ y).reshape(-1, B.shape[1]) @ B.T).reshape(-1)

    x = ts[p].flatten(0, 1) @ ts[p + 1].flatten(1)
    start, table, spectra = x, [], []
    for _ in range(2):  # the left and the right update
        e, x = _restarted_lanczos(heff, x)
        U, S, Vh = torch.linalg.svd(x.reshape(2 * a, 2 * b).cpu(), full_matrices=False)
        P = (S * S).numpy()
        err, kept = _truncated(P, case["chi"], BOND_CUTOFF)
        k = len(kept)
        x = ((U[:, :k] * (S[:k] / S[:k].norm())) @ Vh[:k]).to(DEV)
        table.append([e, err])
        spectra.append(kept)
    x = x * math.copysign(1.0, float((x * start).sum()))
    return {"table": np.array(table), "spectra": _padded(spectra, case["chi"]),
            "two_site": _fixed(_two_site_blocks(x.cpu().numpy(), links[p], links[p + 2]),
                               case["chi"])}


def exact(case, seed):
    kind = case["kind"]
    if kind == "svd":
        blocks = _svd_blocks(case, seed)
        sv = [torch.linalg.svdvals(torch.from_numpy(b)).numpy() for b in blocks]
        err, _ = _truncated(np.sort(np.concatenate(sv) ** 2)[::-1], case["chi"], SVD_CUTOFF)
        return {"kept": None, "values": np.concatenate(sv + [np.array([err])])}
    if kind == "bond":
        return _exact_bond(case, seed) if case["chi"] <= 512 else None
    if kind == "tdvp":  # the exact evolution of the state that the sweeps start from
        N, bonds, ts, _ = _lattice_state(case, seed)
        tau = (-0.05 if case["imaginary"] else -0.05j) * case["sweeps"]
        v = _evolve(torch.from_numpy(_amplitudes(ts)).to(DEV), N, bonds, tau)
        out = dict.fromkeys(("energy", "table", "energies", "linkdims", "spectra", "state"))
        out["sz"] = _sz_profile(v / v.norm(), N)
        return out
    if kind == "dmrg" and case["N"] <= 16:  # the ground energy that the run converges to
        N, bonds = _bonds(case, seed)
        out = dict.fromkeys(("table", "energies", "linkdims", "spectra", "sz", "state"))
        out["energy"] = np.array([_low_state(N, bonds, 70)[0]])
        return out
    return None
