"""Timed workloads of the engine, through its public Python entry points.

Each case is one call (or the short sequence of calls) that a program makes
over and over: Fock builds of one molecule from device or host buffers, closed
and open shell, in FP64 and in the precision form; builds of a batch of
molecules; the stored integral table; the MO integrals MP2 starts from; and a
whole SCF.  Sizes run from one water molecule, where latency and launches
count, to the (H2O)32 / 6-31G* cluster of the benchmark.

`listed()` gives the cases, `draw(rng)` more of the same ranges, `prepare`
what a program holds before the call (geometry, basis, context, density),
`run` one pass, `work` the bytes and operations a pass cannot do without, and
`exact` the same outputs from a plain torch evaluation of the integrals
(McMurchie-Davidson, FP64, no screening), where that is affordable.

Keys of a case:
  kind      rhf | rhf_host | uhf | precision | batch | packed | ovov | scf
  mol       water | alkane | oh | ch3, with `size` molecules or carbon atoms
            (kind batch: `size` molecules drawn from all four)
  basis     a bundled basis
  exact     the exact integral convention (what serving uses) instead of the
            reference's, which differs for (dd|dd) on several centres
  streams   concurrent class streams, graphs: CUDA graph replay
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from hartreefock_b200 import basis_io, engine, molecules, scf

THRESHOLD = 1e-12
_OPTIONS = {"exact": False, "streams": False, "graphs": False}


def _case(name, kind, mol, size, basis, **options):
    return {"name": name, "kind": kind, "mol": mol, "size": size, "basis": basis, **_OPTIONS, **options}


def listed():
    return [
        # the smallest call: one water in a minimal basis, as in the reference's example; launches and latency only
        _case("rhf_water1_sto3g", "rhf", "water", 1, "sto-3g"),
        # an open-shell radical with diffuse functions, one small UHF build of a served stream
        _case("uhf_ch3_631ppgss", "uhf", "ch3", 1, "6-31+g**", streams=True),
        # a mid-size closed shell called from a host program (numpy in, numpy out), replayed as a graph
        _case("rhf_host_water8_631gs", "rhf_host", "water", 8, "6-31g*", exact=True, streams=True, graphs=True),
        # an ordinary closed-shell build with every default
        _case("rhf_water16_631gs", "rhf", "water", 16, "6-31g*"),
        # the benchmark's build
        _case("rhf_water32_631gs", "rhf", "water", 32, "6-31g*", streams=True),
        # a chain molecule with diffuse functions: long contractions, few negligible pairs
        _case("rhf_alkane9_631ppgss", "rhf", "alkane", 9, "6-31+g**", exact=True, streams=True),
        # an open-shell build of ordinary size
        _case("uhf_alkane10_631gs", "uhf", "alkane", 10, "6-31g*", exact=True, streams=True),
        # the precision form as an SCF runs it: a first build from the whole density, then an incremental one
        _case("precision_water10_631gs", "precision", "water", 10, "6-31g*", exact=True),
        # one build of a batch of small molecules, part of them converged (device mask)
        _case("batch96", "batch", "mixed", 96, "sto-3g|6-31g", streams=True),
        # the stored integral table, the reference's own way of working
        _case("packed_water4_631gs", "packed", "water", 4, "6-31g*", exact=True),
        # (ia|jb) integrals for MP2
        _case("ovov_water4_631gs", "ovov", "water", 4, "6-31g*", exact=True),
        # a whole SCF from geometry to density, a fixed number of steps
        _case("scf_water4_631gs", "scf", "water", 4, "6-31g*"),
    ]


def draw(rng):
    """A case of the listed ranges: sizes log-uniform, every kind, basis and option."""
    def size(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))

    kind = rng.choice(["rhf", "rhf", "rhf", "rhf_host", "uhf", "precision", "batch", "packed", "ovov", "scf"])
    opt = {"exact": rng.random() < 0.5, "streams": rng.random() < 0.5, "graphs": False}
    if kind == "batch":
        return {"kind": kind, "mol": "mixed", "size": size(2, 128), "basis": "sto-3g|6-31g", **opt}
    basis = rng.choice(["sto-3g", "6-31g", "6-31g*", "6-31+g**"])
    top = {"rhf": 24, "rhf_host": 16, "uhf": 16, "precision": 16, "packed": 6, "ovov": 5, "scf": 6}[kind]
    if basis == "6-31+g**":  # more functions per atom
        top = max(2, top // 2)
    if kind == "uhf":
        mol = rng.choice(["water", "alkane", "oh", "ch3"])
    else:
        mol = rng.choice(["water", "water", "alkane"])
    if mol == "alkane":
        top = min(top, 12)
    n = 1 if mol in ("oh", "ch3") else size(1, top)
    if kind in ("rhf_host",):
        opt["graphs"] = rng.random() < 0.5
    if kind in ("precision", "packed", "ovov", "scf"):
        opt["streams"] = False
    return {"kind": kind, "mol": mol, "size": n, "basis": basis, **opt}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _geometry(mol, size, seed):
    """(Z, xyz in bohr): the seed places the waters; a chain or radical is
    turned and its bonds vary by a percent."""
    if mol == "water":
        return molecules.water_cluster(size, seed=seed)
    Z, xyz = {"alkane": lambda: molecules.alkane(size), "oh": molecules.hydroxyl, "ch3": molecules.methyl_planar}[mol]()
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    return list(Z), np.asarray(xyz) * (1.0 + 0.01 * rng.uniform(-1, 1)) @ q


def _batch_molecules(case, seed):
    """The batch's composition follows from its size (every seed has the same
    functions), its geometries from the seed."""
    rng = np.random.default_rng(1000 + case["size"])
    geo = np.random.default_rng(2000 + seed)
    bases = case["basis"].split("|")
    out = []
    for k in range(case["size"]):
        mol = ["water", "alkane", "oh", "ch3"][int(rng.choice(4, p=[0.45, 0.35, 0.1, 0.1]))]
        size = int(rng.integers(1, 7 if mol == "water" else 9)) if mol in ("water", "alkane") else 1
        Z, xyz = _geometry(mol, size, int(geo.integers(1 << 30)))
        out.append((Z, xyz, bases[int(rng.integers(len(bases)))]))
    return out


def _density(table, seed, electrons=2.0):
    """A symmetric matrix with the decay of an insulator's density: random
    elements that fall off with the distance of the two centres, on a diagonal
    between zero and the occupation."""
    rng = np.random.default_rng(7 + seed)
    n = table.nbf
    centre = np.zeros((n, 3))
    for s in range(len(table.L)):
        k = (int(table.L[s]) + 1) * (int(table.L[s]) + 2) // 2
        centre[table.ao_offset[s]:table.ao_offset[s] + k] = table.center[s]
    r = np.linalg.norm(centre[:, None] - centre[None], axis=-1)
    A = rng.normal(size=(n, n)) * 0.3
    P = 0.5 * electrons * (0.5 * (A + A.T) * np.exp(-r / 2.0) + np.diag(rng.uniform(0.1, 0.9, size=n)))
    return np.ascontiguousarray(P)


def _orbitals(n, seed):
    q, _ = np.linalg.qr(np.random.default_rng(11 + seed).normal(size=(n, n)))
    return np.ascontiguousarray(q)


def _convention(case):
    return engine.ERI_EXACT if case["exact"] else engine.ERI_REFERENCE


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        mols = _batch_molecules(case, seed)
        eng = engine.BatchEngine(mols, schwarz_threshold=THRESHOLD, eri_convention=_convention(case))
        eng.set_streams(case["streams"])
        P = np.concatenate([_density(t, seed + m).ravel() for m, t in enumerate(eng.tables)])
        active = (np.random.default_rng(seed).random(len(mols)) < 0.75).astype(np.uint8)
        active[0] = 1
        return {"case": case, "eng": eng, "P": torch.from_numpy(P).cuda(), "G": torch.zeros(eng.total, dtype=torch.float64, device="cuda"),
                "active": torch.from_numpy(active).cuda()}
    Z, xyz = _geometry(case["mol"], case["size"], seed)
    if kind == "scf":
        return {"case": case, "Z": Z, "xyz": xyz}
    opts = {}
    if kind == "precision":
        opts = dict(mixed_cutoff=1e-4, density_screening=True, incremental=True)
    eng = engine.Engine(Z, xyz, case["basis"], schwarz_threshold=THRESHOLD, eri_convention=_convention(case), **opts)
    if case["streams"]:
        eng.set_streams(True)
    if case["graphs"]:
        eng.set_graphs(True)
    state = {"case": case, "eng": eng}
    n = eng.nbf
    if kind == "rhf_host":
        state["P"] = torch.from_numpy(_density(eng.table, seed)).pin_memory().numpy()
        state["G"] = torch.zeros(n, n, dtype=torch.float64).pin_memory().numpy()
        return state

    def dev(a):
        return torch.from_numpy(a).cuda()

    def out():
        return torch.zeros(n, n, dtype=torch.float64, device="cuda")

    if kind == "uhf":
        Pb = _density(eng.table, seed + 1, electrons=1.0) * 0.1
        Pa = _density(eng.table, seed, electrons=1.0)
        state.update(Pa=dev(Pa), Pb=dev(Pa + Pb), Ga=out(), Gb=out())
    elif kind == "precision":
        P = _density(eng.table, seed)
        state.update(P=dev(P), P2=dev(P + 1e-3 * _density(eng.table, seed + 1)), G=out(), G2=out())
    elif kind == "packed":
        state["out"] = torch.zeros(eng.packed_size(), dtype=torch.float64, device="cuda")
    elif kind == "ovov":
        nocc = max(1, sum(Z) // 2)
        state.update(C=dev(_orbitals(n, seed)), nocc=nocc)
    else:
        state.update(P=dev(_density(eng.table, seed)), G=out())
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "scf":
        r = scf.run_scf(state["Z"], state["xyz"], case["basis"], alpha=0.5, init_guess=0.75, max_iterations=8,
                        eri_convention=_convention(case))
        return {"energy": r["energy"], "density": r["density"]}
    eng = state["eng"]
    if kind == "rhf":
        eng.fock_rhf_tensor(state["P"], state["G"])
        return state["G"]
    if kind == "rhf_host":
        return eng.fock_rhf(state["P"], out=state["G"])
    if kind == "uhf":
        eng.fock_uhf_tensor(state["Pa"], state["Pb"], state["Ga"], state["Gb"])
        return [state["Ga"], state["Gb"]]
    if kind == "precision":
        eng.fock_reset()
        eng.fock_rhf_tensor(state["P"], state["G"])
        eng.fock_rhf_tensor(state["P2"], state["G2"])
        return [state["G"], state["G2"]]
    if kind == "batch":
        return eng.fock_rhf_async(state["P"], state["G"], state["active"])
    if kind == "packed":
        eng.eri_packed_device(state["out"].data_ptr(), state["out"].numel(), torch.cuda.current_stream().cuda_stream or 1)
        return state["out"]
    return eng.mo_eri_ovov_tensor(state["C"], 0, state["nocc"], state["nocc"], eng.nbf - state["nocc"])


# ---------------------------------------------------------------------------
# necessary work
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _build_flops(mol, size, basis):
    """Operations of one screened Fock build, estimated: shell pairs by the
    overlap of their most diffuse primitives, quartets whose pair estimates
    multiply to the screening threshold, 40 per primitive quartet (distance,
    Boys function, one recursion step) and 14 per function quartet (six J/K
    contributions)."""
    t = basis_io.shell_table(*_geometry(mol, size, 0), basis)
    amin = np.array([t.exponent[o:o + k].min() for o, k in zip(t.prim_offset, t.nprim)])
    nf = (t.L + 1) * (t.L + 2) // 2
    r2 = ((t.center[:, None] - t.center[None]) ** 2).sum(-1)
    logq = -(amin[:, None] * amin[None] / (amin[:, None] + amin[None])) * r2
    i, j = np.tril_indices(len(t.L))
    lq, f, p = logq[i, j], (nf[i] * nf[j]).astype(float), (t.nprim[i] * t.nprim[j]).astype(float)
    o = np.argsort(-lq)
    lq, f, p = lq[o], f[o], p[o]
    cf, cp = np.concatenate([[0], np.cumsum(f)]), np.concatenate([[0], np.cumsum(p)])
    kept = np.searchsorted(-lq, lq - math.log(THRESHOLD), side="right")
    functions, primitives = 0.5 * float((f * cf[kept]).sum()), 0.5 * float((p * cp[kept]).sum())
    return 40.0 * primitives + 14.0 * functions, t.nbf


def work(case):
    kind = case["kind"]
    if kind == "batch":
        flops, elems = 0.0, 0
        for Z, xyz, basis in _batch_molecules(case, 0):
            n = basis_io.shell_table(Z, xyz, basis).nbf
            elems += n * n
            flops += 0.75 * (n ** 4 / 8) * 60
        return {"bytes": 16 * elems, "flops": flops}
    flops, n = _build_flops(case["mol"], case["size"], case["basis"])
    if kind == "uhf":
        return {"bytes": 32 * n * n, "flops": flops * 1.1}
    if kind == "precision":
        return {"bytes": 32 * n * n, "flops": 2 * flops}
    if kind == "packed":
        m = n * (n + 1) // 2
        return {"bytes": 4 * m * (m + 1), "flops": flops}
    if kind == "ovov":
        nocc = max(1, sum(_geometry(case["mol"], case["size"], 0)[0]) // 2)
        ov = nocc * (n - nocc)
        return {"bytes": 8 * (n * n + ov * ov), "flops": flops + 2.0 * n ** 3 * n * nocc}
    if kind == "scf":
        return {"bytes": 8 * n * n, "flops": 8 * (flops + 30.0 * n ** 3)}
    return {"bytes": 16 * n * n, "flops": flops}


# ---------------------------------------------------------------------------
# plain evaluation of the integrals (McMurchie-Davidson in torch, FP64)
# ---------------------------------------------------------------------------
_TERMS, _STEP, _SWITCH = 9, 1.0 / 16.0, 32.0


@functools.lru_cache(maxsize=1)
def _boys_table():
    """F_m(T_i) on the grid T_i = i / 16, m < 9 + 9, from the convergent series."""
    T = np.arange(int(_SWITCH / _STEP) + 2, dtype=np.longdouble) * np.longdouble(_STEP)
    tab = np.zeros((len(T), 9 + _TERMS), dtype=np.longdouble)
    for m in range(tab.shape[1]):
        term = np.ones_like(T) / (2 * m + 1)
        for k in range(400):
            tab[:, m] += term
            term = term * 2 * T / (2 * m + 2 * k + 3)
        tab[:, m] *= np.exp(-T)
    return tab.astype(np.float64)


def _boys(M, T, device):
    """[F_0 .. F_M](T): Taylor expansion of F_M and downward recursion below
    the switch, erf and upward recursion above."""
    tab = torch.from_numpy(_boys_table()).to(device)
    near = T < _SWITCH
    Tn = torch.where(near, T, torch.zeros_like(T))
    i = torch.round(Tn / _STEP).long()
    dt = i * _STEP - Tn
    f, power = torch.zeros_like(T), torch.ones_like(T)
    for k in range(_TERMS):
        f = f + tab[:, M + k][i] * power
        power = power * dt / (k + 1)
    e = torch.exp(-T)
    low = [None] * (M + 1)
    low[M] = f
    for m in range(M - 1, -1, -1):
        low[m] = (2 * Tn * low[m + 1] + e) / (2 * m + 1)
    Tf = torch.where(near, torch.ones_like(T), T)
    g = torch.sqrt(math.pi / Tf) / 2 * torch.erf(torch.sqrt(Tf))
    out = []
    for m in range(M + 1):
        out.append(torch.where(near, low[m], g))
        g = ((2 * m + 1) * g - e) / (2 * Tf)
    return out


def _components(L):
    return [(l, m, L - l - m) for l in range(L, -1, -1) for m in range(L - l, -1, -1)]


def _hermites(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _pair_class(t, la, lb, device):
    """Shell pairs (a, b) of the class, both orders where la == lb, with their
    primitive pairs: exponent, centre, pair index and Hermite coefficients
    [primitive pairs, components a x b, Hermite functions]."""
    A, B = np.nonzero(t.L == la)[0], np.nonzero(t.L == lb)[0]
    pairs = [(a, b) for a in A for b in B]
    ea, eb, ka, kb, RA, RB, idx = [], [], [], [], [], [], []
    norm = lambda e, L: (2 * e / math.pi) ** 0.75 * (4 * e) ** (L / 2.0)
    prim = {s: (t.exponent[t.prim_offset[s]:t.prim_offset[s] + t.nprim[s]], t.coefficient[t.prim_offset[s]:t.prim_offset[s] + t.nprim[s]])
            for s in set(A) | set(B)}
    for k, (a, b) in enumerate(pairs):
        (xa, ca), (xb, cb) = prim[a], prim[b]
        na, nb = len(xa), len(xb)
        ea.append(np.repeat(xa, nb)); eb.append(np.tile(xb, na))
        ka.append(np.repeat(ca * norm(xa, la), nb)); kb.append(np.tile(cb * norm(xb, lb), na))
        RA.append(np.repeat(t.center[a][None], na * nb, 0)); RB.append(np.repeat(t.center[b][None], na * nb, 0))
        idx.append(np.full(na * nb, k))
    if not pairs:
        return None
    ten = lambda x: torch.from_numpy(np.ascontiguousarray(np.concatenate(x))).to(device)
    ea, eb, k, RA, RB, idx = ten(ea), ten(eb), ten(ka) * ten(kb), ten(RA), ten(RB), ten(idx)
    p = ea + eb
    P = (ea[:, None] * RA + eb[:, None] * RB) / p[:, None]
    one = []
    for d in range(3):
        PA, PB, AB = P[:, d] - RA[:, d], P[:, d] - RB[:, d], RA[:, d] - RB[:, d]
        E = {(0, 0, 0): torch.exp(-ea * eb / p * AB * AB)}
        get = lambda i, j, q: E.get((i, j, q), torch.zeros_like(p))
        for i in range(la + 1):
            for j in range(lb + 1):
                if i == j == 0:
                    continue
                for q in range(i + j + 1):
                    i1, j1, X = (i - 1, j, PA) if i > 0 else (i, j - 1, PB)
                    E[(i, j, q)] = get(i1, j1, q - 1) / (2 * p) + X * get(i1, j1, q) + (q + 1) * get(i1, j1, q + 1)
        one.append(E)
    odd = lambda l: math.prod(range(1, 2 * l, 2))
    herm = _hermites(la + lb)
    comp = [(x, y) for x in _components(la) for y in _components(lb)]
    G = torch.zeros(len(p), len(comp), len(herm), dtype=torch.float64, device=device)
    for c, (x, y) in enumerate(comp):
        f = k / math.sqrt(math.prod(odd(l) for l in x + y))
        for h, q in enumerate(herm):
            if all(q[d] <= x[d] + y[d] for d in range(3)):
                G[:, c, h] = f * one[0][(x[0], y[0], q[0])] * one[1][(x[1], y[1], q[1])] * one[2][(x[2], y[2], q[2])]
    ao = np.array([[(t.ao_offset[a] + ia, t.ao_offset[b] + ib) for ia in range((la + 1) * (la + 2) // 2)
                    for ib in range((lb + 1) * (lb + 2) // 2)] for a, b in pairs])
    ao = torch.from_numpy(ao).to(device)
    return {"p": p, "P": P, "G": G, "pair": idx, "npairs": len(pairs), "herm": herm, "L": la + lb, "row": ao[..., 0] * t.nbf + ao[..., 1]}


def _hermite_integrals(L, alpha, X):
    """R_tuv(alpha, X) for t + u + v <= L."""
    R2 = (X * X).sum(-1)
    F = _boys(L, alpha * R2, alpha.device)
    cur = {}
    for n in range(L, -1, -1):
        new = {(0, 0, 0): (-2 * alpha) ** n * F[n]}
        for t, u, v in sorted(_hermites(L - n), key=sum):
            if t + u + v == 0:
                continue
            d = 0 if t else (1 if u else 2)
            low = [t, u, v]
            low[d] -= 1
            r = X[..., d] * cur[tuple(low)]
            if low[d]:
                low2 = list(low)
                low2[d] -= 1
                r = r + low[d] * cur[tuple(low2)]
            new[(t, u, v)] = r
        cur = new
    return cur


def _integrals(t, device):
    """Every (ij|kl) as an [n*n, n*n] matrix."""
    n = t.nbf
    out = torch.zeros(n * n, n * n, dtype=torch.float64, device=device)
    Ls = sorted(set(int(l) for l in t.L))
    classes = [c for c in (_pair_class(t, a, b, device) for a in Ls for b in Ls if a >= b) if c]
    for x, bra in enumerate(classes):
        for ket in classes[:x + 1]:
            hb, hk = len(bra["herm"]), len(ket["herm"])
            sign = [(-1.0) ** sum(h) for h in ket["herm"]]
            chunk = max(1, int(6e7 / (len(ket["p"]) * hb * hk)))
            ncd, nab = ket["G"].shape[1], bra["G"].shape[1]
            block = torch.zeros(bra["npairs"], nab, ket["npairs"] * ncd, dtype=torch.float64, device=device)
            for s in range(0, len(bra["p"]), chunk):
                p, q = bra["p"][s:s + chunk, None], ket["p"][None]
                R = _hermite_integrals(bra["L"] + ket["L"], p * q / (p + q), bra["P"][s:s + chunk, None] - ket["P"][None])
                pre = 2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
                nb = p.shape[0]
                half = torch.zeros(ket["npairs"], nb * hb, ncd, dtype=torch.float64, device=device)
                M = torch.stack([torch.stack([sg * pre * R[tuple(a + b for a, b in zip(h, g))] for h in bra["herm"]], 1)
                                 for g, sg in zip(ket["herm"], sign)], -1)  # [nb, hb, nk, hk]
                V = torch.bmm(M.reshape(nb * hb, -1, hk).transpose(0, 1), ket["G"].transpose(1, 2))  # [nk, nb*hb, ncd]
                half.index_add_(0, ket["pair"], V)
                half = half.reshape(ket["npairs"], nb, hb, ncd).permute(1, 2, 0, 3).reshape(nb, hb, -1)
                block.index_add_(0, bra["pair"][s:s + chunk], torch.bmm(bra["G"][s:s + chunk], half))
            rows, cols = bra["row"].reshape(-1), ket["row"].reshape(-1)
            block = block.reshape(len(rows), len(cols))
            swap = lambda r: (r % n) * n + r // n
            for r in (rows, swap(rows)):
                for c in (cols, swap(cols)):
                    out[r[:, None], c[None]] = block
                    out[c[:, None], r[None]] = block.T
    return out


def _fock(I, P, n):
    """J[P] and K[P]."""
    J = (I @ P.reshape(-1)).reshape(n, n)
    K = torch.zeros_like(J)
    T = I.reshape(n, n, n, n)
    for i in range(n):  # K_ij = sum_kl (ik|jl) P_kl
        K[i] = torch.einsum("kjl,kl->j", T[i], P)
    return J, K


def _packed(I, n):
    """The 8-fold unique integrals in packed order."""
    i, j = np.tril_indices(n)
    ij = torch.from_numpy(i * n + j).to(I.device)
    M = I[ij][:, ij]
    a, b = torch.tril_indices(len(ij), len(ij), device=I.device)
    return M[a, b]


def _several_d_centres(t):
    return len(set(t.atom_of_shell[t.L == 2].tolist())) > 1


def _limit(t):
    """About the largest molecule the plain evaluation takes in a few seconds."""
    return t.nbf <= 200 and int(sum(t.nprim)) <= 700


def exact(case, seed):
    kind = case["kind"]
    device = "cuda" if torch.cuda.is_available() else "cpu"

    def ten(a):
        return torch.from_numpy(a).to(device)

    if kind == "batch":
        mols = _batch_molecules(case, seed)
        active = np.random.default_rng(seed).random(len(mols)) < 0.75
        active[0] = True
        parts = []
        for m, (Z, xyz, basis) in enumerate(mols):
            t = basis_io.shell_table(Z, xyz, basis)
            if not active[m]:
                parts.append(np.zeros(t.nbf ** 2))
                continue
            J, K = _fock(_integrals(t, device), ten(_density(t, seed + m)), t.nbf)
            parts.append((J - 0.5 * K).cpu().numpy().ravel())
        return np.concatenate(parts)
    if kind == "scf":
        return None
    t = basis_io.shell_table(*_geometry(case["mol"], case["size"], seed), case["basis"])
    if not _limit(t) or (not case["exact"] and _several_d_centres(t)):
        return None
    n = t.nbf
    I = _integrals(t, device)
    if kind == "uhf":
        Pa = _density(t, seed, electrons=1.0)
        Pb = Pa + _density(t, seed + 1, electrons=1.0) * 0.1
        Ja, Ka = _fock(I, ten(Pa), n)
        Jb, Kb = _fock(I, ten(Pb), n)
        return [(Ja + Jb - Ka).cpu().numpy(), (Ja + Jb - Kb).cpu().numpy()]
    if kind == "precision":
        P = _density(t, seed)
        out = []
        for D in (P, P + 1e-3 * _density(t, seed + 1)):
            J, K = _fock(I, ten(D), n)
            out.append((J - 0.5 * K).cpu().numpy())
        return out
    if kind == "packed":
        return _packed(I, n).cpu().numpy()
    if kind == "ovov":
        nocc = max(1, sum(_geometry(case["mol"], case["size"], seed)[0]) // 2)
        C = ten(_orbitals(n, seed))
        T = (I.reshape(n * n * n, n) @ C[:, nocc:]).reshape(n * n, n, n - nocc)
        T = torch.einsum("xkb,kj->xjb", T, C[:, :nocc]).reshape(n, n, -1)
        T = torch.einsum("mnx,na->max", T, C[:, nocc:])
        ov = nocc * (n - nocc)
        return torch.einsum("max,mi->iax", T, C[:, :nocc]).reshape(ov, ov).cpu().numpy()
    J, K = _fock(I, ten(_density(t, seed)), n)
    return (J - 0.5 * K).cpu().numpy()
