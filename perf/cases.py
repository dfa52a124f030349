"""What a user of this package has it do, as measurable cases.

A case is one call of a public entry point at one size: a direct-SCF Fock build
(`FockBuilder.jk`, eager or as a replayed capture), the nuclear forces of a
converged density (`rhf_gradient`), the one-electron matrices
(`FockBuilder.one_electron`), a prepared batch of raw shell-quartet integrals
(`EriPlan.run`) and a whole SCF (`scf_diis`).  Molecules are the package's
seeded water clusters and all-trans alkanes with its own basis sets, the raw
batches its random contracted shells over all 21 classes.

The density of a Fock build or of forces is the Wolfsberg-Helmholz guess of the
molecule (D = 2 C_occ C_occ^T of F_ij = 1.75/2 S_ij (e_i + e_j)), computed here
in numpy: idempotent, with the right electron count and the decay of a real one.

`exact` evaluates small cases from the Gaussians alone by McMurchie-Davidson in
64-bit torch (derivatives by autograd).
"""
from __future__ import annotations

import itertools
import math

import numpy as np
import torch

from segfault_py_gb300 import geometry
from segfault_py_gb300.fock import FockBuilder
from segfault_py_gb300.grad import rhf_gradient
from segfault_py_gb300.molecule import Molecule
from segfault_py_gb300.scf import SCFResult, scf_diis

CUTOFF = 1e-12


def listed():
    water, alkane = "water", "alkane"
    return [
        # the smallest Fock build of an SCF: one water, minimal basis, all FP64
        dict(name="fock_h2o_sto3g_fp64", kind="fock", system=water, n=1, basis="sto-3g", precision="fp64",
             fp32_cutoff=1e-5, call="eager"),
        # a small molecule in the FP32 + FP64 mode at the builder's default FP32 cutoff
        dict(name="fock_water2_631gs_mixed", kind="fock", system=water, n=2, basis="6-31g*", precision="mixed",
             fp32_cutoff=1e-5, call="eager"),
        # the benchmark's build: FP32 + double-float, captured once and replayed every SCF iteration
        dict(name="fock_water8_631gs_mixed_df_replay", kind="fock", system=water, n=8, basis="6-31g*",
             precision="mixed_df", fp32_cutoff=1e-2, call="replay"),
        # the accuracy reference of the mixed modes at the benchmark's larger cluster
        dict(name="fock_water16_631gs_fp64", kind="fock", system=water, n=16, basis="6-31g*", precision="fp64",
             fp32_cutoff=1e-2, call="eager"),
        # a mid-sized chain, every quartet in double-float
        dict(name="fock_hexane_631gs_df", kind="fock", system=alkane, n=6, basis="6-31g*", precision="df",
             fp32_cutoff=1e-2, call="eager"),
        # the largest molecule of the benchmark, in the mode it is run in
        dict(name="fock_c20h42_631gss_mixed_df", kind="fock", system=alkane, n=20, basis="6-31g**",
             precision="mixed_df", fp32_cutoff=1e-2, call="eager"),
        # forces of a small molecule in FP64 (geometry optimisation, finite-difference checks)
        dict(name="forces_water2_631gs_fp64", kind="forces", system=water, n=2, basis="6-31g*", precision="fp64",
             fp32_cutoff=1e-2),
        # the benchmark's forces: FP32 + double-float
        dict(name="forces_water8_631gs_mixed_df", kind="forces", system=water, n=8, basis="6-31g*",
             precision="mixed_df", fp32_cutoff=1e-2),
        # S, T, V of a new geometry
        dict(name="one_electron_water16_631gs", kind="one_electron", system=water, n=16, basis="6-31g*"),
        # raw integrals in FP64 for a program that keeps them (dense tensors, checks)
        dict(name="eri_batch_fp64", kind="eri", nq=10007, nshell=300, precision="fp64"),
        # the raw-integral stress batch in double-float
        dict(name="eri_batch_df", kind="eri", nq=60000, nshell=600, precision="df"),
        # a whole SCF from the geometry, defaults of the driver, FP32 + double-float
        dict(name="scf_water2_631gs_mixed_df", kind="scf", system=water, n=2, basis="6-31g*", precision="mixed_df"),
    ]


# largest molecule drawn per precision: no drawn build costs more than the listed (H2O)16 FP64 one
LARGEST = {"fp64": (14, 11), "mixed": (16, 15), "mixed_df": (16, 20), "df": (16, 15)}


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["fock"] * 5 + ["forces"] * 2 + ["one_electron", "eri", "eri", "scf"])
    if kind == "eri":
        precision = rng.choice(["fp64", "df"])
        return dict(kind=kind, nq=_log_int(rng, 500, 40000 if precision == "fp64" else 100000),
                    nshell=rng.randint(80, 600), precision=precision)
    system = rng.choice(["water", "water", "alkane"])
    col, least = (0, 1) if system == "water" else (1, 3)   # the chain builder starts at propane
    basis = rng.choice(["sto-3g", "6-31g", "6-31g*", "6-31g*", "6-31g**"])
    if kind == "one_electron":
        return dict(kind=kind, system=system, n=_log_int(rng, least, 16), basis=basis)
    if kind == "scf":
        return dict(kind=kind, system="water", n=rng.randint(1, 3), basis=basis,
                    precision=rng.choice(["fp64", "mixed_df"]))
    precision = rng.choice(["fp64", "mixed", "mixed_df", "mixed_df", "df"])
    cutoff32 = rng.choice([1e-2, 1e-2, 1e-5])
    if kind == "forces":
        top = 9 if precision == "mixed_df" else 5
        return dict(kind=kind, system=system, n=_log_int(rng, least, top), basis=basis, precision=precision,
                    fp32_cutoff=cutoff32)
    return dict(kind=kind, system=system, n=_log_int(rng, least, LARGEST[precision][col]), basis=basis,
                precision=precision, fp32_cutoff=cutoff32, call=rng.choice(["eager", "eager", "replay"]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _molecule(case, seed):
    make = geometry.water_cluster if case["system"] == "water" else geometry.alkane
    sym, xyz = make(case["n"], seed=seed)
    return Molecule.from_geometry(sym, xyz, case["basis"])


# orbital energies (hartree) of the guess: core s, valence s, valence p, polarisation
LEVELS = {"O": (-20.6, -1.24, -0.63, 1.0), "C": (-11.3, -0.71, -0.41, 1.0), "H": (-0.5, -0.5, 1.0, 1.0)}


def _guess(mol, table):
    """(D, F): Wolfsberg-Helmholz Fock matrix and its aufbau density, numpy FP64."""
    S = _overlap(table)
    e = np.zeros(len(S))
    seen = set()
    for l, at, o in zip(table["l"], table["atom"], table["ao_offset"]):
        lev = LEVELS[mol.symbols[at]]
        first = (at, l) not in seen
        seen.add((at, l))
        e[o:o + ncart(l)] = (lev[0] if first else lev[1]) if l == 0 else lev[1 + l]
    F = 0.875 * S * (e[:, None] + e[None, :])
    np.fill_diagonal(F, e * np.diagonal(S))
    w, U = np.linalg.eigh(S)
    X = (U / np.sqrt(w)) @ U.T
    _, C = np.linalg.eigh(X @ F @ X)
    C = X @ C[:, :mol.nelectron // 2]
    D = 2.0 * C @ C.T
    return 0.5 * (D + D.T), F


def _batch(case, seed):
    """(shell table, quartets): the classes in equal shares (an output length that the seed does not change),
    in random order, of random contracted shells."""
    table = geometry.random_quartet_shells(case["nshell"], seed=seed)
    rng = np.random.default_rng(seed + 1)
    of_l = [np.where(table["l"] == l)[0] for l in range(3)]
    cls = rng.permutation(np.arange(case["nq"]) % len(geometry.QUARTET_CLASSES))
    q = np.empty((case["nq"], 4), dtype=np.int32)
    for k, (bra, ket) in enumerate(geometry.QUARTET_CLASSES):
        sel = np.where(cls == k)[0]
        for col, l in enumerate(bra + ket):
            q[sel, col] = rng.choice(of_l[l], len(sel))
    return table, q


def prepare(case, seed):
    kind = case["kind"]
    if kind == "eri":
        table, q = _batch(case, seed)
        fb = FockBuilder(table)
        return dict(case=case, fb=fb, plan=fb.eri_plan(q))
    mol = _molecule(case, seed)
    if kind == "scf":
        return dict(case=case, mol=mol)
    fb = FockBuilder(mol, cutoff=CUTOFF, fp32_cutoff=case.get("fp32_cutoff", 1e-5),
                     precision=case.get("precision", "fp64"))
    state = dict(case=case, mol=mol, fb=fb)
    if kind == "one_electron":
        return state
    D, F = (torch.tensor(m, device=fb.device) for m in _guess(mol, fb.table))
    state["D"] = D
    if kind == "forces":
        state["res"] = SCFResult(energy=0.0, e_elec=0.0, e_nuc=mol.e_nuc, iterations=0, converged=True, D=D, F=F,
                                 C=None, eps=None, H=None, S=None)
    elif case["call"] == "replay":
        state["J"], state["K"] = torch.empty_like(D), torch.empty_like(D)
        state["graph"] = fb.capture_jk(D, state["J"], state["K"], native=True)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "eri":
        return state["plan"].run(case["precision"])
    if kind == "scf":
        r = scf_diis(state["mol"], precision=case["precision"])
        return dict(energy=r.energy, D=r.D, F=r.F)
    if kind == "one_electron":
        return state["fb"].one_electron()
    if kind == "forces":
        return rhf_gradient(state["mol"], state["res"], state["fb"])
    if case["call"] == "replay":
        state["graph"].replay()
        return state["J"], state["K"]
    return state["fb"].jk(state["D"])


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------
def ncart(l):
    return (l + 1) * (l + 2) // 2


def _screened(table, cutoff):
    """Per class (l of the four shells, number of quartets, primitive quartets) of the canonical shell
    quartets with Q_ab Q_cd >= cutoff, Q from the s-type bound of each primitive pair."""
    l, npr, off, cen = table["l"], table["nprim"], table["prim_offset"], table["center"]
    pairs = {}
    for a, b in itertools.product(range(len(l)), repeat=2):
        if l[a] < l[b] or (l[a] == l[b] and b > a):
            continue
        x, y = table["exps"][off[a]:off[a + 1], None], table["exps"][None, off[b]:off[b + 1]]
        c = np.abs(table["coefs"][off[a]:off[a + 1], None] * table["coefs"][None, off[b]:off[b + 1]])
        p = x + y
        r = math.dist(cen[a], cen[b])
        q = 5.9 * np.sum(c * np.exp(-x * y / p * r * r) / p / (2 * p) ** 0.25
                         * (y / p * r + p ** -0.5) ** l[a] * (x / p * r + p ** -0.5) ** l[b])
        pairs.setdefault((int(l[a]), int(l[b])), []).append((q, int(npr[a] * npr[b])))
    keys = sorted(pairs)
    out = []
    for i, X in enumerate(keys):
        qx = np.array(sorted(pairs[X], reverse=True))
        for Y in keys[:i + 1]:
            qy = np.array(sorted(pairs[Y], reverse=True))
            n = np.searchsorted(-qy[:, 0], -cutoff / np.maximum(qx[:, 0], 1e-300), side="right")
            if X == Y:
                n = np.minimum(n, np.arange(len(qx)) + 1)
            kc = np.concatenate([[0.0], np.cumsum(qy[:, 1])])
            out.append((X + Y, float(n.sum()), float((qx[:, 1] * kc[n]).sum())))
    return out


def work(case):
    kind = case["kind"]
    if kind == "eri":
        table, q = _batch(case, 0)
        l, npr = table["l"][q], table["nprim"][q]
        nc = np.prod((l + 1) * (l + 2) // 2, axis=1).astype(float)
        roots = l.sum(axis=1) // 2 + 1
        return dict(bytes=float(8 * nc.sum() + 16 * case["nq"]),
                    flops=float((4.0 * npr.prod(axis=1) * roots * nc).sum()))
    mol = _molecule(case, 0)
    t = mol.shell_table()
    n = float(sum(ncart(l) for l in t["l"]))
    tables = 8.0 * (2 * len(t["exps"]) + 4 * len(t["l"]) + 4 * mol.natom)
    if kind == "one_electron":
        # one Hermite table (ntuv values, about six operations each) per primitive pair and nucleus
        k = sum(a * b * math.comb(int(la + lb) + 3, 3) for (la, a), (lb, b)
                in itertools.combinations_with_replacement(list(zip(t["l"], t["nprim"])), 2))
        return dict(bytes=tables + 24 * n * n, flops=6.0 * float(k) * mol.natom)
    flops = 0.0
    for ls, nq, prims in _screened(t, CUTOFF):
        nc = float(np.prod([ncart(l) for l in ls]))
        if kind == "forces":   # nine derivative components per output, root and primitive quartet
            flops += prims * ((sum(ls) + 1) // 2 + 1) * 36.0 * nc
        else:
            flops += prims * (sum(ls) // 2 + 1) * 4.0 * nc + 12.0 * nc * nq
    if kind == "forces":
        return dict(bytes=tables + 16 * n * n + 24 * mol.natom, flops=flops)
    if kind == "scf":   # some twelve iterations of a Fock build and an n^3 eigenproblem
        return dict(bytes=tables + 16 * n * n, flops=12.0 * (flops + 20.0 * n ** 3))
    return dict(bytes=tables + 24 * n * n, flops=flops)


# ---------------------------------------------------------------------------
# exact values: McMurchie-Davidson in 64-bit torch
# ---------------------------------------------------------------------------
CART = {0: [(0, 0, 0)], 1: [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
        2: [(2, 0, 0), (1, 1, 0), (1, 0, 1), (0, 2, 0), (0, 1, 1), (0, 0, 2)]}


def _norms(l):
    """Factors of the Cartesian components relative to x^l (each component normalised by itself)."""
    return [math.sqrt(3.0) if l == 2 and max(c) == 1 else 1.0 for c in CART[l]]


def _tuv(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


class _Boys(torch.autograd.Function):
    """F_0 .. F_M of T, stacked last; dF_m/dT = -F_{m+1}."""

    @staticmethod
    def forward(ctx, T, M):
        n = M + 1
        small = T < 35.0
        ts = torch.where(small, T, torch.ones_like(T))
        term = torch.full_like(T, 1.0 / (2 * n + 1))
        s = term.clone()
        for i in range(1, 160):
            term = term * (2.0 * ts / (2 * n + 2 * i + 1))
            s = s + term
        e = torch.exp(-T)
        F = [None] * (n + 1)
        F[n] = torch.exp(-ts) * s
        for m in range(n - 1, -1, -1):
            F[m] = (2.0 * ts * F[m + 1] + torch.exp(-ts)) / (2 * m + 1)
        tl = torch.where(small, torch.ones_like(T), T)
        g = 0.5 * torch.sqrt(math.pi / tl) * torch.erf(torch.sqrt(tl))
        for m in range(n + 1):
            F[m] = torch.where(small, F[m], g)
            g = ((2 * m + 1) * g - e) / (2.0 * tl)
        F = torch.stack(F, dim=-1)
        ctx.save_for_backward(F)
        return F[..., :n].clone()

    @staticmethod
    def backward(ctx, grad):
        F, = ctx.saved_tensors
        return -(grad * F[..., 1:]).sum(dim=-1), None


def _hermite_r(L, p, P):
    """[N, ntuv(L)]: Hermite Coulomb integrals R_tuv(p, P) for the rows P [N, 3]."""
    F = _Boys.apply(p * (P * P).sum(dim=1), L)
    memo = {}

    def R(n, t, u, v):
        k = (n, t, u, v)
        if k not in memo:
            if t:
                r = P[:, 0] * R(n + 1, t - 1, u, v) + ((t - 1) * R(n + 1, t - 2, u, v) if t > 1 else 0.0)
            elif u:
                r = P[:, 1] * R(n + 1, t, u - 1, v) + ((u - 1) * R(n + 1, t, u - 2, v) if u > 1 else 0.0)
            elif v:
                r = P[:, 2] * R(n + 1, t, u, v - 1) + ((v - 1) * R(n + 1, t, u, v - 2) if v > 1 else 0.0)
            else:
                r = (-2.0 * p) ** n * F[:, n]
            memo[k] = r
        return memo[k]

    return torch.stack([R(0, *k) for k in _tuv(L)], dim=1)


def _expansion(la, lb, al, be, A, B):
    """E[d][i][j][t] of each row's primitive pair, the Gaussian product factor in each direction."""
    p = al + be
    out = []
    for d in range(3):
        X = A[:, d] - B[:, d]
        pa, pb = -be / p * X, al / p * X
        E = {(0, 0): [torch.exp(-al * be / p * X * X)]}

        def up(e, x):
            get = lambda t: e[t] if 0 <= t < len(e) else 0.0
            return [get(t - 1) / (2 * p) + x * get(t) + (t + 1) * get(t + 1) for t in range(len(e) + 1)]

        for i in range(la):
            E[(i + 1, 0)] = up(E[(i, 0)], pa)
        for i in range(la + 1):
            for j in range(lb):
                E[(i, j + 1)] = up(E[(i, j)], pb)
        out.append(E)
    return out


def _pair_hermite(la, lb, E):
    """[N, na*nb, ntuv(la+lb)] Hermite coefficients of the component products."""
    zero = torch.zeros_like(E[0][(0, 0)][0])
    rows = []
    for (a, na), (b, nb) in itertools.product(zip(CART[la], _norms(la)), zip(CART[lb], _norms(lb))):
        e = [E[d][(a[d], b[d])] for d in range(3)]
        rows.append(torch.stack([na * nb * e[0][t] * e[1][u] * e[2][v] if t < len(e[0]) and u < len(e[1])
                                 and v < len(e[2]) else zero for t, u, v in _tuv(la + lb)], dim=1))
    return torch.stack(rows, dim=1)


class _Shells:
    """A shell table in 64-bit tensors; `xyz` the shell centres (may carry gradients)."""

    def __init__(self, table, device, xyz=None):
        self.l, self.n, self.o = (np.asarray(table[k]) for k in ("l", "nprim", "prim_offset"))
        self.ao = np.asarray(table["ao_offset"])
        self.exps = torch.tensor(np.asarray(table["exps"]), device=device)
        self.coefs = torch.tensor(np.asarray(table["coefs"]), device=device)
        self.xyz = torch.tensor(np.asarray(table["center"]), device=device) if xyz is None else xyz
        self.device = device

    def primitives(self, shells):
        """Rows (index into the list, one global primitive per shell) of all primitive combinations of the
        shell tuples [M, k]."""
        counts = self.n[shells]
        total = counts.prod(axis=1)
        row = np.repeat(np.arange(len(shells)), total)
        local = np.arange(total.sum()) - np.repeat(np.cumsum(total) - total, total)
        prim = np.empty((len(row), shells.shape[1]), dtype=np.int64)
        for k in range(shells.shape[1] - 1, -1, -1):
            prim[:, k] = self.o[shells[row, k]] + local % counts[row, k]
            local //= counts[row, k]
        return row, prim

    def classes(self, shells):
        ls = self.l[shells]
        for key in np.unique(ls, axis=0):
            yield tuple(int(v) for v in key), np.where((ls == key).all(axis=1))[0]

    def eri(self, quartets, limit=150_000, each=None):
        """Integrals of shell quartets, a list of [na, nb, nc, nd] stacks per class with their rows; `each`, if
        given, takes (rows, block stack) of every chunk instead."""
        found = []
        for (la, lb, lc, ld), sel in self.classes(quartets):
            total = self.n[quartets[sel]].prod(axis=1)
            part = (np.cumsum(total) - 1) // limit
            for k in np.unique(part):
                rows = sel[part == k]
                q = quartets[rows]
                row, prim = self.primitives(q)
                e = [self.exps[prim[:, k]] for k in range(4)]
                c = self.coefs[prim].prod(dim=1)
                X = [self.xyz[q[row, k]] for k in range(4)]
                p, r = e[0] + e[1], e[2] + e[3]
                P = (e[0][:, None] * X[0] + e[1][:, None] * X[1]) / p[:, None]
                Q = (e[2][:, None] * X[2] + e[3][:, None] * X[3]) / r[:, None]
                bra = _pair_hermite(la, lb, _expansion(la, lb, e[0], e[1], X[0], X[1]))
                ket = _pair_hermite(lc, ld, _expansion(lc, ld, e[2], e[3], X[2], X[3]))
                L = la + lb + lc + ld
                R = _hermite_r(L, p * r / (p + r), P - Q)
                at = {k: i for i, k in enumerate(_tuv(L))}
                idx = [[at[tuple(x + y for x, y in zip(m, n))] for n in _tuv(lc + ld)] for m in _tuv(la + lb)]
                sign = torch.tensor([(-1.0) ** sum(n) for n in _tuv(lc + ld)], dtype=R.dtype, device=R.device)
                R = R[:, torch.tensor(idx, device=R.device)] * sign
                f = c * (2.0 * math.pi ** 2.5) / (p * r * torch.sqrt(p + r))
                v = torch.einsum("nih,nhk,njk->nij", bra * f[:, None, None], R, ket)
                out = torch.zeros((len(rows),) + v.shape[1:], dtype=v.dtype, device=v.device)
                out = out.index_add(0, torch.tensor(row, device=v.device), v)
                out = out.reshape(len(rows), ncart(la), ncart(lb), ncart(lc), ncart(ld))
                found.append((rows, out)) if each is None else each(rows, out)
        return found

    def pairs(self):
        m = len(self.l)
        return np.array([(a, b) for a in range(m) for b in range(a + 1)])

    def quartets(self):
        pr = self.pairs()
        i, j = np.tril_indices(len(pr))
        return np.concatenate([pr[i], pr[j]], axis=1)

    def aos(self, shells):
        """AO indices [M, ncart] of a column of shells of one l."""
        l = int(self.l[shells[0]])
        return torch.tensor(self.ao[shells][:, None] + np.arange(ncart(l)), device=self.device)

    def one_electron(self, atoms=None, charges=None):
        """S, and with atoms T and V, as [nao, nao]."""
        n = int(self.ao[-1] + ncart(self.l[-1]))
        mats = [torch.zeros((n, n), dtype=torch.float64, device=self.device) for _ in range(1 if atoms is None else 3)]
        for (la, lb), sel in self.classes(self.pairs()):
            q = self.pairs()[sel]
            row, prim = self.primitives(q)
            al, be = self.exps[prim[:, 0]], self.exps[prim[:, 1]]
            c, p = self.coefs[prim].prod(dim=1), al + be
            A, B = self.xyz[q[row, 0]], self.xyz[q[row, 1]]
            E = _expansion(la, lb + 2, al, be, A, B)
            sp = c * (math.pi / p) ** 1.5
            blocks = []
            S, T = [], []
            for (a, fa), (b, fb) in itertools.product(zip(CART[la], _norms(la)), zip(CART[lb], _norms(lb))):
                s = [{k: E[d][(a[d], b[d] + k)][0] if b[d] + k >= 0 else 0.0 for k in (-2, 0, 2)} for d in range(3)]
                S.append(fa * fb * sp * s[0][0] * s[1][0] * s[2][0])
                t = be * (2 * sum(b) + 3) * s[0][0] * s[1][0] * s[2][0]
                for d in range(3):
                    rest = s[(d + 1) % 3][0] * s[(d + 2) % 3][0]
                    t = t - (2.0 * be * be * s[d][2] + 0.5 * b[d] * (b[d] - 1) * s[d][-2]) * rest
                T.append(fa * fb * sp * t)
            blocks.append(torch.stack(S, dim=1))
            if atoms is not None:
                blocks.append(torch.stack(T, dim=1))
                H = _pair_hermite(la, lb, E)
                P = (al[:, None] * A + be[:, None] * B) / p[:, None]
                m, k = len(P), len(atoms)
                R = _hermite_r(la + lb, p.repeat_interleave(k),
                               (P[:, None, :] - atoms[None]).reshape(-1, 3)).reshape(m, k, -1)
                R = -(R * charges[None, :, None]).sum(dim=1)
                blocks.append(torch.einsum("nih,nh->ni", H, R) * (c * 2.0 * math.pi / p)[:, None])
            i, j = self.aos(q[:, 0]), self.aos(q[:, 1])
            at = torch.tensor(row, device=self.device)
            for k, v in enumerate(blocks):
                v = torch.zeros((len(q), v.shape[1]), dtype=v.dtype, device=v.device).index_add(0, at, v)
                v = v.reshape(len(q), i.shape[1], j.shape[1])
                I, J = i[:, :, None].expand_as(v), j[:, None, :].expand_as(v)
                mats[k] = mats[k].index_put((I, J), v).index_put((J, I), v)
        return mats


def _overlap(table):
    return _Shells(table, "cpu").one_electron()[0].numpy()


def _exact_tensor(sh):
    n = int(sh.ao[-1] + ncart(sh.l[-1]))
    T = torch.zeros((n,) * 4, dtype=torch.float64, device=sh.device)
    quartets = sh.quartets()
    for rows, v in sh.eri(quartets):
        ix = [sh.aos(quartets[rows, k]) for k in range(4)]
        ix = [x.reshape([len(x)] + [-1 if m == k else 1 for m in range(4)]).expand_as(v) for k, x in enumerate(ix)]
        for a, b, c, d in itertools.product((0, 1), (0, 1), (0, 1), (0,)):
            bra = (ix[0], ix[1]) if not a else (ix[1], ix[0])
            ket = (ix[2], ix[3]) if not b else (ix[3], ix[2])
            T[(*bra, *ket) if not c else (*ket, *bra)] = v
    return T


def _exact_jk(T, D):
    return torch.einsum("pqrs,rs->pq", T, D), torch.einsum("prqs,rs->pq", T, D)


def _exact_scf(mol, table, dev, tol=1e-8, maxiter=100):
    """The driver's iteration: Pulay extrapolation from the third step on, stop at |dE| <= tol."""
    atoms, Z = (torch.tensor(np.ascontiguousarray(x), device=dev) for x in (mol.xyz__, mol.numbers.astype(float)))
    sh = _Shells(table, dev)
    T4 = _exact_tensor(sh)
    S, T, V = sh.one_electron(atoms, Z)
    H = T + V
    w, U = torch.linalg.eigh(S)
    X = (U / torch.sqrt(w)) @ U.T
    F, Fs, res, last = H, [], [], math.inf
    i, j = torch.triu_indices(len(Z), len(Z), 1, device=dev)
    nuc = float((Z[i] * Z[j] / torch.linalg.norm(atoms[i] - atoms[j], dim=1)).sum())
    for step in range(maxiter + 1):
        C = X @ torch.linalg.eigh(X @ F @ X)[1][:, :mol.nelectron // 2]
        D = 2.0 * C @ C.T
        J, K = _exact_jk(T4, D)
        F = H + J - 0.5 * K
        e = float(0.5 * (D * (H + F)).sum())
        if abs(e - last) <= tol:
            break
        last = e
        if step < 2:
            continue
        Fs, res = Fs[-6:] + [F], res[-6:] + [X @ (F @ D @ S - S @ D @ F) @ X]
        n = len(Fs)
        B = torch.full((n + 1, n + 1), -1.0, dtype=F.dtype, device=dev)
        B[n, n] = 0.0
        B[:n, :n] = torch.tensor([[float((x * y).sum()) for x in res] for y in res], dtype=F.dtype)
        rhs = torch.zeros(n + 1, dtype=F.dtype, device=dev)
        rhs[n] = -1.0
        F = torch.einsum("i,iab->ab", torch.linalg.solve(B, rhs)[:n], torch.stack(Fs))
    return dict(energy=e + nuc, D=D, F=F)


def _exact_forces(mol, table, D, F):
    dev = D.device
    atoms, Z = (torch.tensor(np.ascontiguousarray(x), device=dev) for x in (mol.xyz__, mol.numbers.astype(float)))
    atoms.requires_grad_(True)
    sh = _Shells(table, dev, xyz=atoms[torch.tensor(np.asarray(table["atom"], dtype=np.int64), device=dev)])
    S, T, V = sh.one_electron(atoms, Z)
    E = (D * (T + V)).sum() - (0.5 * (D @ F @ D) * S).sum()
    i, j = torch.triu_indices(len(Z), len(Z), 1, device=dev)
    E = E + (Z[i] * Z[j] / torch.linalg.norm(atoms[i] - atoms[j], dim=1)).sum()
    E.backward(retain_graph=True)
    quartets = sh.quartets()
    same = lambda x, y: 0.5 if x == y else 1.0
    weight = np.array([8.0 * same(a, b) * same(c, d) * same((a, b), (c, d)) for a, b, c, d in quartets.tolist()])

    def each(rows, v):
        a, b, c, d = (sh.aos(quartets[rows, k]) for k in range(4))
        B = lambda x, y: D[x[:, :, None], y[:, None, :]]
        G = (0.5 * torch.einsum("nij,nkl->nijkl", B(a, b), B(c, d))
             - 0.125 * (torch.einsum("nik,njl->nijkl", B(a, c), B(b, d))
                        + torch.einsum("nil,njk->nijkl", B(a, d), B(b, c))))
        w = torch.tensor(weight[rows], device=dev)
        (G * v * w[:, None, None, None, None]).sum().backward(retain_graph=True)

    sh.eri(quartets, limit=40_000, each=each)
    return atoms.grad.detach()


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "eri":
        if case["nq"] > 12000:
            return None
        table, q = _batch(case, seed)
        q = np.asarray(q, dtype=np.int64)
        nc = np.prod((table["l"][q] + 1) * (table["l"][q] + 2) // 2, axis=1).astype(np.int64)
        off = np.cumsum(nc) - nc
        out = torch.empty(int(nc.sum()), dtype=torch.float64, device=dev)

        def each(rows, v):
            at = torch.tensor(off[rows], device=dev)[:, None] + torch.arange(v[0].numel(), device=dev)
            out[at] = v.reshape(len(rows), -1)

        _Shells(table, dev).eri(q, each=each)
        return out
    mol = _molecule(case, seed)
    table = mol.shell_table()
    if kind == "one_electron":
        xyz, Z = (torch.tensor(np.ascontiguousarray(x), device=dev) for x in (mol.xyz__, mol.numbers.astype(float)))
        return tuple(_Shells(table, dev).one_electron(xyz, Z))
    if mol.nao > 40:
        return None
    if kind == "scf":
        return _exact_scf(mol, table, dev)
    D, F = (torch.tensor(m, device=dev) for m in _guess(mol, table))
    if kind == "forces":
        return _exact_forces(mol, table, D, F)
    return _exact_jk(_exact_tensor(_Shells(table, dev)), D)
