"""The engine's measured workloads: what a program that uses it calls, over
the sizes it calls it with.

A case is a dict of plain values.  `prepare` makes what such a program holds
before the call (a basis and its plan, the densities on the GPU), `run` is
one call through the public entry points, `work` the bytes and flops the call
cannot do without, `tolerance` how far another correct implementation of the
same precision may be off, and `exact` the same numbers by plain torch in 64
bits: McMurchie-Davidson integrals from Hermite expansions and Boys values,
with none of the engine's code.

Systems are seeded random clusters.  Recipe "cluster" is the 64-atom
workload's shells (s x3, p x2 contracted to degree 3, d x2, f x1: 31 AO an
atom), "small" the 6-atom workload's (s x3, p x2, d x1: 15 AO an atom) and
"split" a split-valence set with polarisation (s contracted to 6, 3, 1, p to
3, 1, one d: 15 AO an atom), whose contraction degrees are ragged.
"""

from __future__ import annotations

import itertools
import math

import numpy as np
import torch

from felizjueves_b200 import _lib, configs
from felizjueves_b200.batch import BatchBuilder
from felizjueves_b200.df import DFEngine
from felizjueves_b200.fock import FockEngine
from felizjueves_b200.shell import Basis, Shell, primitive_norm

TAU = 1e-12


def listed() -> list[dict]:
    return [
        # one SCF iteration's G build of a small molecule, replayed as the
        # loop's captured graph (the 6-atom workload): latency and launches
        fock("scf_small_6at", "small", 6, graph=True),
        # the smallest molecule of the uneven batch, built once
        fock("fock_3at", "cluster", 3),
        # an ordinary odd-sized molecule with f functions
        fock("fock_13at", "cluster", 13),
        # a large molecule: throughput of every class kernel
        fock("fock_32at", "cluster", 32),
        # the mixed-precision build (default 1e-9 rule, with its error check)
        # inside an SCF loop of a small molecule
        fock("routed_scf_7at", "cluster", 7, graph=True, threshold=1e-9),
        # the mixed-precision build of a large molecule
        fock("routed_24at", "cluster", 24, threshold=1e-8),
        # many small molecules of uneven size in one merged build, replayed as
        # its captured graph
        {"name": "batch_12mol", "kind": "batch", "molecules": 12, "max_atoms": 12, "threshold": 0.0},
        # J alone (a J-only or hybrid-free functional), FP64
        {"name": "coulomb_9at", "kind": "coulomb", "recipe": "cluster", "atoms": 9, "threshold": 0.0},
        # J alone with the FP32 tier for small record pairs
        {"name": "coulomb_mixed_16at", "kind": "coulomb", "recipe": "cluster", "atoms": 16, "threshold": 1e-9},
        # density fitting when (mn|P) is not held: integrals, J and K
        {"name": "df_streamed_16at", "kind": "df_streamed", "atoms": 16, "block": 768},
        # density fitting with the factors held: the contractions alone
        {"name": "df_jk_8at", "kind": "df_jk", "atoms": 8},
        # S, T, V and H of the 64-atom workload, once per geometry
        {"name": "onee_64at", "kind": "onee", "recipe": "cluster", "atoms": 64},
    ]


def fock(name: str | None, recipe: str, atoms: int, *, graph: bool = False, threshold: float = 0.0) -> dict:
    c = {"kind": "fock", "recipe": recipe, "atoms": atoms, "graph": graph, "threshold": threshold}
    return dict(c, name=name) if name else c


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    kind = rng.choice(["fock"] * 5 + ["routed"] * 3 + ["batch", "coulomb", "coulomb", "df_streamed", "df_jk", "onee"])
    if kind == "fock":
        recipe = rng.choice(["cluster", "cluster", "small", "split"])
        hi = {"cluster": 29, "small": 29, "split": 17}[recipe]
        return fock(None, recipe, _log_int(rng, 3, hi), graph=rng.random() < 0.5)
    if kind == "routed":
        return fock(None, "cluster", _log_int(rng, 3, 26), graph=rng.random() < 0.5,
                    threshold=rng.choice([1e-9, 1e-8]))
    if kind == "batch":
        return {"kind": "batch", "molecules": rng.randint(2, 16), "max_atoms": rng.randint(4, 13),
                "threshold": rng.choice([0.0, 1e-9])}
    if kind == "coulomb":
        return {"kind": "coulomb", "recipe": rng.choice(["cluster", "small"]), "atoms": _log_int(rng, 3, 17),
                "threshold": rng.choice([0.0, 1e-9])}
    if kind == "df_streamed":
        return {"kind": "df_streamed", "atoms": _log_int(rng, 3, 19), "block": rng.choice([384, 768])}
    if kind == "df_jk":
        return {"kind": "df_jk", "atoms": _log_int(rng, 2, 12)}
    return {"kind": "onee", "recipe": rng.choice(["cluster", "small"]), "atoms": _log_int(rng, 3, 64)}


# -- inputs ---------------------------------------------------------------------


def _system(recipe: str, atoms: int, seed: int):
    """(workload, nuclei) of a seeded cluster in one of the recipes."""
    if recipe == "cluster":
        w = configs.cluster(atoms, seed)
    else:
        rng = np.random.default_rng(seed)
        xyz = configs.sample_geometry(rng, atoms, (atoms / configs.C1_DENSITY) ** (1.0 / 3.0), 0.9)
        shells = [s for c in xyz for s in (_split_shells if recipe == "split" else configs.atom_shells)(
            tuple(map(float, c)))]
        B = Basis(tuple(shells))
        w = configs.Workload(f"{recipe}{atoms}", B, configs.random_density(rng, B.n_ao, 2 * atoms), TAU, 4, xyz,
                             seed, 2 * atoms)
    return w, [(float(1 + i % 9), tuple(map(float, c))) for i, c in enumerate(w.coords)]


def _split_shells(centre) -> list[Shell]:
    def shell(l, ex, co):
        return Shell(l, centre, ex, [k * primitive_norm(l, e) for e, k in zip(ex, co)])

    ex6 = [0.6 * 3.6 ** k for k in range(6)]
    return [shell(0, ex6, [0.05, 0.25, 0.45, 0.28, 0.12, 0.04]),
            shell(0, [9.0, 2.1, 0.65], [-0.12, -0.14, 1.15]), shell(0, [0.25], [1.0]),
            shell(1, [9.0, 2.1, 0.65], [0.07, 0.34, 0.73]), shell(1, [0.25], [1.0]),
            shell(2, [0.8], [1.0])]


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "batch":
        # the sizes are the case's, the geometries and densities the seed's
        sizes = np.random.default_rng(case["molecules"]).integers(3, case["max_atoms"] + 1, size=case["molecules"])
        bb = BatchBuilder([configs.cluster(int(n), 1000 * (seed % 100000) + i) for i, n in enumerate(sizes)])
        t = case["threshold"]
        bb.capture_merged("build", _lib.FJB_ROUTED if t else _lib.FJB_FP64, t)
        return {"batch": bb}
    w, nuclei = _system(case.get("recipe", "cluster"), case["atoms"], seed)
    if kind in ("df_streamed", "df_jk"):
        df = DFEngine(w.basis, configs.aux_basis(w))
        D = torch.tensor(w.D, device="cuda")
        factor = df.metric_factor()
        if kind == "df_streamed":
            return {"df": df, "D": D, "factor": factor, "block": case["block"]}
        n = w.n_ao
        T = df.eri3_block(0, len(df.aux.shells), tau=TAU).view(n * n, df.aux.n_ao)
        return {"df": df, "D": D, "B": (T @ factor[0]).T.reshape(-1, n, n).contiguous()}
    eng = FockEngine(w.basis)
    if kind == "onee":
        return {"engine": eng, "nuclei": nuclei}
    D = torch.tensor(w.D, device="cuda")
    if kind == "coulomb":
        return {"engine": eng, "D": D, "J": torch.empty_like(D), "threshold": case["threshold"]}
    eng.plan(w.D, TAU, w.n_mag, export=False)
    return {"engine": eng, "D": D, "out": tuple(torch.empty_like(D) for _ in range(3)), "graph": case["graph"],
            "threshold": case["threshold"]}


def run(state: dict):
    if "batch" in state:
        state["batch"].replay("build")
        return state["batch"].out
    if "block" in state:
        return state["df"].jk_streamed(state["D"], tau=TAU, block=state["block"], factor=state["factor"])
    if "B" in state:
        return state["df"].jk(state["D"], "bf16x3", B=state["B"])
    eng = state["engine"]
    if "nuclei" in state:
        return eng.one_electron(state["nuclei"])
    if "J" in state:
        return eng.coulomb(state["D"], tau=TAU, J=state["J"], threshold=state["threshold"])
    J, K, G = state["out"]
    t = state["threshold"]
    return eng.build(state["D"], J=J, K=K, G=G, precision=_lib.FJB_ROUTED if t else _lib.FJB_FP64, threshold=t,
                     graph=state["graph"])


# -- the least work -------------------------------------------------------------

# GFLOP of one build by the per-quartet operation counts of the engine's cost
# table, over the quartets the screen keeps at TAU (seeded clusters).
_GFLOP = ((3, 1.14), (6, 11.5), (8, 28.9), (13, 164.0), (16, 294.0), (24, 990.0), (32, 2021.0), (40, 4206.0))


def _fock_flops(recipe: str, atoms: int) -> float:
    x, y = zip(*((math.log(n), math.log(g)) for n, g in _GFLOP))
    g = math.exp(float(np.interp(math.log(max(atoms, 3)), x, y))) * 1e9
    return g if recipe == "cluster" else 0.115 * g  # 1.33 GFLOP at 6 atoms of the "small" recipe


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "batch":
        mean = (3 + case["max_atoms"]) / 2
        return {"bytes": case["molecules"] * 4 * 8 * (31 * mean) ** 2,
                "flops": case["molecules"] * 1.3 * _fock_flops("cluster", mean)}
    atoms, recipe = case["atoms"], case.get("recipe", "cluster")
    n = atoms * (31 if recipe == "cluster" else 15)
    if kind in ("fock", "coulomb"):
        # J alone: the Hermite contraction of the surviving record pairs
        f = _fock_flops(recipe, atoms) * (1.2 if kind == "coulomb" else 1.0)
        return {"bytes": 8 * n * n * (4 if kind == "fock" else 2), "flops": f}
    if kind == "onee":
        shells = atoms * (8 if recipe == "cluster" else 6)
        return {"bytes": 4 * 8 * n * n, "flops": shells * (shells + 1) / 2 * 4.5 * (300.0 + 250.0 * atoms)}
    nx, occ = 90 * atoms, 2 * atoms
    if kind == "df_jk":
        return {"bytes": 8 * (nx * n * n + 3 * n * n), "flops": 4.0 * nx * n ** 3 + 4.0 * nx * n * n}
    return {"bytes": 8 * (3 * n * n + nx * nx),
            "flops": 150.0 * n * n * nx + 4.0 * n * n * nx + 2.0 * n * n * nx * occ + 2.0 * n * occ * nx * (nx + n)}


def tolerance(case: dict) -> dict:
    kind = case["kind"]
    if kind == "df_jk":
        # K from six products of BF16 parts summed in FP32
        return {"rel": 2e-5, "max": 8e-4}
    if kind == "df_streamed":
        # the same, behind a metric inverse of condition 1e12
        return {"rel": 1e-4, "max": 2e-3}
    if kind == "onee":
        return {"rel": 1e-13, "max": 1e-11}
    if kind == "coulomb":
        return {"rel": 1e-13 if not case["threshold"] else 1e-12, "max": 1e-11 if not case["threshold"] else 1e-10}
    if case["threshold"]:
        # FP32 recurrences on quartets whose bound is under the threshold:
        # about four times the distance to the FP64 build
        return {"rel": 2e-11, "max": 2e-9}
    # about four times the distance to exact() (1e-14 to 4e-14 in G: the
    # screen at TAU and the pair records' rounding)
    return {"rel": 5e-14, "max": 2e-12}


# -- the same in plain torch, 64 bits --------------------------------------------

# ERI elements an exact() may form: 496 AO, about 15 s on the GPU
_MOST_ELEMENTS = 2.6e10


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "batch":
        return None
    dev = torch.device("cuda")
    if kind == "df_jk":
        s = prepare(case, seed)
        B, D = s["B"], s["D"]
        J = torch.einsum("qmn,q->mn", B, torch.einsum("qmn,mn->q", B, D))
        return J, torch.einsum("qml,qln->mn", torch.matmul(B, D), B)
    if kind == "df_streamed":
        return None  # set by the metric's smallest eigenvalues, not by the sums
    w, nuclei = _system(case["recipe"], case["atoms"], seed)
    if kind == "onee":
        return _one_electron(w.basis, nuclei, dev)
    if float(w.n_ao) ** 4 > _MOST_ELEMENTS:
        return None
    J, K = _jk(w.basis, torch.tensor(w.D, device=dev), kind == "fock")
    return J if kind == "coulomb" else (J, K, J - 0.5 * K)


def _tuv(L: int):
    return [(t, u, v) for n in range(L + 1) for t in range(n, -1, -1) for u in range(n - t, -1, -1)
            for v in (n - t - u,)]


def _cart(l: int):
    return [(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]


def _boys(L: int, T):
    """F_0..F_L(T): a convergent series at the top order and downward
    recursion below T = 35, F_0's error function and upward above."""
    lo = T.clamp(max=35.0)
    term = torch.full_like(T, 1.0 / (2 * L + 1))
    s = term.clone()
    for i in range(1, 140):
        term = term * (2.0 * lo) / (2 * L + 2 * i + 1)
        s += term
    e = torch.exp(-T)
    elo = torch.exp(-lo)
    F = [None] * (L + 1)
    F[L] = s * elo
    for m in range(L - 1, -1, -1):
        F[m] = (2.0 * lo * F[m + 1] + elo) / (2 * m + 1)
    hi = T.clamp(min=35.0)
    far = 0.5 * torch.sqrt(math.pi / hi) * torch.erf(torch.sqrt(hi))
    big = T > 35.0
    for m in range(L + 1):
        F[m] = torch.where(big, far, F[m])
        far = ((2 * m + 1) * far - e) / (2.0 * hi)
    return F


def _hermite_coulomb(L: int, alpha, d, pref):
    """pref R_tuv(alpha, d) for every t + u + v <= L, by McMurchie-Davidson."""
    F = _boys(L, alpha * (d[0] ** 2 + d[1] ** 2 + d[2] ** 2))
    scale = [pref]
    for _ in range(L):
        scale.append(scale[-1] * (-2.0 * alpha))
    cur = {(0, 0, 0): scale[L] * F[L]}
    for m in range(L - 1, -1, -1):
        new = {(0, 0, 0): scale[m] * F[m]}
        for tuv in _tuv(L - m)[1:]:
            ax = next(k for k in range(3) if tuv[k])
            one = tuple(x - (k == ax) for k, x in enumerate(tuv))
            r = d[ax] * cur[one]
            if tuv[ax] > 1:
                r = r + (tuv[ax] - 1) * cur[tuple(x - 2 * (k == ax) for k, x in enumerate(tuv))]
            new[tuv] = r
        cur = new
    return cur


def _e_table(la: int, lb: int, a, b, X):
    """E_t^{ij} of one axis for exponents a, b and separation X = A - B."""
    p = a + b
    E = {(0, 0, 0): torch.exp(-a * b / p * X * X)}
    pa, pb = -b / p * X, a / p * X

    def get(i, j, t):
        return E.get((i, j, t), 0.0)

    for i, j in itertools.product(range(la + 1), range(lb + 1)):
        if i == j == 0:
            continue
        i0, j0, sh = (i - 1, j, pa) if i else (i, j - 1, pb)
        for t in range(i + j + 1):
            E[i, j, t] = sh * get(i0, j0, t) + get(i0, j0, t - 1) / (2 * p) + (t + 1) * get(i0, j0, t + 1)
    return E


class _Group:
    """The shells of one l and one contraction degree."""

    def __init__(self, basis, l: int, deg: int, dev):
        idx = [s for s, sh in enumerate(basis.shells) if sh.l == l and sh.n_prim == deg]
        sh = [basis.shells[s] for s in idx]
        self.l, self.n, self.deg = l, len(idx), deg
        self.at = torch.tensor([s.centre for s in sh], dtype=torch.float64, device=dev)
        self.ex = torch.tensor([s.exponents for s in sh], dtype=torch.float64, device=dev)
        self.co = torch.tensor([s.coefficients for s in sh], dtype=torch.float64, device=dev)
        self.nc = len(_cart(l))
        off = torch.tensor([basis.offsets[s] for s in idx], device=dev)
        self.ao = (off[:, None] + torch.arange(self.nc, device=dev)[None, :]).reshape(-1)


def _groups(basis, dev):
    keys = sorted({(s.l, s.n_prim) for s in basis.shells})
    return [_Group(basis, l, d, dev) for l, d in keys]


class _Pairs:
    """Every shell pair of two groups: Hermite expansions per primitive pair.
    E: (n_a n_b, deg_a deg_b, nc_a nc_b, n_tuv); p, P per (pair, primitive)."""

    def __init__(self, A: _Group, B: _Group):
        self.A, self.B, self.L = A, B, A.l + B.l
        sh = (A.n, B.n, A.deg, B.deg)
        a = A.ex[:, None, :, None].expand(sh)
        b = B.ex[None, :, None, :].expand(sh)
        cc = (A.co[:, None, :, None] * B.co[None, :, None, :]).expand(sh)
        self.p = a + b
        Ra, Rb = A.at[:, None, None, None, :], B.at[None, :, None, None, :]
        self.P = (a[..., None] * Ra + b[..., None] * Rb) / self.p[..., None]
        ax = [_e_table(A.l, B.l, a, b, (Ra - Rb)[..., k].expand(sh)) for k in range(3)]
        tuv = _tuv(self.L)
        E = torch.zeros(sh + (A.nc * B.nc, len(tuv)), dtype=torch.float64, device=a.device)
        for f, (i, j) in enumerate(itertools.product(_cart(A.l), _cart(B.l))):
            for h, (t, u, v) in enumerate(tuv):
                if t <= i[0] + j[0] and u <= i[1] + j[1] and v <= i[2] + j[2]:
                    E[..., f, h] = cc * ax[0][i[0], j[0], t] * ax[1][i[1], j[1], u] * ax[2][i[2], j[2], v]
        n, k = A.n * B.n, A.deg * B.deg
        self.n, self.k, self.tuv = n, k, tuv
        self.E = E.reshape(n, k, A.nc * B.nc, len(tuv))
        self.p, self.P = self.p.reshape(n * k), self.P.reshape(n * k, 3)


def _eri_rows(X: _Pairs, a0: int, a1: int, Y: _Pairs):
    """(ab|cd) for a in [a0, a1) of X's first group: (a, na, b, nb, c, nc, d, nd)."""
    r0, r1 = a0 * X.B.n, a1 * X.B.n
    p, P = X.p[r0 * X.k:r1 * X.k, None], X.P[r0 * X.k:r1 * X.k, None]
    q, Q = Y.p[None, :], Y.P[None, :]
    pref = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
    d = [(P - Q)[..., k] for k in range(3)]
    R = _hermite_coulomb(X.L + Y.L, p * q / (p + q), d, pref)
    n, hx, hy = r1 - r0, len(X.tuv), len(Y.tuv)
    Ex = X.E[r0:r1]
    V = None
    for h, t in enumerate(X.tuv):
        M = torch.stack([R[t[0] + u[0], t[1] + u[1], t[2] + u[2]] * (-1.0) ** sum(u) for u in Y.tuv], -1)
        M = M.view(n * X.k, Y.n, Y.k * hy).transpose(0, 1)                  # (cd, ab prim, cd prim tuv)
        W = torch.bmm(M, Y.E.permute(0, 1, 3, 2).reshape(Y.n, Y.k * hy, -1))  # (cd, ab prim, ncd)
        W = W.transpose(0, 1).reshape(n, X.k, Y.n * W.shape[-1])
        W = torch.bmm(Ex[..., h].transpose(1, 2), W)                        # (ab, nab, cd ncd)
        V = W if V is None else V + W
    A, B, C, D = X.A, X.B, Y.A, Y.B
    V = V.view(a1 - a0, B.n, A.nc, B.nc, C.n, D.n, C.nc, D.nc).permute(0, 2, 1, 3, 4, 6, 5, 7)
    return V.reshape((a1 - a0) * A.nc, B.n * B.nc, C.n * C.nc, D.n * D.nc)


def _jk(basis, Dm, with_k: bool):
    dev = Dm.device
    g = _groups(basis, dev)
    pairs = [_Pairs(g[i], g[j]) for i in range(len(g)) for j in range(i, len(g))]
    J, K = torch.zeros_like(Dm), torch.zeros_like(Dm)
    for X in pairs:
        for Y in pairs:
            A, B, C, D = X.A.ao, X.B.ao, Y.A.ao, Y.B.ao
            row = X.B.n * (X.k * Y.n * Y.k * 2 * len(_tuv(X.L + Y.L)) + 3 * X.A.nc * X.B.nc * len(C) * len(D)
                           + 4 * X.k * Y.n * (Y.k * len(Y.tuv) + Y.A.nc * Y.B.nc))
            step = max(1, int(2.5e9 / row))
            for a0 in range(0, X.A.n, step):
                a1 = min(X.A.n, a0 + step)
                V = _eri_rows(X, a0, a1, Y)
                a = A[a0 * X.A.nc:a1 * X.A.nc]
                Jab = torch.einsum("abcd,cd->ab", V, Dm[C][:, D]) * (1.0 if Y.A is Y.B else 2.0)
                J[a[:, None], B[None, :]] += Jab
                if X.A is not X.B:
                    J[B[:, None], a[None, :]] += Jab.T
                if not with_k:
                    continue

                def add(sub, rows, cols, dr, dc):
                    K[rows[:, None], cols[None, :]] += torch.einsum(sub, V, Dm[dr][:, dc])

                add("abcd,bd->ac", a, C, B, D)
                if Y.A is not Y.B:
                    add("abcd,bc->ad", a, D, B, C)
                if X.A is not X.B:
                    add("abcd,ad->bc", B, C, a, D)
                    if Y.A is not Y.B:
                        add("abcd,ac->bd", B, D, a, C)
    return J, K


def _one_electron(basis, nuclei, dev):
    n = basis.n_ao
    S, T, V = (torch.zeros(n, n, dtype=torch.float64, device=dev) for _ in range(3))
    Z = torch.tensor([z for z, _ in nuclei], dtype=torch.float64, device=dev)
    C = torch.tensor([c for _, c in nuclei], dtype=torch.float64, device=dev)
    g = _groups(basis, dev)
    for i, j in itertools.combinations_with_replacement(range(len(g)), 2):
        A, B = g[i], g[j]
        sh = (A.n, B.n, A.deg, B.deg)
        a, b = A.ex[:, None, :, None].expand(sh), B.ex[None, :, None, :].expand(sh)
        cc = A.co[:, None, :, None] * B.co[None, :, None, :] * (math.pi / (a + b)) ** 1.5
        X = (A.at[:, None, None, None, :] - B.at[None, :, None, None, :])
        ax = [_e_table(A.l, B.l + 2, a, b, X[..., k].expand(sh)) for k in range(3)]
        zero = torch.zeros(sh, dtype=torch.float64, device=dev)

        def s(k, m, l):
            return ax[k][m, l, 0] if l >= 0 else zero

        def kin(k, m, l):
            return -2.0 * b * b * s(k, m, l + 2) + b * (2 * l + 1) * s(k, m, l) - 0.5 * l * (l - 1) * s(k, m, l - 2)

        P = _Pairs(A, B)
        for c, z in zip(C.split(16), Z.split(16)):
            d = [P.P[:, None, k] - c[None, :, k] for k in range(3)]
            pref = -(2.0 * math.pi / P.p)[:, None] * z[None, :]
            R = _hermite_coulomb(P.L, P.p[:, None].expand(d[0].shape), d, pref)
            Rh = torch.stack([R[t].sum(1) for t in P.tuv], -1).view(P.n, P.k, len(P.tuv))
            v = torch.einsum("nkfh,nkh->nf", P.E, Rh).view(A.n, B.n, A.nc, B.nc)
            V[A.ao[:, None], B.ao[None, :]] += v.permute(0, 2, 1, 3).reshape(A.n * A.nc, B.n * B.nc)
        for M, parts in ((S, "sss"), (T, "kss sks ssk")):
            blk = torch.zeros(A.n, A.nc, B.n, B.nc, dtype=torch.float64, device=dev)
            for f, m in enumerate(_cart(A.l)):
                for h, l in enumerate(_cart(B.l)):
                    tot = 0.0
                    for p in parts.split():
                        x = [(kin if p[k] == "k" else s)(k, m[k], l[k]) for k in range(3)]
                        tot = tot + (cc * x[0] * x[1] * x[2]).sum((2, 3))
                    blk[:, f, :, h] = tot
            M[A.ao[:, None], B.ao[None, :]] = blk.reshape(A.n * A.nc, B.n * B.nc)
        if i != j:
            for M in (S, T, V):
                M[B.ao[:, None], A.ao[None, :]] = M[A.ao[:, None], B.ao[None, :]].T
    return S, T, V, T + V
