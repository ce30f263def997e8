"""Performance cases: what a user of this framework has it do, through its public entry points.

A case is a dict with a ``kind`` (one entry point), a system size and the options of the
call; ``listed()`` names twelve, ``draw(rng)`` gives more of the same ranges.  Systems are
the repository's seeded water clusters in its own basis sets, the smallest call being one
water in a minimal basis and the largest (H2O)16 / 6-31G** (N = 400), the benchmark's
molecule.  ``exact`` restates every integral, Fock matrix, gradient and network step in
plain torch / numpy float64 (sizes it can do in seconds), from textbook formulas:
Hermite expansions, the Boys function by its series, automatic differentiation for the
nuclear gradient.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mcmurchie-davidson_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from mmd import _native  # noqa: E402
from mmd.batch import BatchRHF  # noqa: E402
from mmd.clusters import geometry_string, water_cluster_coords  # noqa: E402
from mmd.guess import B631G, B631GSS, DensityMLP  # noqa: E402
from mmd.integrals.fock import formPT  # noqa: E402
from mmd.integrals.shells import shells_from_bfs  # noqa: E402
from mmd.integrals.twoe import clear_context_cache  # noqa: E402
from mmd.molecule import BASIS_DIR, Molecule, get_basis  # noqa: E402

ANGSTROM = 0.52917721092
TOL = 1e-12  # the SCF's default Schwarz x density threshold (acc2e)
# functions per water molecule
NWATER = {"sto-3g": 7, "3-21g": 13, "dz": 14, "6-31g": 13, "6-31gs": 19, "6-31gss": 25, "6-31ppgss": 31}
NHID, NIN = 256, 53


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference user's smallest call: formPT on host arrays, one water, minimal basis
        {"name": "formpt_water_sto3g", "kind": "formpt", "n": 1, "basis": "sto-3g", "density": "full"},
        # an SCF iteration's Fock build of an ordinary molecule, density on the device
        {"name": "fock_h2o4_631gss", "kind": "fock", "n": 4, "basis": "6-31gss", "density": "full", "fp32_below": 0.0},
        # the same for the benchmark's molecule: the largest
        {"name": "fock_h2o16_631gss", "kind": "fock", "n": 16, "basis": "6-31gss", "density": "full",
         "fp32_below": 0.0},
        # a late SCF iteration's increment of the density, mixed precision
        {"name": "fock_h2o16_mixed_inc", "kind": "fock", "n": 16, "basis": "6-31gss", "density": "increment",
         "fp32_below": 1e-5},
        # one batched build of many clusters of 1..8 waters (training-data generation)
        {"name": "fock_batch48_631g", "kind": "batch", "count": 48, "basis": "6-31g", "fp32_below": 0.0},
        # a new geometry: basis, shell pairs, one-electron integrals, Schwarz table
        {"name": "setup_h2o8_631gss", "kind": "setup", "n": 8, "basis": "6-31gss"},
        # the whole ERI tensor of a conventional SCF, N = 75
        {"name": "eri_h2o3_631gss", "kind": "eri", "n": 3, "basis": "6-31gss"},
        # Coulomb and exchange matrices from a stored tensor (conventional SCF, real-time TDHF)
        {"name": "jk_n100", "kind": "jk", "N": 100},
        # analytic nuclear forces of a converged molecule
        {"name": "forces_h2o2_631gss", "kind": "forces", "n": 2, "basis": "6-31gss"},
        # AO -> MO transform of the ERI tensor (MP2, CIS, TDHF)
        {"name": "ao2mo_n76", "kind": "ao2mo", "N": 76},
        # one training step of the guess network at its training batch
        {"name": "mlp_train_8192", "kind": "mlp", "rows": 8192, "basis": "6-31gss", "train": True},
        # a whole direct RHF
        {"name": "rhf_h2o3_631g", "kind": "rhf", "n": 3, "basis": "6-31g"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(["formpt", "fock", "fock", "fock", "batch", "setup", "eri", "jk", "forces", "ao2mo", "mlp",
                       "rhf"])
    basis = rng.choice(["sto-3g", "3-21g", "dz", "6-31g", "6-31gs", "6-31gss", "6-31gss", "6-31ppgss"])
    per = NWATER[basis]
    if kind == "formpt":
        return {"kind": kind, "n": _log_int(rng, 1, 4), "basis": basis, "density": rng.choice(["full", "increment"])}
    if kind == "fock":
        return {"kind": kind, "n": _log_int(rng, 1, max(1, 360 // per)) if per < 31 else _log_int(rng, 1, 10),
                "basis": basis, "density": rng.choice(["full", "increment"]),
                "fp32_below": rng.choice([0.0, 0.0, 1e-5, 1e-3])}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 2, 48), "basis": rng.choice(["sto-3g", "6-31g"]),
                "fp32_below": rng.choice([0.0, 1e-5])}
    if kind == "setup":
        return {"kind": kind, "n": _log_int(rng, 1, 10), "basis": basis}
    if kind == "eri":
        return {"kind": kind, "n": _log_int(rng, 1, max(1, 75 // per)), "basis": basis}
    if kind in ("jk", "ao2mo"):
        return {"kind": kind, "N": _log_int(rng, 7, 110 if kind == "jk" else 76)}
    if kind == "forces":
        return {"kind": kind, "n": _log_int(rng, 1, max(1, 50 // per)), "basis": basis}
    if kind == "mlp":
        return {"kind": kind, "rows": _log_int(rng, 33, 8192), "basis": rng.choice(["6-31g", "6-31gss"]),
                "train": rng.random() < 0.6}
    return {"kind": "rhf", "n": _log_int(rng, 1, max(1, 39 // per)), "basis": basis}


# ------------------------------------------------------------------ inputs
def _rng(seed, tag):
    return np.random.default_rng([int(seed) & 0x7fffffff, tag])


def _system(n, seed):
    """Atomic numbers and coordinates (bohr) of the seeded cluster, and its geometry string."""
    sym, xyz = water_cluster_coords(n, int(seed))
    text = geometry_string(sym, xyz)
    rows = [ln.split() for ln in text.strip().split("\n")[1:]]
    xyz = np.array([[float(x) for x in r[1:]] for r in rows]) / ANGSTROM
    return np.array([8 if s == "O" else 1 for s in sym]), xyz, text


def _function_atoms(basis, Z):
    data = get_basis(os.path.join(BASIS_DIR, basis + ".gbs"))
    ncomp = {"S": 1, "P": 3, "D": 6}
    return np.concatenate([np.full(sum(ncomp[m] for m, _ in data[int(z)]), a) for a, z in enumerate(Z)])


def _density(basis, Z, xyz, seed, kind, tag=1):
    """A symmetric density-like matrix: random elements that decay over the distance of
    the two centres as an insulator's density matrix does; an increment is 1e-3 of it."""
    at = _function_atoms(basis, Z)
    R = np.linalg.norm(xyz[:, None] - xyz[None, :], axis=-1)[np.ix_(at, at)]
    A = _rng(seed, tag).standard_normal(R.shape)
    return (1e-3 if kind == "increment" else 1.0) * 0.25 * (A + A.T) * np.exp(-R / 2.0)


def _batch_systems(case, seed):
    """(waters, geometry seed) of every cluster: the sizes belong to the case, the
    geometries to the seed."""
    sizes = _rng(case["count"], 6).integers(1, 9, case["count"])
    return [(int(n), int(s)) for n, s in zip(sizes, _rng(seed, 7).integers(1, 1 << 30, case["count"]))]


def _symmetric_tensor(N, seed):
    """A tensor with the eight-fold symmetry of the ERIs, T = sum_x B_pq^x B_rs^x, its
    factors decaying away from the diagonal like products of distant functions."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    x = torch.rand(N, generator=g, device="cuda", dtype=torch.float64) * N
    B = torch.randn((N, N, 2 * N), generator=g, device="cuda", dtype=torch.float64)
    B = (B + B.transpose(0, 1)) * torch.exp(-(x[:, None] - x[None, :]).abs() / 8.0)[:, :, None] / N
    B = B.reshape(N * N, -1)
    return (B @ B.T).view(N, N, N, N)


def _random_symmetric(N, seed):
    A = _rng(seed, 3).standard_normal((N, N))
    return torch.as_tensor(0.5 * (A + A.T), device="cuda")


def _mlp_inputs(case, seed):
    """Feature rows as the guess builds them (pair type one-hot, distance on Gaussians,
    bond directions, relative rotation), block targets with their masks, and weights."""
    gb = B631GSS if case["basis"] == "6-31gss" else B631G
    rng, B = _rng(seed, 5), case["rows"]
    X = np.zeros((B, NIN))
    X[np.arange(B), rng.integers(0, 6, B)] = 1.0
    d = rng.uniform(1.5, 8.0, B)
    X[:, 6:38] = np.exp(-((d[:, None] - np.linspace(0.5, 8.0, 32)) / 0.24) ** 2)
    u = rng.standard_normal((B, 2, 3))
    X[:, 38:44] = (u / np.linalg.norm(u, axis=2, keepdims=True)).reshape(B, 6)
    X[:, 44:53] = rng.uniform(-1, 1, (B, 9))
    nm = gb.nmax
    size = rng.choice([gb.nfunc[1], gb.nfunc[8]], (B, 2))
    k = np.arange(nm)
    M = ((k[None, :, None] < size[:, 0, None, None]) & (k[None, None, :] < size[:, 1, None, None])).reshape(B, -1)
    T = rng.standard_normal((B, gb.nout)) * 0.3 * M
    W = {}
    for i, (o, n) in enumerate([(NHID, NIN), (NHID, NHID), (gb.nout, NHID)]):
        W[f"W{i}"] = (rng.standard_normal((o, n)) / math.sqrt(n)).astype(np.float32)
        W[f"b{i}"] = (0.1 * rng.standard_normal(o)).astype(np.float32)
    return gb, X.astype(np.float32), T.astype(np.float32), M.astype(np.float32), W


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("formpt", "fock", "eri", "forces"):
        Z, xyz, text = _system(case["n"], seed)
        mol = Molecule(text, case["basis"])
        s = {"kind": kind, "mol": mol, "case": case}
        if kind == "formpt":
            s["P"] = _density(case["basis"], Z, xyz, seed, case["density"])
            s["P_old"] = np.zeros_like(s["P"])
            s["screen"] = mol.screen
        elif kind == "fock":
            P = _density(case["basis"], Z, xyz, seed, case["density"])
            s["dP"] = torch.as_tensor(P, device="cuda").reshape(-1)
            s["G"] = torch.empty_like(s["dP"])
            s["ctx"] = mol.context
        elif kind == "eri":
            s["ctx"] = mol.context
            s["out"] = torch.empty((mol.nbasis,) * 4, dtype=torch.float64, device="cuda")
        else:
            mol.P = _density(case["basis"], Z, xyz, seed, "full").astype(complex)
            mol.F = _density(case["basis"], Z, xyz, seed, "full", tag=2).astype(complex)
            mol.is_converged = True
            s["ctx"] = mol.context
        return s
    if kind == "batch":
        systems = _batch_systems(case, seed)
        b = BatchRHF([_system(n, k)[2] for n, k in systems], case["basis"], fp32_below=case["fp32_below"])
        dP = np.zeros((b.B, b.Nmax, b.Nmax))
        for m, (n, k) in enumerate(systems):
            Z, xyz, _ = _system(n, k)
            dP[m, :b.N[m], :b.N[m]] = _density(case["basis"], Z, xyz, k, "full")
        return {"kind": kind, "batch": b, "dP": torch.as_tensor(dP, device="cuda")}
    if kind in ("setup", "rhf"):
        return {"kind": kind, "geometry": _system(case["n"], seed)[2], "basis": case["basis"]}
    if kind == "jk":
        T = _symmetric_tensor(case["N"], seed)
        P = _random_symmetric(case["N"], seed)
        return {"kind": kind, "ctx": _native.scratch_context(), "T": T, "P": P, "J": torch.empty_like(P),
                "K": torch.empty_like(P)}
    if kind == "ao2mo":
        T = _symmetric_tensor(case["N"], seed).reshape(-1)
        C = torch.linalg.qr(_random_symmetric(case["N"], seed).cpu())[0].contiguous().cuda()
        return {"kind": kind, "T": T, "C": C, "out": torch.empty_like(T), "work": torch.empty_like(T)}
    gb, X, T, M, W = _mlp_inputs(case, seed)
    return {"kind": kind, "net": DensityMLP(weights=W, gb=gb), "train": case["train"],
            "X": torch.as_tensor(X, device="cuda"), "T": torch.as_tensor(T, device="cuda"),
            "M": torch.as_tensor(M, device="cuda")}


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "formpt":
        mol = state["mol"]
        return formPT(state["P"], state["P_old"], mol.bfs, mol.nbasis, state["screen"], TOL)
    if kind == "fock":
        return state["ctx"].fock(state["dP"], state["G"], tol=TOL, fp32_below=state["case"]["fp32_below"])
    if kind == "batch":
        return state["batch"].fock(state["dP"])
    if kind == "setup":
        clear_context_cache()  # a geometry not seen before
        mol = Molecule(state["geometry"], state["basis"])
        mol.build(direct=True)
        return {"S": mol.S, "T": mol.T, "V": mol.V, "M": mol.M, "X": mol.X, "screen": mol.context.screen()}
    if kind == "eri":
        return state["ctx"].eri_tensor(state["out"])
    if kind == "jk":
        return state["ctx"].jk_dense(state["T"], state["P"], state["J"], state["K"])
    if kind == "forces":
        return state["mol"].forces()
    if kind == "ao2mo":
        return _native.ao2mo(state["C"], state["T"], state["out"], state["work"])
    if kind == "mlp":
        net = state["net"]
        if not state["train"]:
            return net.predict(state["X"])
        acts = net.forward(state["X"])
        loss, dY = net.loss_grad(acts[-1][2], state["T"], state["M"])
        grads = net.backward(acts, dY)
        net.adam(grads, lr=2e-3)
        return {"loss": loss, "grads": grads, "W": net.W, "b": net.b}
    mol = Molecule(state["geometry"], state["basis"])
    energy = mol.RHF(doPrint=False, direct=True, conver=1e-9)
    return {"energy": float(energy), "P": mol.P, "F": mol.F, "MO": mol.MO}


# ------------------------------------------------------------------ work
def _significant(basis, n, seed=0):
    """Primitive pairs (p, weight) of the cluster whose Gaussian product is not negligible,
    and the shell pairs' function counts: a model of what the screening leaves."""
    Z, xyz, _ = _system(n, seed)
    sh = _shells(basis, Z, xyz)
    nf = np.array([(s["L"] + 1) * (s["L"] + 2) // 2 for s in sh])
    amin = np.array([s["exps"].min() for s in sh])
    cen = np.array([s["center"] for s in sh])
    R2 = ((cen[:, None] - cen[None]) ** 2).sum(-1)
    i, j = np.tril_indices(len(sh))
    ov = np.exp(-amin[i] * amin[j] / (amin[i] + amin[j]) * R2[i, j])
    prim = np.zeros(len(i))
    for x, (a, b) in enumerate(zip(i, j)):
        ea, eb = sh[a]["exps"], sh[b]["exps"]
        mu = ea[:, None] * eb[None] / (ea[:, None] + eb[None])
        prim[x] = (mu * R2[a, b] < 40.0).sum()
    keep = (ov > 1e-10) & (prim > 0)
    return ov[keep], prim[keep], (nf[i] * nf[j])[keep]


def _quartet_work(basis, n, scale=1.0):
    """FLOPs of the surviving quartets: 40 per primitive quartet (distance, Boys, recursion)
    and 12 per function quartet (scatter), of the pairs whose overlap product passes."""
    ov, prim, fun = _significant(basis, n)
    o = np.argsort(-ov)
    ov, prim, fun = ov[o], prim[o], fun[o]
    cp, cf = np.concatenate([[0], np.cumsum(prim)]), np.concatenate([[0], np.cumsum(fun)])
    last = np.searchsorted(-ov, -(TOL / scale) / ov, side="right")
    return float((40.0 * prim * cp[last] + 12.0 * fun * cf[last]).sum() / 2)


def work(case):
    kind = case["kind"]
    if kind in ("formpt", "fock"):
        N = NWATER[case["basis"]] * case["n"]
        scale = 1e-3 if case["density"] == "increment" else 1.0
        return {"bytes": 16.0 * N * N, "flops": _quartet_work(case["basis"], case["n"], scale)}
    if kind == "batch":
        sizes = [n for n, _ in _batch_systems(case, 0)]
        per = {n: _quartet_work(case["basis"], n) for n in set(sizes)}
        N = NWATER[case["basis"]]
        return {"bytes": sum(16.0 * (N * n) ** 2 for n in sizes), "flops": sum(per[n] for n in sizes)}
    if kind == "setup":
        N = NWATER[case["basis"]] * case["n"]
        _, prim, _ = _significant(case["basis"], case["n"])
        return {"bytes": 8.0 * N * N * 7, "flops": float(prim.sum()) * (100.0 + 60.0 * 3 * case["n"])}
    if kind in ("eri", "forces"):
        N = NWATER[case["basis"]] * case["n"]
        ov, prim, fun = _significant(case["basis"], case["n"])
        full = 40.0 * prim.sum() ** 2 / 2 + 6.0 * fun.sum() ** 2 / 2
        return {"bytes": 8.0 * N ** 4 if kind == "eri" else 16.0 * N * N, "flops": full * (1 if kind == "eri" else 6)}
    if kind == "jk":
        N = case["N"]
        return {"bytes": 8.0 * (N ** 4 + 3 * N * N), "flops": 4.0 * N ** 4}
    if kind == "ao2mo":
        N = case["N"]
        return {"bytes": 16.0 * N ** 4, "flops": 8.0 * N ** 5}
    if kind == "mlp":
        nout = 225 if case["basis"] == "6-31gss" else 81
        par = NIN * NHID + NHID * NHID + NHID * nout
        B = case["rows"]
        rows = NIN + (2 * nout if case["train"] else nout)
        return {"bytes": 4.0 * B * rows + (22.0 if case["train"] else 2.0) * par,
                "flops": 2.0 * B * (par * (3 if case["train"] else 1) - (NIN * NHID if case["train"] else 0))}
    N = NWATER[case["basis"]] * case["n"]
    return {"bytes": 16.0 * N * N, "flops": 12.0 * _quartet_work(case["basis"], case["n"], 1e-2)}


# ------------------------------------------------------------------ 64-bit restatement
def _comps(L):
    return [(x, y, L - x - y) for x in range(L, -1, -1) for y in range(L - x, -1, -1)]


def _fact2(k):
    return math.prod(range(k, 0, -2)) if k > 0 else 1


def _shells(basis, Z, xyz):
    """Contracted shells: exponents and weights normalised for the (L, 0, 0) component's
    radial part, without the component factor 1/sqrt((2l-1)!!(2m-1)!!(2n-1)!!)."""
    data = get_basis(os.path.join(BASIS_DIR, basis + ".gbs"))
    out, f = [], 0
    for a, z in enumerate(Z):
        for label, prims in data[int(z)]:
            L = "SPD".index(label)
            e, c = np.array([p[0] for p in prims]), np.array([p[1] for p in prims])
            w = c * np.sqrt(2.0 ** (2 * L + 1.5) * e ** (L + 1.5) / math.pi ** 1.5)
            n2 = math.pi ** 1.5 / 2.0 ** L * (w[:, None] * w / (e[:, None] + e) ** (L + 1.5)).sum()
            out.append({"L": L, "atom": a, "center": xyz[a], "exps": e, "w": w / math.sqrt(n2), "f": f})
            f += (L + 1) * (L + 2) // 2
    return out


class _BoysStack(torch.autograd.Function):
    """F_0..F_M (last dimension) of T; dF_m/dT = -F_{m+1}."""

    @staticmethod
    def forward(ctx, T, M):
        F = _boys(T, M + 1)
        ctx.save_for_backward(F)
        return F[..., :-1]

    @staticmethod
    def backward(ctx, g):
        (F,) = ctx.saved_tensors
        return -(g * F[..., 1:]).sum(-1), None


def _boys(T, M):
    """F_m(T) = int_0^1 t^2m exp(-T t^2) dt, m = 0..M: Kummer's series at M and downward
    recursion below 36, erf and upward recursion above."""
    lo = T < 36.0
    t = torch.where(lo, T, torch.ones_like(T))
    e = torch.exp(-t)
    term = torch.full_like(t, 1.0 / (2 * M + 1))
    s = term.clone()
    for i in range(1, 150):
        term = term * (2.0 * t) / (2 * M + 2 * i + 1)
        s = s + term
    low = [e * s]
    for m in range(M, 0, -1):
        low.append((2.0 * t * low[-1] + e) / (2 * m - 1))
    low = torch.stack(low[::-1], -1)
    u = torch.where(lo, torch.full_like(T, 40.0), T)
    eu = torch.exp(-u)
    up = [0.5 * torch.sqrt(math.pi / u) * torch.erf(torch.sqrt(u))]
    for m in range(M):
        up.append(((2 * m + 1) * up[-1] - eu) / (2.0 * u))
    return torch.where(lo[..., None], low, torch.stack(up, -1))


def _herm(L):
    return [(t, u, n - t - u) for n in range(L + 1) for t in range(n, -1, -1) for u in range(n - t, -1, -1)]


def _r_table(L, alpha, D):
    """R_tuv (last dimension, the order of _herm) for exponent alpha and distances D[..., 3]."""
    F = _BoysStack.apply(alpha * (D * D).sum(-1), L)
    R = {}
    for n in range(L, -1, -1):
        R[(n, 0, 0, 0)] = (-2.0 * alpha) ** n * F[..., n]
        for t, u, v in _herm(L - n)[1:]:
            k = 0 if t else (1 if u else 2)
            h = [t, u, v]
            h[k] -= 1
            val = D[..., k] * R[(n + 1, *h)]
            if h[k] > 0:
                c = h[k]
                h[k] -= 1
                val = val + c * R[(n + 1, *h)]
            R[(n, t, u, v)] = val
    return torch.stack([R[(0, *h)] for h in _herm(L)], -1)


def _e_1d(la, lb, p, XPA, XPB):
    """One-dimensional Hermite coefficients E[i][j][t], without the Gaussian factor."""
    one, i2p = torch.ones_like(p), 0.5 / p
    E = {(0, 0): [one]}

    def up(row, X):
        out = []
        for t in range(len(row) + 1):
            v = 0.0
            if t > 0:
                v = v + i2p * row[t - 1]
            if t < len(row):
                v = v + X * row[t]
            if t + 1 < len(row):
                v = v + (t + 1) * row[t + 1]
            out.append(v)
        return out

    for i in range(la + 1):
        if i:
            E[(i, 0)] = up(E[(i - 1, 0)], XPA)
        for j in range(1, lb + 1):
            E[(i, j)] = up(E[(i, j - 1)], XPB)
    return E


class _Pairs:
    """Shell pairs of one (la, lb) class: primitive products and their Hermite expansions
    lam[primitive pair, component pair, tuv] over the Gaussian factor, weights included."""

    def __init__(self, sh, cls, xyz):
        self.la, self.lb = la, lb = cls
        self.pairs = [(a, b) for a in range(len(sh)) for b in range(len(sh))
                      if (sh[a]["L"], sh[b]["L"]) == cls and (la != lb or a >= b)]
        rows = [(x, sh[a]["atom"], sh[b]["atom"], ea, eb, wa * wb) for x, (a, b) in enumerate(self.pairs)
                for ea, wa in zip(sh[a]["exps"], sh[a]["w"]) for eb, wb in zip(sh[b]["exps"], sh[b]["w"])]
        if not rows:
            return
        r = torch.tensor(rows, dtype=torch.float64, device="cuda")
        self.index = r[:, 0].long()
        A, B = xyz[r[:, 1].long()], xyz[r[:, 2].long()]
        self.ea, self.eb = ea, eb = r[:, 3], r[:, 4]
        self.p = p = ea + eb
        self.P = (ea[:, None] * A + eb[:, None] * B) / p[:, None]
        self.K = r[:, 5] * torch.exp(-ea * eb / p * ((A - B) ** 2).sum(-1))
        self.E = [_e_1d(la, lb + 2, p, self.P[:, d] - A[:, d], self.P[:, d] - B[:, d]) for d in range(3)]
        self.ca, self.cb = _comps(la), _comps(lb)
        cols = []
        for a in self.ca:
            for b in self.cb:
                nab = 1.0 / math.sqrt(math.prod(_fact2(2 * x - 1) for x in a + b))
                ex = [self.E[d][(a[d], b[d])] for d in range(3)]
                zero = torch.zeros_like(p)
                cols.append(torch.stack([nab * ex[0][t] * ex[1][u] * ex[2][v]
                                         if t < len(ex[0]) and u < len(ex[1]) and v < len(ex[2]) else zero
                                         for t, u, v in _herm(la + lb)], -1))
        self.lam = torch.stack(cols, 1)
        fa = torch.tensor([[sh[a]["f"] + i for i in range(len(self.ca)) for _ in self.cb] for a, _ in self.pairs],
                          device="cuda")
        fb = torch.tensor([[sh[b]["f"] + j for _ in self.ca for j in range(len(self.cb))] for _, b in self.pairs],
                          device="cuda")
        self.fi, self.fj = fa, fb  # function indices [pair, component pair]
        i, j = torch.maximum(fa, fb), torch.minimum(fa, fb)
        self.tri = i * (i + 1) // 2 + j


def _pair_classes(sh, xyz):
    top = max(s["L"] for s in sh)
    out = [_Pairs(sh, (la, lb), xyz) for la in range(top + 1) for lb in range(la + 1)]
    return [p for p in out if p.pairs]


def _eri_block(b, k):
    """(bra pair, ab, ket pair, cd) contracted ERIs of two pair classes, yielded in pieces
    of bra primitive pairs to be added up: (bra pair index, values)."""
    Lb, Lk = b.la + b.lb, k.la + k.lb
    hb, hk, slot = _herm(Lb), _herm(Lk), {h: x for x, h in enumerate(_herm(Lb + Lk))}
    comb = torch.tensor([[slot[tuple(x + y for x, y in zip(g, h))] for h in hk] for g in hb], device="cuda")
    sign = torch.tensor([(-1.0) ** sum(h) for h in hk], dtype=torch.float64, device="cuda")
    lam_k = k.lam * sign
    step = max(1, int(6e7 // (len(k.p) * max(len(slot) * (Lb + Lk + 1), len(hb) * max(len(hk), lam_k.shape[1])))))
    for s in range(0, len(b.p), step):
        e = slice(s, s + step)
        p, q = b.p[e, None], k.p[None]
        R = _r_table(Lb + Lk, p * q / (p + q), b.P[e, None] - k.P[None])
        pref = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q)) * b.K[e, None] * k.K[None]
        W = torch.einsum("bktu,kcu->bktc", (R * pref[..., None])[..., comb], lam_k)
        W = torch.zeros((W.shape[0], len(k.pairs)) + W.shape[2:], dtype=W.dtype, device="cuda").index_add(
            1, k.index, W)
        yield b.index[e], torch.einsum("bat,bktc->bakc", b.lam[e], W)


def _eri_matrix(sh, xyz, N):
    """Symmetric matrix of (ij|kl) over the function pairs i >= j, k >= l."""
    n2 = N * (N + 1) // 2
    V = torch.zeros((n2, n2), dtype=torch.float64, device="cuda")
    cl = _pair_classes(sh, xyz)
    for x, b in enumerate(cl):
        for k in cl[:x + 1]:
            blk = torch.zeros((len(b.pairs), b.lam.shape[1], len(k.pairs), k.lam.shape[1]), dtype=torch.float64,
                              device="cuda")
            for idx, piece in _eri_block(b, k):
                blk.index_add_(0, idx, piece)
            r, c = b.tri.reshape(-1), k.tri.reshape(-1)
            blk = blk.reshape(len(r), len(c))
            V[r[:, None], c[None]] = blk
            V[c[:, None], r[None]] = blk.T
    return V


def _pairs_of(N):
    i, j = np.tril_indices(N)
    return torch.as_tensor(i, device="cuda"), torch.as_tensor(j, device="cuda")


def _exact_fock(V, dP):
    """G(dP) with the Schwarz x density test, degeneracies and six updates per unique
    function quartet of the reference's direct Fock build."""
    N = dP.shape[0]
    I, J = _pairs_of(N)
    sq = torch.sqrt(torch.diagonal(V))
    G = torch.zeros(N * N, dtype=torch.float64, device="cuda")
    D, dpair = dP.reshape(-1), dP[I, J]
    for s in range(0, len(I), 1024):
        i, j, r = I[s:s + 1024, None], J[s:s + 1024, None], torch.arange(s, min(s + 1024, len(I)), device="cuda")
        q = torch.arange(int(r[-1]) + 1, device="cuda")
        k, l = I[None, :len(q)], J[None, :len(q)]
        dik, djl, dil, djk = D[i * N + k], D[j * N + l], D[i * N + l], D[j * N + k]
        dij, dkl = dpair[r, None], dpair[None, :len(q)]
        dm = torch.maximum(4.0 * torch.maximum(dij.abs(), dkl.abs()), torch.maximum(
            torch.maximum(dik.abs(), dil.abs()), torch.maximum(djk.abs(), djl.abs())))
        keep = (q[None] <= r[:, None]) & (sq[r, None] * sq[None, :len(q)] * dm >= TOL)
        v = torch.where(keep, V[r, :len(q)] * (1.0 + (i != j)) * (1.0 + (k != l)) * (1.0 + (q[None] != r[:, None])), 0)
        full = v.shape
        for pos, val in ((i * N + j, dkl * v), (k * N + l, dij * v), (i * N + k, -0.25 * djl * v),
                         (j * N + l, -0.25 * dik * v), (i * N + l, -0.25 * djk * v), (k * N + j, -0.25 * dil * v)):
            G.index_add_(0, pos.expand(full).reshape(-1), val.reshape(-1))
    return G.view(N, N)


def _one_electron(sh, xyz, Z, N, origin):
    """S, T, V and the dipole integrals about origin (differentiable in xyz)."""
    zero = lambda: torch.zeros((N, N), dtype=torch.float64, device="cuda")  # noqa: E731
    S, T, V, M = zero(), zero(), zero(), [zero(), zero(), zero()]
    Zt = torch.as_tensor(np.asarray(Z, dtype=float), device="cuda")
    for b in _pair_classes(sh, xyz):
        s3 = (math.pi / b.p) ** 1.5 * b.K
        h = _r_table(b.la + b.lb, b.p[:, None].expand(-1, len(Z)), b.P[:, None] - xyz[None])
        att = -(2.0 * math.pi / b.p * b.K)[:, None] * torch.einsum("pat,pct,c->pa", b.lam, h, Zt)
        cs, ct, cm = [], [], [[], [], []]
        for a in b.ca:
            for c in b.cb:
                nab = 1.0 / math.sqrt(math.prod(_fact2(2 * x - 1) for x in a + c))
                s, k, m = [], [], []
                for d in range(3):
                    E, la, lb = b.E[d], a[d], c[d]
                    e0 = E[(la, lb)]
                    s.append(e0[0])
                    kin = b.eb * (2 * lb + 1) * e0[0] - 2.0 * b.eb ** 2 * E[(la, lb + 2)][0]
                    if lb >= 2:
                        kin = kin - 0.5 * lb * (lb - 1) * E[(la, lb - 2)][0]
                    k.append(kin)
                    m.append((e0[1] if len(e0) > 1 else 0.0) + (b.P[:, d] - origin[d]) * e0[0])
                cs.append(nab * s3 * s[0] * s[1] * s[2])
                ct.append(nab * s3 * (k[0] * s[1] * s[2] + s[0] * k[1] * s[2] + s[0] * s[1] * k[2]))
                for d in range(3):
                    w = list(s)
                    w[d] = m[d]
                    cm[d].append(nab * s3 * w[0] * w[1] * w[2])
        shape = (len(b.pairs), len(cs))
        add = lambda x: torch.zeros(shape, dtype=torch.float64, device="cuda").index_add(0, b.index, x)  # noqa: E731
        r, c = b.fi.reshape(-1), b.fj.reshape(-1)
        put = lambda X, x: X.index_put((r, c), x.reshape(-1)).index_put((c, r), x.reshape(-1))  # noqa: E731
        S, T, V = put(S, add(torch.stack(cs, 1))), put(T, add(torch.stack(ct, 1))), put(V, add(att))
        M = [put(M[d], add(torch.stack(cm[d], 1))) for d in range(3)]
    return S, T, V, torch.stack(M)


def _diagonal_eris(sh, xyz, N):
    """(ij|ij) of every function pair: the Schwarz table."""
    out = torch.zeros(N * (N + 1) // 2, dtype=torch.float64, device="cuda")
    for b in _pair_classes(sh, xyz):
        hb, slot = _herm(b.la + b.lb), {h: x for x, h in enumerate(_herm(2 * (b.la + b.lb)))}
        comb = torch.tensor([[slot[tuple(x + y for x, y in zip(g, h))] for h in hb] for g in hb], device="cuda")
        sign = torch.tensor([(-1.0) ** sum(h) for h in hb], dtype=torch.float64, device="cuda")
        acc = torch.zeros((len(b.pairs), b.lam.shape[1]), dtype=torch.float64, device="cuda")
        # all primitive quartets (x, y) of each pair, by the pair's primitive count
        count = torch.bincount(b.index, minlength=len(b.pairs))
        start = torch.cumsum(count, 0) - count
        for K in sorted(set(count.tolist())):
            which = torch.nonzero(count == K)[:, 0]
            for w in which.split(max(1, int(2e7 // (K * K * len(slot))))):
                x = start[w][:, None, None] + torch.arange(K, device="cuda")[None, :, None] + torch.zeros(
                    K, dtype=torch.long, device="cuda")
                x, y = x.reshape(-1), x.transpose(1, 2).reshape(-1)
                p, q = b.p[x], b.p[y]
                R = _r_table(2 * (b.la + b.lb), p * q / (p + q), b.P[x] - b.P[y])
                R = R * (2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q)) * b.K[x] * b.K[y])[:, None]
                v = torch.einsum("xat,xtu,xau->xa", b.lam[x], R[:, comb], b.lam[y] * sign)
                acc.index_add_(0, b.index[x], v)
        out[b.tri.reshape(-1)] = acc.reshape(-1)
    return out


def _exact_forces(case, seed):
    Z, xyz0, _ = _system(case["n"], seed)
    xyz = torch.tensor(xyz0, device="cuda", requires_grad=True)
    sh = _shells(case["basis"], Z, xyz0)
    N = NWATER[case["basis"]] * case["n"]
    P = torch.as_tensor(_density(case["basis"], Z, xyz0, seed, "full"), device="cuda")
    W = P @ torch.as_tensor(_density(case["basis"], Z, xyz0, seed, "full", tag=2), device="cuda") @ P
    S, T, V, _ = _one_electron(sh, xyz, Z, N, [0.0, 0.0, 0.0])
    Zt = torch.as_tensor(Z.astype(float), device="cuda")
    i, j = np.triu_indices(len(Z), 1)
    nuc = (Zt[i] * Zt[j] / torch.linalg.norm(xyz[i] - xyz[j], dim=-1)).sum()
    (2.0 * (P * (T + V)).sum() - 2.0 * (W * S).sum() + nuc).backward()
    count = len(_pair_classes(sh, xyz.detach()))
    for x in range(count):
        for y in range(x + 1):
            cl = _pair_classes(sh, xyz)  # a graph for each block
            b, k = cl[x], cl[y]
            i, j = b.fi[:, :, None, None], b.fj[:, :, None, None]
            m, n = k.fi[None, None], k.fj[None, None]
            gam = 2.0 * P[i, j] * P[m, n] - 0.5 * (P[i, m] * P[j, n] + P[i, n] * P[j, m])
            # whole shells: (a, b) and (b, a) of two different shells, and bra-ket of two classes
            fb = torch.tensor([1.0 if p == q else 2.0 for p, q in b.pairs], dtype=torch.float64, device="cuda")
            fk = torch.tensor([1.0 if p == q else 2.0 for p, q in k.pairs], dtype=torch.float64, device="cuda")
            gam = gam * fb[:, None, None, None] * fk[None, None, :, None] * (1.0 if x == y else 2.0)
            e = sum((gam[idx] * piece).sum() for idx, piece in _eri_block(b, k))
            e.backward()
    return -xyz.grad


def _exact_mlp(case, seed):
    _, X, T, M, W = _mlp_inputs(case, seed)
    d = lambda a: torch.as_tensor(a, device="cuda").double()  # noqa: E731
    Wb = [torch.as_tensor(W[f"W{i}"], device="cuda").to(torch.bfloat16).double().requires_grad_() for i in range(3)]
    b = [d(W[f"b{i}"]).requires_grad_() for i in range(3)]
    h = d(X)
    for i in range(3):
        h = h @ Wb[i].T + b[i]
        if i < 2:
            h = torch.nn.functional.silu(h)
    if not case["train"]:
        return h.detach()
    loss = (((h - d(T)) * d(M)) ** 2).sum() / d(M).sum()
    loss.backward()
    step = lambda w, g: w - 2e-3 * g / (g.abs() + 1e-8)  # noqa: E731  (Adam's first step)
    return {"loss": loss.detach().reshape(1), "grads": [(w.grad, x.grad) for w, x in zip(Wb, b)],
            "W": [step(d(W[f"W{i}"]), Wb[i].grad) for i in range(3)],
            "b": [step(d(W[f"b{i}"]), b[i].grad) for i in range(3)]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        return _exact_mlp(case, seed)
    if kind == "jk":
        T, P = _symmetric_tensor(case["N"], seed), _random_symmetric(case["N"], seed)
        return [torch.einsum("pqrs,sr->pq", T, P), torch.einsum("psqr,sr->pq", T, P)]
    if kind == "ao2mo":
        N = case["N"]
        x = _symmetric_tensor(N, seed)
        C = torch.linalg.qr(_random_symmetric(N, seed).cpu())[0].cuda()
        for _ in range(4):  # contract the first index, append the new one last
            x = torch.tensordot(x, C, dims=([0], [0]))
        return x.reshape(-1)
    if kind == "rhf":
        return None
    if kind == "batch":
        if sum((n * NWATER[case["basis"]]) ** 4 for n, _ in _batch_systems(case, seed)) > 6e8:
            return None
        parts = []
        for n, k in _batch_systems(case, seed):
            Z, xyz, _ = _system(n, k)
            N = NWATER[case["basis"]] * n
            V = _eri_matrix(_shells(case["basis"], Z, xyz), torch.as_tensor(xyz, device="cuda"), N)
            parts.append(_exact_fock(V, torch.as_tensor(_density(case["basis"], Z, xyz, k, "full"),
                                                        device="cuda")).reshape(-1))
        return torch.cat(parts)
    Z, xyz, _ = _system(case["n"], seed)
    N = NWATER[case["basis"]] * case["n"]
    sh, x = _shells(case["basis"], Z, xyz), torch.as_tensor(xyz, device="cuda")
    if kind == "setup":
        origin = (Z[:, None] * xyz).sum(0) / Z.sum()
        S, T, V, M = _one_electron(sh, x, Z, N, origin)
        w, U = np.linalg.eigh(S.cpu().numpy())
        return {"S": S, "T": T, "V": V, "M": M, "X": (U / np.sqrt(w)) @ U.T,
                "screen": _diagonal_eris(sh, x, N)}
    if N > 100:
        return None
    if kind == "forces":
        return _exact_forces(case, seed)
    V = _eri_matrix(sh, x, N)
    if kind == "eri":
        i = torch.arange(N, device="cuda")
        tri = torch.maximum(i[:, None], i[None]) * (torch.maximum(i[:, None], i[None]) + 1) // 2 + torch.minimum(
            i[:, None], i[None])
        return V[tri.reshape(-1)][:, tri.reshape(-1)].view(N, N, N, N)
    G = _exact_fock(V, torch.as_tensor(_density(case["basis"], Z, xyz, seed, case["density"]), device="cuda"))
    return G.to(torch.complex128) if kind == "formpt" else G.reshape(-1)
