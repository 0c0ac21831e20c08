"""Performance cases of the density-fitting backend, through its public entry points.

Six kinds of work, each over the range of molecules that programs bring:

* ``jk``     J and K of occupied orbitals with B resident (``Plan.jk``): the inner
             step of an SCF written on the library;
* ``build``  everything from the metric to B, then J and K (``Plan.build`` and
             ``Plan.jk``): the step of a new geometry;
* ``fock``   energy and Fock matrix of a density (``B200DFCoulomb.fock``): what
             dftax evaluates in every iteration, one or two spin channels;
* ``grad``   nuclear gradient of the fitted energy (``Plan.energy_grad``): one step
             of a geometry optimization;
* ``xc``     exchange-correlation energy and matrix on the Becke grid
             (``KS.xc_energy``);
* ``scf``    a whole solve from the geometry (``KS`` and ``scf``).

The molecules are the package's seeded water clusters and alkanes (hydrogen to
oxygen; orbital shells up to f and auxiliary shells up to g with carbon), in both
precisions. ``exact`` restates every kind in plain torch float64: McMurchie-Davidson
integrals by dense recursions, an eigendecomposition of the metric, dense
contractions and autograd; it shares no code with the library (the input arrays and
the quadrature points, which are given to both, come from the package).
"""

import math

import numpy as np
import torch

from dftax_b200 import B200DFCoulomb, Plan, df, systems
from dftax_b200.grid import becke, becke_grid
from dftax_b200.ks import KS, scf

DEV = "cuda"
F64 = torch.float64
CUTOFF = 1e-7        # metric eigenvalues kept above this share of the largest
HYBRID = 0.25        # exact exchange of PBE0


def listed():
    return [
        # one small molecule: an SCF inner step that is all launches and latency
        {"name": "jk_water1_fp64", "op": "jk", "system": "water", "n": 1, "precision": "fp64"},
        # an ordinary cluster in full precision
        {"name": "jk_water12_fp64", "op": "jk", "system": "water", "n": 12, "precision": "fp64"},
        # an odd occupation (41 orbitals) with f and g shells
        {"name": "jk_alkane10_mixed", "op": "jk", "system": "alkane", "n": 10, "precision": "mixed"},
        # the largest configured cluster held in memory: tens of GB per step
        {"name": "jk_water32_mixed", "op": "jk", "system": "water", "n": 32, "precision": "mixed"},
        # a new geometry of a small molecule (scans, serving)
        {"name": "build_water2_fp64", "op": "build", "system": "water", "n": 2, "precision": "fp64"},
        # the benchmark's own step
        {"name": "build_water16_mixed", "op": "build", "system": "water", "n": 16, "precision": "mixed"},
        # a screened chain in full precision
        {"name": "build_alkane8_fp64", "op": "build", "system": "alkane", "n": 8, "precision": "fp64",
         "screen": 1e-10},
        # the drop-in interface in a closed-shell SCF
        {"name": "fock_water6_fp64", "op": "fock", "system": "water", "n": 6, "precision": "fp64",
         "spins": 1},
        # and for an open shell of an ordinary chain
        {"name": "fock_alkane6_open_mixed", "op": "fock", "system": "alkane", "n": 6,
         "precision": "mixed", "spins": 2},
        # one force evaluation
        {"name": "grad_water4_fp64", "op": "grad", "system": "water", "n": 4, "precision": "fp64",
         "spins": 1},
        # one quadrature on the default grid
        {"name": "xc_water6", "op": "xc", "system": "water", "n": 6, "precision": "fp64"},
        # a whole request: geometry in, converged density out
        {"name": "scf_water3_mixed", "op": "scf", "system": "water", "n": 3, "precision": "mixed"},
    ]


# molecules per kind: (largest water cluster, largest alkane)
RANGES = {"jk": (32, 12), "build": (16, 8), "fock": (12, 8), "grad": (6, 3), "xc": (8, 4),
          "scf": (5, 3)}


def draw(rng):
    op = rng.choice(["jk", "jk", "build", "build", "fock", "grad", "xc", "scf"])
    system = rng.choice(["water", "water", "alkane"])
    top = RANGES[op][0 if system == "water" else 1]
    n = min(top, int(math.exp(rng.uniform(0.0, math.log(top + 1.0)))))
    case = {"op": op, "system": system, "n": n, "precision": rng.choice(["fp64", "mixed"])}
    if op in ("fock", "grad"):
        case["spins"] = rng.choice([1, 1, 2])
    if op in ("jk", "build") and system == "alkane" and rng.random() < 0.5:
        case["screen"] = rng.choice([1e-10, 1e-12])
    if op in ("jk", "build"):
        # columns of the coefficient block: the occupied ones, or those of a smaller core
        case["drop"] = rng.choice([0, 0, 1, 2])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _molecule(case, seed):
    if case["system"] == "water":
        sym, xyz = systems.water_cluster(case["n"], seed=seed)
    else:
        sym, xyz = systems.alkane(case["n"], seed=seed)
    orb, aux = systems.basis_for(sym, xyz)
    return sym, xyz, orb, aux, systems.n_electrons(sym) // 2


def _columns(case, nocc):
    return max(1, nocc - case.get("drop", 0))


def _orbitals(nao, ncol, seed):
    g = torch.Generator().manual_seed(1000 + seed)
    q, _ = torch.linalg.qr(torch.randn(nao, ncol, generator=g, dtype=F64))
    return q.contiguous().to(DEV)


def _density(case, nao, nocc, seed):
    """Spin-stacked density of orthonormal occupied orbitals."""
    if case.get("spins", 1) == 1:
        c = _orbitals(nao, nocc, seed)
        return 2.0 * (c @ c.T)[None]
    a, b = _orbitals(nao, nocc, seed), _orbitals(nao, max(1, nocc - 1), seed + 500)
    return torch.stack([a @ a.T, b @ b.T])


def _aufbau(S, H, nocc, seed):
    """Closed-shell density of a slightly perturbed one-electron Hamiltonian."""
    s, U = torch.linalg.eigh(S)
    X = U[:, s > CUTOFF] / s[s > CUTOFF].sqrt()
    g = torch.Generator().manual_seed(2000 + seed)
    r = torch.randn(S.shape, generator=g, dtype=F64).to(S.device)
    C = X @ torch.linalg.eigh(X.T @ (H + 0.02 * S @ (r + r.T) @ S) @ X)[1][:, :nocc]
    return 2.0 * C @ C.T


def prepare(case, seed):
    sym, xyz, orb, aux, nocc = _molecule(case, seed)
    op = case["op"]
    state = {"case": case, "sym": sym, "xyz": xyz, "orb": orb, "aux": aux}
    if op == "scf":
        return state
    if op == "xc":
        state["ks"] = KS(sym, xyz, orb, coulomb=df(aux, precision=case["precision"]), xc="PBE0")
        S, T, V = state["ks"].one_electron()
        state["P"] = _aufbau(S, T + V, nocc, seed)
        return state
    if op == "fock":
        state["term"] = B200DFCoulomb(orb, aux, HYBRID, precision=case["precision"])
        state["P"] = _density(case, orb.nao, nocc, seed)
        return state
    state["plan"] = Plan(orb, aux, screen=case.get("screen"), precision=case["precision"])
    state["plan"].build()
    if op == "grad":
        state["P"] = _density(case, orb.nao, nocc, seed)
    else:
        state["C"] = _orbitals(orb.nao, _columns(case, nocc), seed)
    return state


def run(state):
    op = state["case"]["op"]
    if op == "jk":
        J, K = state["plan"].jk(state["C"])
        return {"J": J, "K": K}
    if op == "build":
        state["plan"].build()
        J, K = state["plan"].jk(state["C"])
        return {"J": J, "K": K}
    if op == "fock":
        e, F = state["term"].fock(state["P"])
        return {"e": e, "F": F}
    if op == "grad":
        e, g = state["plan"].energy_grad(state["P"], HYBRID, state["xyz"])
        return {"e": e, "g": g}
    if op == "xc":
        e, V = state["ks"].xc_energy(state["P"])
        return {"e": e, "V": V}
    ks = KS(state["sym"], state["xyz"], state["orb"], xc="PBE0",
            coulomb=df(state["aux"], precision=state["case"]["precision"]))
    r = scf(ks, guess="sad")
    ks.close()
    ks.plan.close()
    return {"e": r.e_tot, "eps": r.mo_energy, "P": r.P}


def _sizes(case):
    """(AO pairs, nao, naux, fitted directions, occupied columns), from the formulas of the sets."""
    n = case["n"]
    if case["system"] == "water":
        nao, naux, nocc = 30 * n, 141 * n, 5 * n
    else:
        nao, naux, nocc = 39 * n + 6 * (2 * n + 2), 144 * n + 28 * (2 * n + 2), 4 * n + 1
    nfit = int(0.87 * naux)   # about: the rest falls below the metric's cutoff
    return nao * (nao + 1) // 2, nao, naux, nfit, _columns(case, nocc)


def work(case):
    pairs, nao, naux, nfit, nocc = _sizes(case)
    spins = case.get("spins", 1)
    b_bytes, nn = 8.0 * pairs * nfit, 8.0 * nao * nao
    j = 4.0 * pairs * nfit
    k = 2.0 * nao * nao * nfit * nocc + 1.0 * nao * nao * nfit * nocc
    fit = 2.0 * pairs * naux * nfit + 9.0 * naux ** 3     # B and the metric's factor
    points = 9500.0 * (3 * case["n"] if case["system"] == "water" else 3 * case["n"] + 2)
    quad = 4.0 * points * min(nao, 150) ** 2              # the functions that reach a point
    op = case["op"]
    if op == "jk":
        return {"bytes": b_bytes + 8.0 * nao * nocc + 2 * nn, "flops": j + k}
    if op == "build":
        return {"bytes": b_bytes + 2 * nn, "flops": fit + j + k}
    if op == "fock":
        return {"bytes": b_bytes + 2 * spins * nn, "flops": j + spins * k}
    if op == "grad":
        # half transforms, the back transform to pairs, B^T H and H L^T
        return {"bytes": b_bytes + spins * nn,
                "flops": spins * 4.0 * nao * nao * nfit * nocc + 2.0 * pairs * nfit * (nfit + naux)}
    if op == "xc":
        return {"bytes": 32.0 * points + 2 * nn, "flops": quad}
    return {"bytes": b_bytes + 32.0 * points + 2 * nn, "flops": fit + 14.0 * (j + k + quad)}


def tolerance(case):
    # float64 J, K, E: two correct evaluations of the metric differ by the rounding that its
    # condition number (up to 1e7 kept) amplifies; 1.2e-10 was seen against exact(). Mixed
    # plans truncate their digits at 32 to 40 bits: 1.1e-8 was seen
    if case["op"] == "scf":
        return {"rel": 1e-6}    # the commutator's convergence threshold; 1e-7 was seen
    if case["op"] == "xc":
        return {"rel": 1e-12}
    if case["op"] == "grad":
        # the metric's derivative carries V+ twice: two forms of V+ move the gradient by
        # 6e-9 (water) and 4e-8 (carbon sets, which drop more directions)
        return {"rel": 1e-7 if case["system"] == "water" else 1e-6}
    return {"rel": 5e-10 if case["precision"] == "fp64" else 5e-8}


# ---------------------------------------------------------------------------
# 64-bit restatement in plain torch
# ---------------------------------------------------------------------------

def _comps(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _herm(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


class _Boys(torch.autograd.Function):
    """F_0 .. F_M of T in the last axis; dF_m/dT = -F_{m+1}."""

    @staticmethod
    def values(T, M):
        small = T < 32.0
        ts = torch.where(small, T, torch.zeros_like(T))
        term = torch.full_like(T, 1.0 / (2 * M + 1))
        acc = term.clone()
        for k in range(1, 150):
            term = term * (2.0 * ts / (2 * M + 2 * k + 1))
            acc = acc + term
        ex = torch.exp(-T)
        down = [None] * (M + 1)
        down[M] = acc * torch.exp(-ts)
        for m in range(M, 0, -1):
            down[m - 1] = (2.0 * ts * down[m] + torch.exp(-ts)) / (2 * m - 1)
        tl = torch.where(small, torch.full_like(T, 32.0), T)
        up = 0.5 * torch.sqrt(math.pi / tl) * torch.erf(torch.sqrt(tl))
        out = []
        for m in range(M + 1):
            out.append(torch.where(small, down[m], up))
            up = ((2 * m + 1) * up - ex) / (2.0 * tl)
        return torch.stack(out, -1)

    @staticmethod
    def forward(ctx, T, M):
        F = _Boys.values(T, M + 1)
        ctx.save_for_backward(F[..., 1:])
        return F[..., :-1]

    @staticmethod
    def backward(ctx, g):
        return -(g * ctx.saved_tensors[0]).sum(-1), None


def _hermite_r(alpha, d, L):
    """R_tuv of all t + u + v <= L, stacked last in the order of _herm(L)."""
    F = _Boys.apply(alpha * (d * d).sum(-1), L)
    x, y, z = d.unbind(-1)
    cur = {}
    for m in range(L, -1, -1):
        new = {(0, 0, 0): (-2.0 * alpha) ** m * F[..., m]}
        for t, u, v in sorted(_herm(L - m), key=sum):
            if t:
                r = x * cur[t - 1, u, v]
                if t > 1:
                    r = r + (t - 1) * cur[t - 2, u, v]
            elif u:
                r = y * cur[t, u - 1, v]
                if u > 1:
                    r = r + (u - 1) * cur[t, u - 2, v]
            elif v:
                r = z * cur[t, u, v - 1]
                if v > 1:
                    r = r + (v - 1) * cur[t, u, v - 2]
            else:
                continue
            new[t, u, v] = r
        cur = new
    return torch.stack([cur[h] for h in _herm(L)], -1)


class _Shells:
    """Shells of a basis (one primitive each), grouped by l, with spherical blocks."""

    def __init__(self, b):
        an = np.asarray(b.angular)
        rows = np.nonzero((an[:, 1] == 0) & (an[:, 2] == 0))[0]
        assert b.exponents.shape[1] == 1
        self.l = an[rows, 0]
        self.out0 = np.concatenate([[0], np.cumsum(2 * self.l + 1)[:-1]])
        self.n, self.nout = len(rows), int((2 * self.l + 1).sum())
        self.ex = torch.tensor(np.asarray(b.exponents)[rows, 0], device=DEV)
        self.co = torch.tensor(np.asarray(b.coefficients)[rows, 0], device=DEV)
        self.cen = torch.tensor(np.asarray(b.centers)[rows], device=DEV, dtype=F64)
        self.blk = {}
        for r, l, o in zip(rows, self.l, self.out0):
            if l not in self.blk:
                nc = len(_comps(l))
                self.blk[l] = torch.tensor(b.cart2sph[r:r + nc, o:o + 2 * l + 1], device=DEV)

    def of(self, l):
        return torch.tensor(np.nonzero(self.l == l)[0], device=DEV)

    def columns(self, idx, l):
        o = torch.tensor(self.out0, device=DEV)[idx]
        return o[:, None] + torch.arange(2 * l + 1, device=DEV)[None]


def _e_axis(a, b, AB, la, lb):
    """Hermite coefficients of one axis, (N, la + 1, lb + 1, la + lb + 1)."""
    p = a + b
    pa, pb, h = -b / p * AB, a / p * AB, 0.5 / p
    zero = torch.zeros_like(p)
    E = {(0, 0): [torch.exp(-a * b / p * AB * AB)]}

    def up(prev, s):
        n = len(prev)
        g = lambda t: prev[t] if 0 <= t < n else zero  # noqa: E731
        return [h * g(t - 1) + s * g(t) + (t + 1) * g(t + 1) for t in range(n + 1)]

    for i in range(la + 1):
        if i:
            E[i, 0] = up(E[i - 1, 0], pa)
        for j in range(1, lb + 1):
            E[i, j] = up(E[i, j - 1], pb)
    full = lambda e: torch.stack(e + [zero] * (la + lb + 1 - len(e)), -1)  # noqa: E731
    return torch.stack([torch.stack([full(E[i, j]) for j in range(lb + 1)], 1)
                        for i in range(la + 1)], 1)


def _pairs(sh, cen, ia, ib, la, lb):
    """Exponent, center and spherical Hermite coefficients (N, na nb, nherm) of shell pairs."""
    a, b = sh.ex[ia], sh.ex[ib]
    A, B = cen[ia], cen[ib]
    p = a + b
    P = (a[:, None] * A + b[:, None] * B) / p[:, None]
    E = [_e_axis(a, b, A[:, x] - B[:, x], la, lb) for x in range(3)]
    ca, cb, h = _comps(la), _comps(lb), _herm(la + lb)
    H = 1.0
    for x in range(3):
        i = torch.tensor([c[x] for c in ca], device=DEV)[:, None, None]
        j = torch.tensor([c[x] for c in cb], device=DEV)[None, :, None]
        t = torch.tensor([c[x] for c in h], device=DEV)[None, None, :]
        H = H * E[x][:, i, j, t]
    H = torch.einsum("nabh,ai,bj->nijh", H, sh.blk[la], sh.blk[lb])
    w = (sh.co[ia] * sh.co[ib])[:, None, None]
    return p, P, H.flatten(1, 2) * w


def _singles(sh, cen, idx, l):
    """The same of single shells."""
    q = sh.ex[idx]
    E = _e_axis(q, torch.zeros_like(q), torch.zeros_like(q), l, 0)[:, :, 0]
    c, h = _comps(l), _herm(l)
    H = 1.0
    for x in range(3):
        i = torch.tensor([k[x] for k in c], device=DEV)[:, None]
        t = torch.tensor([k[x] for k in h], device=DEV)[None, :]
        H = H * E[:, i, t]
    H = torch.einsum("nch,ci->nih", H, sh.blk[l])
    return q, cen[idx], H * sh.co[idx][:, None, None]


def _coulomb(bra, Lb, ket, Lk):
    """(N, M, nbra, nket) Coulomb integrals of two sets of Hermite expansions."""
    p, P, Hb = bra
    q, Q, Hk = ket
    pq = p[:, None] * q[None]
    s = p[:, None] + q[None]
    R = _hermite_r(pq / s, P[:, None] - Q[None], Lb + Lk)
    at = {h: i for i, h in enumerate(_herm(Lb + Lk))}
    hb, hk = _herm(Lb), _herm(Lk)
    idx = torch.tensor([[at[b[0] + k[0], b[1] + k[1], b[2] + k[2]] for k in hk] for b in hb],
                       device=DEV)
    sign = torch.tensor([(-1.0) ** sum(k) for k in hk], device=DEV, dtype=F64)
    pref = 2.0 * math.pi ** 2.5 / (pq * torch.sqrt(s))
    W = torch.einsum("nmhk,mck->nmhc", R[..., idx], Hk * sign)
    return torch.einsum("nmhc,nbh,nm->nmbc", W, Hb, pref)


def _three_blocks(orb, aux, co, ca):
    """Blocks of (ij|P) over unique shell pairs: (index of rows i, j, columns P, values)."""
    for la in sorted(set(orb.l), reverse=True):
        for lb in sorted(set(orb.l)):
            if lb > la:
                continue
            I, J = orb.of(la), orb.of(lb)
            ia, ib = (x.flatten() for x in torch.meshgrid(I, J, indexing="ij"))
            if la == lb:
                ia, ib = ia[ia >= ib], ib[ia >= ib]
            for lc in sorted(set(aux.l)):
                c = aux.of(lc)
                L = la + lb + lc
                per = len(c) * (4 * len(_herm(L)) + len(_herm(la + lb)) * (len(_herm(lc)) + 2 * lc + 1)
                                + 300) * 8
                step = max(1, int(1.5e9 // per))
                for s in range(0, len(ia), step):
                    x, y = ia[s:s + step], ib[s:s + step]
                    v = _coulomb(_pairs(orb, co, x, y, la, lb), la + lb, _singles(aux, ca, c, lc), lc)
                    yield orb.columns(x, la), orb.columns(y, lb), aux.columns(c, lc), v


def _block_index(ri, rj, cp):
    i = ri[:, None, :, None, None]
    j = rj[:, None, None, :, None]
    return i, j, cp[None, :, None, None, :]


def _three_center(orb, aux):
    T = torch.zeros(orb.nout, orb.nout, aux.nout, device=DEV, dtype=F64)
    for ri, rj, cp, v in _three_blocks(orb, aux, orb.cen, aux.cen):
        i, j, P = _block_index(ri, rj, cp)
        v = v.reshape(v.shape[0], v.shape[1], ri.shape[1], rj.shape[1], -1)
        T[i, j, P] = v
        T[j, i, P] = v
    return T


def _two_blocks(aux, ca):
    for la in sorted(set(aux.l)):
        for lb in sorted(set(aux.l)):
            a, b = aux.of(la), aux.of(lb)
            v = _coulomb(_singles(aux, ca, a, la), la, _singles(aux, ca, b, lb), lb)
            yield aux.columns(a, la)[:, None, :, None], aux.columns(b, lb)[None, :, None, :], v


def _metric(aux):
    V = torch.zeros(aux.nout, aux.nout, device=DEV, dtype=F64)
    for i, j, v in _two_blocks(aux, aux.cen):
        V[i, j] = v
    return V


def _fit(orb, aux):
    """B = (ij|P) L with L L^T the cut pseudo-inverse of the metric, and L."""
    w, U = torch.linalg.eigh(_metric(aux))
    keep = w > CUTOFF * w[-1]
    L = U[:, keep] / w[keep].sqrt()
    T = _three_center(orb, aux)
    return (T.reshape(-1, aux.nout) @ L).reshape(orb.nout, orb.nout, -1), L


def _j_of(B, D):
    n = B.shape[0]
    g = torch.einsum("mnx,mn->x", B, D)
    return (B.reshape(n * n, -1) @ g).reshape(n, n), g


def _k_of(B, C):
    K = torch.zeros(B.shape[0], B.shape[0], device=DEV, dtype=F64)
    for x in range(0, B.shape[2], 256):
        X = torch.einsum("mnx,ni->mxi", B[:, :, x:x + 256], C).flatten(1)
        K += X @ X.T
    return K


def _fock_of(B, P, factors):
    """Energy and P-gradient of the fitted Coulomb and hybrid exchange."""
    J, g = _j_of(B, P.sum(0))
    e, F = 0.5 * float(g @ g), []
    half = 0.5 if P.shape[0] == 1 else 1.0
    for Ps, C in zip(P, factors):
        K = _k_of(B, C)
        e -= 0.5 * half * HYBRID * float((Ps * K).sum())
        F.append(J - half * HYBRID * K)
    return e, torch.stack(F)


def _factors(P):
    out = []
    for Ps in P:
        w, U = torch.linalg.eigh(Ps)
        keep = w > 1e-10 * w[-1]
        out.append(U[:, keep] * w[keep].sqrt())
    return out


def _gradient(orb, aux, P, xyz):
    B, L = _fit(orb, aux)
    g = torch.einsum("mnx,mn->x", B, P.sum(0))
    k = -(0.25 if P.shape[0] == 1 else 0.5) * HYBRID
    H = g * P.sum(0)[..., None]
    for Ps in P:
        H = H + 2.0 * k * torch.einsum("ma,abx,bn->mnx", Ps, B, Ps)
    M = H.flatten(0, 1).T @ B.flatten(0, 1)
    e = 0.5 * float(torch.trace(M))
    W = L @ M @ L.T
    G = H @ L.T
    del B, H
    co, ca = orb.cen.clone().requires_grad_(True), aux.cen.clone().requires_grad_(True)
    for ri, rj, cp, v in _three_blocks(orb, aux, co, ca):
        i, j, p = _block_index(ri, rj, cp)
        w = G[i, j, p] + torch.where((ri[:, :1] == rj[:, :1])[:, None, None, :, None],
                                     torch.zeros((), device=DEV, dtype=F64), G[j, i, p])
        (v * w.flatten(2, 3)).sum().backward()
    for i, j, v in _two_blocks(aux, ca):
        (-0.5 * (v * W[i, j]).sum()).backward()
    atoms = torch.tensor(np.asarray(xyz), device=DEV)
    out = torch.zeros_like(atoms)
    for sh, d in ((orb, co.grad), (aux, ca.grad)):
        out.index_add_(0, torch.cdist(sh.cen, atoms).argmin(1), d)
    return e, out


def _ao(b, pts):
    """Function values (g, nao) and gradients (3, g, nao) at points."""
    an = torch.tensor(np.asarray(b.angular), device=DEV)
    d = pts[:, None] - torch.tensor(np.asarray(b.centers), device=DEV)[None]
    a = torch.tensor(np.asarray(b.exponents)[:, 0], device=DEV)
    rad = torch.tensor(np.asarray(b.coefficients)[:, 0], device=DEV) * torch.exp(-a * (d * d).sum(-1))
    c2s = torch.tensor(b.cart2sph, device=DEV)
    pw = [d[..., x] ** an[:, x] for x in range(3)]
    val = pw[0] * pw[1] * pw[2] * rad
    grad = []
    for x in range(3):
        lo = an[:, x] * d[..., x] ** (an[:, x] - 1).clamp(min=0)
        grad.append((lo * pw[(x + 1) % 3] * pw[(x + 2) % 3] * rad - 2.0 * a * d[..., x] * val) @ c2s)
    return val @ c2s, torch.stack(grad)


def _pbe0(rho, grad):
    """Energy density per volume of 3/4 PBE exchange and PBE correlation, unpolarized."""
    s2g = (grad * grad).sum(-1) + 1e-60
    kf = (3.0 * math.pi ** 2 * rho) ** (1.0 / 3.0)
    s2 = s2g / (2.0 * kf * rho) ** 2
    kappa, mu = 0.804, 0.2195149727645171
    ex = -3.0 * kf / (4.0 * math.pi) * (1.0 + kappa - kappa / (1.0 + mu * s2 / kappa))
    rs = (3.0 / (4.0 * math.pi * rho)) ** (1.0 / 3.0)
    q = rs.sqrt()
    A, a1, b1, b2, b3, b4 = 0.0310907, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294
    pw = -2.0 * A * (1.0 + a1 * rs) * torch.log1p(1.0 / (2.0 * A * (b1 * q + b2 * rs + b3 * rs * q + b4 * rs * rs)))
    gamma, beta = (1.0 - math.log(2.0)) / math.pi ** 2, 0.06672455060314922
    t2 = s2g / (4.0 * (4.0 * kf / math.pi) * rho ** 2)
    Ac = beta / (gamma * torch.expm1(-pw / gamma))
    f = t2 + Ac * t2 * t2
    return rho * (0.75 * ex + pw + gamma * torch.log1p(beta / gamma * f / (1.0 + Ac * f)))


class _Quadrature:
    def __init__(self, orb, sym, xyz):
        pts, w = becke_grid(sym, xyz, becke())
        self.parts = []
        for s in range(0, len(w), 20000):
            self.parts.append((_ao(orb, torch.tensor(pts[s:s + 20000], device=DEV)),
                               torch.tensor(w[s:s + 20000], device=DEV)))

    def __call__(self, P):
        e, V = 0.0, torch.zeros_like(P)
        for (phi, dphi), w in self.parts:
            X = phi @ P
            rho = (X * phi).sum(1).requires_grad_(True)
            gr = 2.0 * torch.stack([(X * d).sum(1) for d in dphi], -1).requires_grad_(True)
            live = rho > 1e-10
            dens = torch.zeros_like(rho)
            dens[live] = _pbe0(rho[live], gr[live])
            tot = (w * dens).sum()
            vr, vg = torch.autograd.grad(tot, (rho, gr))
            Wm = 0.5 * vr[:, None] * phi + sum(vg[:, x:x + 1] * dphi[x] for x in range(3))
            A = phi.T @ Wm
            e, V = e + float(tot.detach()), V + A + A.T
        return e, V


def _one_electron(orb, xyz, Z):
    S, T, V = (torch.zeros(orb.nout, orb.nout, device=DEV, dtype=F64) for _ in range(3))
    big = torch.full((len(Z),), 1e18, device=DEV, dtype=F64)   # point charges
    pts = (big, torch.tensor(np.asarray(xyz), device=DEV), (-Z * (big / math.pi) ** 1.5)[:, None, None])
    for la in sorted(set(orb.l)):
        for lb in sorted(set(orb.l)):
            ia, ib = (x.flatten() for x in torch.meshgrid(orb.of(la), orb.of(lb), indexing="ij"))
            a, b, AB = orb.ex[ia], orb.ex[ib], orb.cen[ia] - orb.cen[ib]
            E = [_e_axis(a, b, AB[:, x], la, lb + 2)[..., 0] for x in range(3)]
            ov, kin = [], []
            for ca in _comps(la):
                for cb in _comps(lb):
                    s = [E[x][:, ca[x], cb[x]] for x in range(3)]
                    k = 0.0
                    for x in range(3):
                        j = cb[x]
                        d = -2.0 * b * b * E[x][:, ca[x], j + 2] + b * (2 * j + 1) * s[x]
                        if j > 1:
                            d = d - 0.5 * j * (j - 1) * E[x][:, ca[x], j - 2]
                        k = k + d * s[(x + 1) % 3] * s[(x + 2) % 3]
                    ov.append(s[0] * s[1] * s[2])
                    kin.append(k)
            w = orb.co[ia] * orb.co[ib] * (math.pi / (a + b)) ** 1.5
            i, j = orb.columns(ia, la)[:, :, None], orb.columns(ib, lb)[:, None, :]
            for M, m in ((S, ov), (T, kin)):
                m = (torch.stack(m, -1) * w[:, None]).reshape(len(ia), len(_comps(la)), -1)
                M[i, j] = torch.einsum("nab,ai,bj->nij", m, orb.blk[la], orb.blk[lb])
            v = _coulomb(_pairs(orb, orb.cen, ia, ib, la, lb), la + lb, pts, 0)
            V[i, j] = v.sum((1, 3)).reshape(len(ia), 2 * la + 1, 2 * lb + 1)
    return S, T, V


def _solve(orb_b, aux_b, sym, xyz, nocc):
    orb, aux = _Shells(orb_b), _Shells(aux_b)
    Z = torch.tensor([float(systems.NUCLEAR_CHARGE[s]) for s in sym], device=DEV, dtype=F64)
    S, T, V = _one_electron(orb, xyz, Z)
    B, _ = _fit(orb, aux)
    quad = _Quadrature(orb_b, sym, xyz)
    at = torch.tensor(np.asarray(xyz), device=DEV)
    R = torch.cdist(at, at) + torch.eye(len(Z), device=DEV, dtype=F64)
    enn = 0.5 * float((Z[:, None] * Z[None] / R).sum() - (Z * Z).sum())
    s, U = torch.linalg.eigh(S)
    X = U[:, s > CUTOFF] / s[s > CUTOFF].sqrt()

    def aufbau(F):
        eps, C = torch.linalg.eigh(X.T @ F @ X)
        return eps, X @ C[:, :nocc]

    _, C = aufbau(T + V)
    Fs, errs, last = [], [], 0.0
    for _ in range(100):
        P = 2.0 * C @ C.T
        e2, F2 = _fock_of(B, P[None], [math.sqrt(2.0) * C])
        exc, vxc = quad(P)
        F = T + V + F2[0] + vxc
        e = enn + float((P * (T + V)).sum()) + e2 + exc
        err = X.T @ (F @ P @ S - S @ P @ F) @ X
        Fs, errs = (Fs + [F])[-8:], (errs + [err])[-8:]
        m = len(Fs)
        A = torch.zeros(m + 1, m + 1, dtype=F64)
        A[:m, :m] = torch.tensor([[float((x * y).sum()) for y in errs] for x in errs])
        A[m, :m] = A[:m, m] = 1.0
        rhs = torch.zeros(m + 1, dtype=F64)
        rhs[m] = 1.0
        c = torch.linalg.lstsq(A, rhs[:, None]).solution[:m, 0]
        eps, C = aufbau(sum(float(x) * y for x, y in zip(c, Fs)))
        if abs(e - last) < 1e-10 and float(err.abs().max()) < 1e-8:
            break
        last = e
    return e, eps, P


def exact(case, seed):
    pairs, nao, naux, nfit, _ = _sizes(case)
    if nao * nao * naux > 5.5e8:    # over 20 seconds, or tens of GB
        return None
    sym, xyz, orb_b, aux_b, nocc = _molecule(case, seed)
    op = case["op"]
    if op == "scf":
        e, eps, P = _solve(orb_b, aux_b, sym, xyz, nocc)
        return {"e": e, "eps": eps[None], "P": P[None]}
    orb, aux = _Shells(orb_b), _Shells(aux_b)
    if op == "xc":
        Z = torch.tensor([float(systems.NUCLEAR_CHARGE[s]) for s in sym], device=DEV, dtype=F64)
        S, T, V = _one_electron(orb, xyz, Z)
        e, V = _Quadrature(orb_b, sym, xyz)(_aufbau(S, T + V, nocc, seed))
        return {"e": e, "V": V}
    if op == "grad":
        e, g = _gradient(orb, aux, _density(case, nao, nocc, seed), xyz)
        return {"e": e, "g": g}
    B, _ = _fit(orb, aux)
    if op == "fock":
        P = _density(case, nao, nocc, seed)
        e, F = _fock_of(B, P, _factors(P))
        return {"e": e, "F": F}
    C = _orbitals(nao, _columns(case, nocc), seed)
    return {"J": _j_of(B, C @ C.T)[0], "K": _k_of(B, C)}
