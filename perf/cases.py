"""Performance cases of the two-electron path, through its public entry points.

Every case is a plain dict.  ``kind`` names the entry point:

  eri      MolGpu.eri_quartets       shell-quartet integrals (Drv2El / Eval_IJKL)
  cho      MolGpu.cho_drv            pivoted Cholesky decomposition of the ERIs
  jk       MolGpu.cho_jk             Coulomb/exchange of one density
  jkbatch  MolGpu.cho_jk_batch       of several densities (alpha and beta)
  fock     MolGpu.choscf_lk          Fock update from a density matrix
  grad     MolGpu.drvg1              two-electron nuclear gradient

and ``system`` / ``natom`` the synthetic molecule (openmolcas_b200/basis.py):
the basis types and their shares are those of the repository's configurations.
The base geometry belongs to the case; the seed displaces every atom a little
(a step of a geometry optimisation) and draws the densities, so that work and
sizes do not depend on the seed while every input does.  The number of Cholesky
vectors follows the geometry, so the decompositions move and mirror the whole
molecule instead: all integrals change in sign or rounding, the pivots do not.
"""
from __future__ import annotations

import itertools
import math

import numpy as np
import torch

from openmolcas_b200 import basis as B
from openmolcas_b200.molgpu import MolGpu

# basis types and their shares, as in basis.CONFIGS
SYSTEMS = {
    "water": [("3s2p1d", 1), ("2s1p", 2)],           # one heavy, two light atoms
    "3s2p1d": [("3s2p1d", 1)],                       # the 84-function cluster's basis
    "mix": [("3s2p1d", 5), ("2s1p", 1)],             # the 1500-function cluster's mix
    "4s3p2d": [("4s3p2d", 1)],                       # the gradient cluster's basis
    "uneven": [("2s1p_r", 3), ("4s3p2d1f_r", 2)],    # uneven classes up to f, 1-12 primitives
}
PRECISIONS = {"fp64": MolGpu.PREC_FP64, "mixed": MolGpu.PREC_MIXED}
CUTINT = 1e-12


def listed():
    return [
        # one shell quartet at a time: the per-quartet kernel pointer of the
        # integral driver (d, p | p, s of a small molecule): pure latency
        dict(name="eri_one_quartet", kind="eri", system="water", natom=3, quartets=1),
        # conventional integrals of a small molecule: every unique quartet once
        dict(name="eri_small_molecule", kind="eri", system="water", natom=3, quartets=0),
        # one large batch of the 40-atom cluster with uneven classes (general
        # contractions, s to f, 1 to 12 primitives): integral throughput
        dict(name="eri_uneven_batch", kind="eri", system="uneven", natom=40, quartets=200000),
        # the decomposition that opens a small calculation
        dict(name="cho_84bf", kind="cho", system="3s2p1d", natom=6, thrcom=1e-4),
        # the decomposition of an ordinary molecule at the tighter threshold
        dict(name="cho_300bf", kind="cho", system="mix", natom=24, thrcom=1e-6),
        # J/K of one SCF iteration of a small molecule (default precision)
        dict(name="jk_84bf_fp64", kind="jk", system="3s2p1d", natom=6, thrcom=1e-4, rank=15, precision="fp64"),
        # the Fock update from a density matrix (density decomposed first)
        dict(name="fock_300bf_fp64", kind="fock", system="mix", natom=24, thrcom=1e-4, rank=41, precision="fp64"),
        # unrestricted SCF: alpha and beta of uneven rank in one pass
        dict(name="jk_uhf_403bf_mixed", kind="jkbatch", system="mix", natom=32, thrcom=1e-4, rank=53, ndens=2,
             precision="mixed"),
        # J/K of one SCF iteration of a large molecule (few vectors per function keep its set-up short)
        dict(name="jk_1250bf_mixed", kind="jk", system="mix", natom=100, thrcom=1e-3, rank=167, precision="mixed"),
        # forces of a small molecule
        dict(name="grad_small_molecule", kind="grad", system="water", natom=3, rank=5, spin=False, exfac=1.0),
        # forces of an open shell with a hybrid functional's exchange fraction
        dict(name="grad_open_shell_138bf", kind="grad", system="4s3p2d", natom=6, rank=12, spin=True, exfac=0.2),
        # forces of the 20-atom cluster: the largest work
        dict(name="grad_460bf", kind="grad", system="4s3p2d", natom=20, rank=40, spin=False, exfac=1.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eri", "eri", "cho", "jk", "jk", "jkbatch", "fock", "grad", "grad"])
    if kind == "eri":
        system = rng.choice(["water", "3s2p1d", "4s3p2d", "uneven"])
        natom = _log_int(rng, 3, 40 if system != "4s3p2d" else 20)
        return dict(kind=kind, system=system, natom=natom, quartets=_log_int(rng, 1, 200000))
    if kind == "cho":
        system = rng.choice(["water", "3s2p1d", "mix"])
        return dict(kind=kind, system=system, natom=_log_int(rng, 3, 24), thrcom=rng.choice([1e-4, 1e-5, 1e-6]))
    if kind == "grad":
        system = rng.choice(["water", "3s2p1d", "4s3p2d"])
        return dict(kind=kind, system=system, natom=_log_int(rng, 2, 24 if system != "4s3p2d" else 14),
                    rank=rng.randint(1, 20), spin=rng.random() < 0.4, exfac=rng.choice([1.0, 1.0, 0.2, 0.0]))
    natom = _log_int(rng, 3, 40)
    nbf = natom * 12
    case = dict(kind=kind, system=rng.choice(["3s2p1d", "mix"]), natom=natom, thrcom=rng.choice([1e-4, 1e-5]),
                rank=max(1, int(nbf * rng.uniform(0.05, 0.2))), precision=rng.choice(["fp64", "mixed", "mixed"]))
    if kind == "jkbatch":
        case["ndens"] = rng.choice([2, 2, 3])
    return case


# ------------------------------------------------------------------ inputs
def _base(case):
    """The case's molecule before the seed displaces it."""
    shares = SYSTEMS[case["system"]]
    natom, total = case["natom"], sum(k for _, k in shares)
    mix = [(t, max(0, round(k * natom / total))) for t, k in shares]
    mix[0] = (mix[0][0], natom - sum(k for _, k in mix[1:]))
    return B.make_molecule(case["system"], natom, mix, 7 * natom + len(case["system"]))


def _molecule(case, seed):
    m = _base(case)
    rng = np.random.default_rng([seed, 1])
    if case["kind"] == "cho":
        return m.at(m.coords * rng.choice([-1.0, 1.0], 3) + rng.uniform(-3.0, 3.0, 3))
    return m.at(m.coords + rng.uniform(-0.05, 0.05, m.coords.shape))


def _factors(case, seed, nbf):
    """Density factors C (nbf x r), one per density; the ranks differ by one."""
    out = []
    for d in range(case.get("ndens", 1)):
        r = max(1, min(nbf, case["rank"] - d))
        out.append(np.random.default_rng([seed, 2, d]).standard_normal((nbf, r)) / math.sqrt(r))
    return out


def _densities(case, seed, nbf):
    """Total density and spin density (or None) of a gradient case."""
    (Ca,) = _factors(dict(case, ndens=1), seed, nbf)
    if not case["spin"]:
        return Ca @ Ca.T, None
    Cb = Ca[:, :max(1, Ca.shape[1] - 2)]
    return 0.5 * (Ca @ Ca.T + Cb @ Cb.T), 0.5 * (Ca @ Ca.T - Cb @ Cb.T)


def _quartets(case, m):
    """The case's canonical quartets (i >= j, k >= l, ij >= kl): all unique ones
    for quartets = 0, else a sample of them (one quartet: the (dp|ps)-like
    quartet of the highest shells)."""
    ns = len(m.shells)
    ii, jj = np.tril_indices(ns)
    npair = ii.size
    nall = npair * (npair + 1) // 2
    nq = case["quartets"]
    if nq == 0 or nq >= nall:
        P, Q = np.tril_indices(npair)
    elif nq == 1:
        l = np.array([s.l for s in m.shells])
        i = int(np.argmax(l))
        p, s = int(np.flatnonzero(l == 1)[0]), int(np.flatnonzero(l == 0)[0])
        tri = lambda a, b: max(a, b) * (max(a, b) + 1) // 2 + min(a, b)
        pq = sorted([tri(i, p), tri(p, s)], reverse=True)
        P, Q = np.array(pq[:1]), np.array(pq[1:])
    else:
        t = np.sort(np.random.default_rng(3).choice(nall, nq, replace=False))
        P = ((np.sqrt(8.0 * t + 1.0) - 1.0) / 2.0).astype(np.int64)
        P += (P + 1) * (P + 2) // 2 <= t
        P -= P * (P + 1) // 2 > t
        Q = t - P * (P + 1) // 2
    return np.stack([ii[P], jj[P], ii[Q], jj[Q]], axis=1).astype(np.int32)


def prepare(case, seed):
    m = _molecule(case, seed)
    g = MolGpu(m)
    st = dict(case=case, g=g)
    dev = f"cuda:{g.device}"
    if case["kind"] == "eri":
        st["q"] = _quartets(case, m)
    elif case["kind"] == "grad":
        D, DS = _densities(case, seed, m.nbf)
        st["D"] = torch.from_numpy(D).to(dev)
        st["DS"] = None if DS is None else torch.from_numpy(DS).to(dev)
        g.schwarz()
    elif case["kind"] != "cho":
        g.cho_drv(thrcom=case["thrcom"])
        st["C"] = [torch.from_numpy(C).to(dev) for C in _factors(case, seed, m.nbf)]
        if case["kind"] == "fock":
            st["D"] = st["C"][0] @ st["C"][0].t()
            st["F"] = torch.empty((m.nbf, m.nbf), dtype=torch.float64, device=dev)
    torch.cuda.synchronize()
    return st


def run(st):
    case, g = st["case"], st["g"]
    kind = case["kind"]
    if kind == "eri":
        return g.eri_quartets(st["q"])
    if kind == "cho":
        g.cho_drv(thrcom=case["thrcom"])
        return (g.cho_vectors(), g.cho_diag()) + g.cho_pivots()
    if kind == "grad":
        return g.drvg1(st["D"], cutint=CUTINT, exfac=case["exfac"], DS=st["DS"])
    prec = PRECISIONS[case["precision"]]
    if kind == "jk":
        return g.cho_jk(st["C"][0], precision=prec)
    if kind == "jkbatch":
        return g.cho_jk_batch(st["C"], precision=prec)
    st["F"].zero_()
    nvec = g.choscf_lk(st["D"], 0.5, st["F"], precision=prec)
    return st["F"], nvec


# -------------------------------------------------------------------- work
def _pair_table(m):
    """Per canonical shell pair: la, lb, contracted products, primitive pairs
    whose overlap factor is not negligible."""
    rows = []
    for i, a in enumerate(m.shells):
        for b in m.shells[:i + 1]:
            r2 = float(((a.center - b.center) ** 2).sum())
            mu = a.exps[:, None] * b.exps[None, :] / (a.exps[:, None] + b.exps[None, :])
            rows.append((a.l, b.l, a.ncontr * b.ncontr, max(1, int((mu * r2 < 41.0).sum()))))
    return np.array(rows)


def _cart(l):
    return (l + 1) * (l + 2) / 2


def _comp(l):
    return np.where(l >= 2, 2 * l + 1, _cart(l))


def _eri_work(P, Q):
    """(outputs, flops) summed over quartets of pair rows P x Q (Rys quadrature,
    contraction after [e0|f0], transfer and spherical transform per block)."""
    la, lb, nij, nab = P.T.astype(float)
    lc, ld, nkl, ncd = Q.T.astype(float)
    nef = [0.0, 0.0]
    for x, (l1, l2) in enumerate(((la, lb), (lc, ld))):
        lo, hi = np.maximum(l1, l2), l1 + l2
        nef[x] = (hi + 1) * (hi + 2) * (hi + 3) / 6 - lo * (lo + 1) * (lo + 2) / 6
    ne, nf = nef
    nr = np.floor((la + lb + lc + ld) / 2) + 1
    out = nij * nkl * _comp(la) * _comp(lb) * _comp(lc) * _comp(ld)
    prim = nab * ncd * (28 * nr + 30 + 12 * nr * (la + lb + 1) * (lc + ld + 1) + 3 * nr * ne * nf + 2 * nij * ne * nf)
    sab = _comp(la) * _comp(lb)
    block = 2 * nij * nkl * nf * (ncd * ne + sab * ne + sab * _comp(lc) * _comp(ld))
    return float(out.sum()), float((prim + block).sum())


def _grad_flops(rows):
    """Flops of the derivative integrals contracted with the two-particle
    density over the unique quartets (per primitive quartet: roots, 2D
    recursion and transfer, primitive density, 24 per component and root)."""
    keys, inv = np.unique(rows[:, :3], axis=0, return_inverse=True)
    prims = np.bincount(inv.ravel(), weights=rows[:, 3], minlength=len(keys))
    total = 0.0
    for (la, lb, nij), pa in zip(keys, prims):
        for (lc, ld, nkl), pc in zip(keys, prims):
            nr, nc4 = (la + lb + lc + ld + 3) // 2, _cart(la) * _cart(lb) * _cart(lc) * _cart(ld)
            n2d = (la + 1) * (lb + 1) * (lc + 1) * (ld + 1)
            per = 28 * nr + 30 + 3 * nr * (4 * (la + lb + 2) * (lc + ld + 2) + 12 * n2d) + 24 * nc4 * nr
            total += 0.5 * pa * pc * (per + (2 * nij * nc4 if nij * nkl > 1 else 0))
    return total


def _nvec(case, nbf):
    """Cholesky vectors to expect (two per function and decade of the threshold)."""
    return nbf * max(1.0, -2.0 * math.log10(case["thrcom"]) - 3.4)


def work(case):
    m = _base(case)
    n, rows = m.nbf, _pair_table(m)
    nrs = n * (n + 1) / 2
    if case["kind"] == "eri":
        q = _quartets(case, m).astype(np.int64)
        tri = lambda a, b: a * (a + 1) // 2 + b
        out, flops = _eri_work(rows[tri(q[:, 0], q[:, 1])], rows[tri(q[:, 2], q[:, 3])])
        return {"bytes": 8 * out + 24 * len(q), "flops": flops}
    if case["kind"] == "grad":
        return {"bytes": 8.0 * n * n * (2 if case["spin"] else 1) + 24 * m.natom, "flops": _grad_flops(rows)}
    M = _nvec(case, n)
    if case["kind"] == "cho":
        # subtraction of the previous vectors, and one column of integrals per vector
        P = rows[np.random.default_rng(4).integers(0, len(rows), 4000)]
        Q = rows[np.random.default_rng(5).integers(0, len(rows), 4000)]
        out, flops = _eri_work(P, Q)
        return {"bytes": 8.0 * nrs * M, "flops": nrs * M * M + flops / out * nrs * M}
    ranks = [max(1, case["rank"] - d) for d in range(case.get("ndens", 1))]
    flops = sum(3.0 * n * n * r * M + 4.0 * nrs * M for r in ranks)
    return {"bytes": 8.0 * nrs * M + 8.0 * sum(n * r + 2 * n * n for r in ranks), "flops": flops}


# ------------------------------------------- 64-bit values in plain numpy
# McMurchie-Davidson: every primitive pair is expanded in Hermite Gaussians,
# integrals are products of two expansions with the Hermite Coulomb integrals.
def _boys(mmax, T):
    """F_0..F_mmax (T: 1D): series and downward recursion, asymptotic above 40."""
    F = np.empty((mmax + 1,) + T.shape)
    small = np.minimum(T, 40.0)
    term = np.full_like(T, 1.0 / (2 * mmax + 1))
    acc = term.copy()
    for k in range(1, 220):
        term = term * (2.0 * small) / (2 * mmax + 2 * k + 1)
        acc += term
    ex = np.exp(-small)
    F[mmax] = ex * acc
    for k in range(mmax, 0, -1):
        F[k - 1] = (2.0 * small * F[k] + ex) / (2 * k - 1)
    big = T > 40.0
    if big.any():
        t = T[big]
        f = 0.5 * np.sqrt(math.pi / t)
        F[0, big] = f
        for k in range(mmax):
            f = (2 * k + 1) * f / (2 * t)
            F[k + 1, big] = f
    return F


def _hermite_1d(imax, jmax, a, b, ab):
    """E[i][j][t] (arrays over primitive pairs) of x_A^i x_B^j."""
    p = a + b
    XPA, XPB = -b / p * ab, a / p * ab
    E = {(0, 0): [np.exp(-a * b / p * ab * ab)]}

    def step(e, X):
        n = len(e)
        z = np.zeros_like(p)
        get = lambda t: e[t] if 0 <= t < n else z
        return [get(t - 1) / (2 * p) + X * get(t) + (t + 1) * get(t + 1) for t in range(n + 1)]

    for i in range(imax + 1):
        if i:
            E[i, 0] = step(E[i - 1, 0], XPA)
        for j in range(1, jmax + 1):
            E[i, j] = step(E[i, j - 1], XPB)
    return E


def _cart_list(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _sph(l):
    """Real spherical components (rows) over Cartesians, m = -l..l; s and p as they are."""
    if l < 2:
        return np.eye((l + 1) * (l + 2) // 2)
    poly = {2: [{(1, 1, 0): 1}, {(0, 1, 1): 1}, {(0, 0, 2): 2, (2, 0, 0): -1, (0, 2, 0): -1}, {(1, 0, 1): 1},
                {(2, 0, 0): 1, (0, 2, 0): -1}],
            3: [{(2, 1, 0): 3, (0, 3, 0): -1}, {(1, 1, 1): 1}, {(0, 1, 2): 4, (2, 1, 0): -1, (0, 3, 0): -1},
                {(0, 0, 3): 2, (2, 0, 1): -3, (0, 2, 1): -3}, {(1, 0, 2): 4, (3, 0, 0): -1, (1, 2, 0): -1},
                {(2, 0, 1): 1, (0, 2, 1): -1}, {(3, 0, 0): 1, (1, 2, 0): -3}]}[l]
    df = lambda k: math.prod(range(k - 1, 0, -2)) if k % 2 == 0 else 0
    carts = _cart_list(l)
    S = np.zeros((len(poly), len(carts)))
    for row, q in zip(S, poly):
        n2 = sum(u * v * math.prod(df(x + y) for x, y in zip(s, t)) for (s, u), (t, v) in
                 itertools.product(q.items(), q.items()))
        for s, u in q.items():
            row[carts.index(s)] = u / math.sqrt(n2)
    return S


def _tuv(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _expansion(a, b, L, da=None, db=None):
    """[primitive pair, (contracted pair, component pair), tuv] of shells a, b
    (first index of each pair fastest); da / db: derivative of a / b along that axis."""
    x, y = (v.ravel() for v in np.meshgrid(a.exps, b.exps, indexing="ij"))
    E = [_hermite_1d(a.l + 1, b.l + 1, x, y, a.center[d] - b.center[d]) for d in range(3)]
    tuv = _tuv(L)

    def prim(ca, cb):
        out = np.zeros((x.size, len(tuv)))
        if min(ca) < 0 or min(cb) < 0:
            return out
        e = [E[d][ca[d], cb[d]] for d in range(3)]
        for k, t in enumerate(tuv):
            if all(t[d] < len(e[d]) for d in range(3)):
                out[:, k] = e[0][t[0]] * e[1][t[1]] * e[2][t[2]]
        return out

    def deriv(ca, cb, which, axis, z):
        up, dn = [list(ca), list(cb)], [list(ca), list(cb)]
        up[which][axis] += 1
        dn[which][axis] -= 1
        return 2 * z[:, None] * prim(*map(tuple, up)) - (ca, cb)[which][axis] * prim(*map(tuple, dn))

    cart = np.empty((len(_cart_list(b.l)), len(_cart_list(a.l)), x.size, len(tuv)))
    for kb, cb in enumerate(_cart_list(b.l)):
        for ka, ca in enumerate(_cart_list(a.l)):
            cart[kb, ka] = deriv(ca, cb, 0, da, x) if da is not None else \
                deriv(ca, cb, 1, db, y) if db is not None else prim(ca, cb)
    sph = np.einsum("yb,xa,bapt->yxpt", _sph(b.l), _sph(a.l), cart)
    coef = np.einsum("xi,yj->xyji", a.coef, b.coef).reshape(x.size, b.ncontr, a.ncontr)
    out = np.einsum("pji,yxpt->pyxjit", coef, sph)
    return out.reshape(x.size, -1, len(tuv))


class _PairBlock:
    def __init__(self, a, b, order):
        x, y = (v.ravel() for v in np.meshgrid(a.exps, b.exps, indexing="ij"))
        self.L, self.zeta = a.l + b.l + order, x + y
        self.P = (x[:, None] * a.center + y[:, None] * b.center) / self.zeta[:, None]
        self.E = _expansion(a, b, self.L)
        self.dA = [_expansion(a, b, self.L, da=d) for d in range(3)] if order else None
        self.dB = [_expansion(a, b, self.L, db=d) for d in range(3)] if order else None


def _coulomb(p, q):
    """Hermite Coulomb integrals [bra prim, bra tuv, ket prim, ket tuv]."""
    L = p.L + q.L
    z, e = p.zeta[:, None], q.zeta[None, :]
    rho = (z * e / (z + e)).ravel()
    R = [(p.P[:, None, d] - q.P[None, :, d]).ravel() for d in range(3)]
    F = _boys(L, rho * (R[0] ** 2 + R[1] ** 2 + R[2] ** 2))
    pref = (2 * math.pi ** 2.5 / (z * e * np.sqrt(z + e))).ravel()
    H = {(0, 0, 0): [pref * (-2 * rho) ** n * F[n] for n in range(L + 1)]}
    for t in sorted(_tuv(L), key=sum)[1:]:
        d = next(k for k in range(3) if t[k])
        lo = tuple(t[k] - (k == d) for k in range(3))
        lo2 = tuple(t[k] - 2 * (k == d) for k in range(3))
        H[t] = [R[d] * H[lo][n + 1] + (lo[d] * H[lo2][n + 1] if lo[d] else 0.0) for n in range(L - sum(t) + 1)]
    A = np.empty((len(p.zeta), len(_tuv(p.L)), len(q.zeta), len(_tuv(q.L))))
    for i, s in enumerate(_tuv(p.L)):
        for j, t in enumerate(_tuv(q.L)):
            A[:, i, :, j] = ((-1) ** sum(t) * H[s[0] + t[0], s[1] + t[1], s[2] + t[2]][0]).reshape(A.shape[0], A.shape[2])
    return A


def _contract(Ep, A, Eq):
    h = np.tensordot(Ep.transpose(1, 0, 2), A, axes=([1, 2], [0, 1]))
    return np.tensordot(h, Eq.transpose(1, 0, 2), axes=([1, 2], [1, 2]))


def _exact_eri(case, seed):
    m = _molecule(case, seed)
    sh, blocks, out = m.shells, {}, []
    q = _quartets(case, m)
    pair = lambda i, j: blocks.setdefault((i, j), None) or blocks.__setitem__((i, j), _PairBlock(sh[i], sh[j], 0)) \
        or blocks[i, j]
    off = [0]
    for i, j, k, l in q.tolist():
        p, r = pair(i, j), pair(k, l)
        v = _contract(p.E, _coulomb(p, r), r.E)
        a, b, c, d = (sh[x] for x in (i, j, k, l))
        # bra (sb, sa, jb, ia) x ket (sd, sc, ld, kc) -> sd sc sb sa | l k j i, i fastest
        v = v.reshape(b.ncomp, a.ncomp, b.ncontr * a.ncontr, d.ncomp, c.ncomp, d.ncontr * c.ncontr)
        out.append(v.transpose(3, 4, 0, 1, 5, 2).ravel())
        off.append(off[-1] + out[-1].size)
    return torch.from_numpy(np.concatenate(out)), np.array(off, dtype=np.int64)


def _exact_grad(case, seed):
    m = _molecule(case, seed)
    sh = m.shells
    D, DS = _densities(case, seed, m.nbf)
    first = np.cumsum([0] + [s.nbf for s in sh])
    # (component, contracted) functions of a shell pair: (sb, sa, jb, ia)
    block = lambda M, x, y: M[first[x]:first[x + 1], first[y]:first[y + 1]].reshape(
        sh[x].ncomp, sh[x].ncontr, sh[y].ncomp, sh[y].ncontr)
    pairs = [(i, j) for i in range(len(sh)) for j in range(i + 1)]
    blocks = {p: _PairBlock(sh[p[0]], sh[p[1]], 1) for p in pairs}
    grad = np.zeros((m.natom, 3))
    for x, (i, j) in enumerate(pairs):
        for (k, l) in pairs[:x + 1]:
            at = [sh[s].atom for s in (i, j, k, l)]
            if len(set(at)) == 1:
                continue
            deg = (1 if i == j else 2) * (1 if k == l else 2) * (1 if (i, j) == (k, l) else 2)
            G = np.einsum("aibj,ckdl->baji" "dclk", block(D, i, j), block(D, k, l))
            for M in (D, DS):
                if M is not None:
                    for u, v in ((k, l), (l, k)):
                        s = ("aick,bjdl" if u == k else "aidl,bjck") + "->bajidclk"
                        G = G - 0.25 * case["exfac"] * np.einsum(s, block(M, i, u), block(M, j, v))
            p, r = blocks[i, j], blocks[k, l]
            A = _coulomb(p, r)
            nb = p.E.shape[1]
            ket = np.tensordot(A, r.E, axes=([2, 3], [0, 2]))          # [p, tuv, ket]
            W = np.tensordot(ket, G.reshape(nb, -1), axes=([2], [1]))  # [p, tuv, bra]
            bra = np.tensordot(p.E, G.reshape(nb, -1), axes=([1], [0]))  # [p, tuv, ket]
            V = np.tensordot(A, bra, axes=([0, 1], [0, 1]))            # [q, tuv, ket]
            for d in range(3):
                f = [float(np.einsum("pbt,ptb->", p.dA[d], W)), float(np.einsum("pbt,ptb->", p.dB[d], W)),
                     float(np.einsum("qkt,qtk->", r.dA[d], V))]
                f.append(-sum(f))
                for c in range(4):
                    grad[at[c], d] += 0.5 * deg * f[c]
    return torch.from_numpy(grad)


def exact(case, seed):
    """Integrals and forces of the smallest molecules in 64 bits.  None for the
    others: plain numpy would take minutes.  The vectors, and J, K and Fock
    matrices over them, have no value apart from the decomposition's own pivot
    choices."""
    if case["kind"] not in ("eri", "grad"):
        return None
    m = _base(case)
    ns = len(m.shells)
    npair = ns * (ns + 1) // 2
    nq = npair * (npair + 1) // 2
    if case["kind"] == "eri":
        if case["quartets"]:
            nq = min(nq, case["quartets"])
        return _exact_eri(case, seed) if nq <= 500 else None
    return _exact_grad(case, seed) if nq <= 500 else None
