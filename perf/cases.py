"""The calls that a program built on this framework spends its time in, for measuring them.

Every case is a molecule of contracted Cartesian shells (the even-tempered
synthetic recipe of `vlxb.basis`, seeded), its density and one public call
sequence:

  build     resident lists -> 36 + 54 class calls -> AO J, K and the energy: one SCF iteration
  exchange  the exchange class calls only, range-separated operator (omega > 0), AO K
  fresh     a new geometry: device list build, AO map, class calls, AO J, K and the energy
  delta     an incremental iteration: density difference into the resident lists, class calls,
            AO contraction, update of the running J and K, the energy
  batch     several small molecules, one class call per class for all of them, in a CUDA graph
  gradj     nuclear gradient of the Coulomb energy
  gradk     nuclear gradient of the exchange energy

`cut` > 0 lets quartets below that bound run in single precision, inside the
library's default error budget.  Sizes: `atoms` at `volume` bohr^3 each, `s`,
`p`, `d`, `f` contracted shells per atom of `degree` primitives with
exponents alpha0 * ratio^k.
"""
import itertools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "vlx-twoe-ints_b200"))

from vlxb import aomap, basis, batchfuse, devlists, fock, gradient  # noqa: E402
from vlxb._lib import lib  # noqa: E402
from vlxb.tune import apply_schedule  # noqa: E402

TRIPLE = {"s": 4, "p": 3, "d": 2, "f": 0, "degree": 3, "alpha0": 0.05, "ratio": 2.5}  # the benchmark's 4s3p2d shells
SMALL = {"s": 3, "p": 2, "d": 0, "f": 0, "degree": 3, "alpha0": 0.1, "ratio": 3.0}    # the 3s2p shells of small runs
TINY = {"s": 1, "p": 1, "d": 1, "f": 0, "degree": 2, "alpha0": 0.3, "ratio": 2.5}     # the smoke run's shells


def _case(kind, atoms, shells, volume=30.0, threshold=1e-12, omega=0.0, cut=0.0, mols=1, name=None):
    c = {"kind": kind, "atoms": atoms, "volume": volume, "threshold": threshold, "omega": omega, "cut": cut,
         "mols": mols, **shells}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: two atoms, every class present, bound by launches and host work
        _case("build", 2, TINY, volume=13.5, name="build 2 atoms 1s1p1d"),
        # a small molecule without polarisation functions (5 atoms, 45 AOs)
        _case("build", 5, SMALL, volume=43.2, name="build 5 atoms 3s2p"),
        # a diatomic in the polarised basis: many classes, little work in each
        _case("build", 2, TRIPLE, name="build 2 atoms 4s3p2d"),
        # one step of a geometry optimisation or a new request to a server: nothing resident yet
        _case("fresh", 5, TRIPLE, name="fresh 5 atoms 4s3p2d"),
        # the largest: one iteration on 14 atoms, 350 AOs
        _case("build", 14, TRIPLE, name="build 14 atoms 4s3p2d"),
        # the same kind of iteration with single precision below a bound
        _case("build", 8, TRIPLE, cut=1e-6, name="mixed 8 atoms 4s3p2d"),
        # long-range exchange of a range-separated hybrid functional
        _case("exchange", 6, TRIPLE, omega=0.33, name="exchange 6 atoms omega"),
        # a late SCF iteration: the density difference screens most of the work away
        _case("delta", 9, TRIPLE, volume=25.0, threshold=1e-11, name="delta 9 atoms 4s3p2d"),
        # a screening run over small molecules (3 to 5 atoms)
        _case("batch", 4, TRIPLE, mols=6, name="batch 6 molecules"),
        # forces: Coulomb and exchange part
        _case("gradj", 6, TRIPLE, name="gradj 6 atoms 4s3p2d"),
        _case("gradk", 5, TRIPLE, name="gradk 5 atoms 4s3p2d"),
        # f functions: 100 + 160 classes on a diatomic
        _case("build", 2, {**TINY, "f": 1}, volume=13.5, name="build 2 atoms 1s1p1d1f"),
    ]


def draw(rng):
    """One more case: the kinds by use, atoms over the logarithm of each kind's range, shells and primitives varied."""
    kind, lo, hi = rng.choice([("build", 2, 9), ("build", 2, 9), ("build", 3, 11), ("mixed", 3, 8), ("exchange", 2, 7),
                               ("fresh", 2, 8), ("delta", 3, 9), ("batch", 3, 5), ("gradj", 2, 7), ("gradk", 2, 4),
                               ("f", 1, 2)])
    atoms = min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))
    shells = dict(rng.choice([TRIPLE, TRIPLE, SMALL]))
    shells["s"] = rng.randint(1, shells["s"])
    shells["p"] = rng.randint(1, shells["p"])
    shells["d"] = rng.randint(0, 2)
    shells["degree"] = rng.choice([1, 2, 3, 3, 3])
    volume = round(rng.uniform(20.0, 45.0), 2)
    if kind == "f":
        return _case("build", atoms, {**TINY, "f": 1, "degree": rng.randint(1, 2)}, volume=round(rng.uniform(10, 30), 2))
    if kind == "mixed":
        return _case("build", atoms, shells, volume, cut=1e-6)
    if kind == "exchange":
        return _case("exchange", atoms, shells, volume, omega=round(rng.uniform(0.1, 0.5), 3))
    if kind == "delta":
        return _case("delta", atoms, shells, volume, threshold=1e-11)
    if kind == "batch":
        return _case("batch", atoms, shells, volume, mols=rng.randint(2, 7))
    return _case(kind, atoms, shells, volume)


# ------------------------------------------------------------------ inputs

def _molecule(case, atoms, seed):
    """Geometry, shells and density of one molecule."""
    side = (atoms * case["volume"]) ** (1.0 / 3.0)
    recipe = {l: case[x] for l, x in enumerate("spdf") if case[x]}
    wl = basis.config_custom(atoms, max(side, 2.0), recipe, case["degree"], case["alpha0"], case["ratio"], 2 * atoms,
                             case["threshold"], seed)
    return wl.mol, wl.D


def _difference(mol, seed):
    """A density difference of a late iteration: symmetric, of Frobenius norm 1e-3."""
    P = np.random.default_rng(seed + 77).standard_normal((mol.naos, mol.naos))
    P = P + P.T
    return P * (1e-3 / np.linalg.norm(P))


def prepare(case, seed):
    L = lib()
    L.init(0)
    apply_schedule()
    kind, thr = case["kind"], case["threshold"]
    st = {"kind": kind, "cut": case["cut"], "omega": case["omega"], "threshold": thr, "L": L}
    if kind == "batch":
        mols = [_molecule(case, case["atoms"] - 1 + m % 3, 1000 * seed + m) for m in range(case["mols"])]
        st["fused"] = batchfuse.FusedBatch([m for m, _ in mols], [D for _, D in mols], thr)
        st["maps"] = [aomap.AOMap(rl) for rl in st["fused"].rls]
        st["fused"].capture()
        return st
    mol, D = _molecule(case, case["atoms"], seed)
    st["mol"], st["D"] = mol, torch.from_numpy(np.ascontiguousarray(D)).cuda()
    if kind == "fresh":
        return st
    st["dl"] = devlists.build_device_lists(mol, st["D"].clone(), thr)
    if kind == "gradj":
        st["grad"] = gradient.CoulombGradient(st["dl"], mol)
    elif kind == "gradk":
        st["grad"] = gradient.ExchangeGradient(st["dl"], mol)
    else:
        st["map"] = aomap.AOMap.from_device(st["dl"])
        st["flatJ"], st["matJ"], st["flatK"], st["matK"] = st["map"].alloc_outputs()
        if kind == "delta":
            st["dD"] = torch.from_numpy(_difference(mol, seed)).cuda()
            g = torch.Generator(device="cuda").manual_seed(seed)
            st["J"], st["K"] = (torch.randn(st["D"].shape, dtype=torch.float64, device="cuda", generator=g)
                                for _ in range(2))
    return st


# ------------------------------------------------------------------ the calls

def _matrices(st, dl, am, flatJ, matJ, flatK, matK):
    flatJ.zero_()
    flatK.zero_()
    if st["cut"] > 0.0:
        st["L"].set_fp32_cut(st["cut"])
    try:
        fock.build_jk(dl, matJ=matJ, matK=matK)
    finally:
        if st["cut"] > 0.0:
            st["L"].set_fp32_cut(0.0)
    return am.to_ao("J", flatJ), am.to_ao("K", flatK)


def run(st):
    kind = st["kind"]
    if kind == "batch":
        fb, out = st["fused"], []
        fb.run()
        for m, am in enumerate(st["maps"]):  # each molecule's AO matrices from its slices of the outputs
            flatJ = torch.cat([fb.matJ[k][slice(*fb.jslices[k][m])] for k in am.J.keys])
            flatK = torch.cat([fb.matK[k][slice(*fb.kslices[k][m])] for k in am.K.keys])
            out.append({"J": am.to_ao("J", flatJ), "K": am.to_ao("K", flatK)})
        return out
    if kind in ("gradj", "gradk"):
        return st["grad"].compute()
    if kind == "exchange":
        st["flatK"].zero_()
        fock.build_jk(st["dl"], omega=st["omega"], matJ=st["matJ"], matK=st["matK"], do_j=False)
        return {"K": st["map"].to_ao("K", st["flatK"])}
    if kind == "fresh":
        dl = devlists.build_device_lists(st["mol"], st["D"], st["threshold"])
        am = aomap.AOMap.from_device(dl)
        J, K = _matrices(st, dl, am, *am.alloc_outputs())
        return {"J": J, "K": K, "E": aomap.energy(st["D"], J, K)}
    outputs = (st["flatJ"], st["matJ"], st["flatK"], st["matK"])
    if kind == "delta":
        devlists.set_density(st["dl"], st["dD"])
        dJ, dK = _matrices(st, st["dl"], st["map"], *outputs)
        J, K = st["J"] + dJ, st["K"] + dK
        return {"dJ": dJ, "dK": dK, "J": J, "K": K, "E": aomap.energy(st["D"], J, K)}
    J, K = _matrices(st, st["dl"], st["map"], *outputs)
    return {"J": J, "K": K, "E": aomap.energy(st["D"], J, K)}


# ------------------------------------------------------------------ work

def _nh(l):
    return (l + 1) * (l + 2) * (l + 3) // 6


def _nc(l):
    return (l + 1) * (l + 2) // 2


def work(case):
    """Bytes: shell data and density in, results out.  Operations, before screening: per primitive shell quartet the
    Hermite integrals and their contraction with both sides (Coulomb), one multiply-add per component quartet and
    quadrature root (exchange); a gradient needs six sums of that kind."""
    n = {l: case["atoms"] * case[x] * case["degree"] for l, x in enumerate("spdf") if case[x]}
    do_j = case["kind"] not in ("exchange", "gradk")
    do_k = case["kind"] != "gradj"
    grad = 1 if case["kind"] in ("gradj", "gradk") else 0
    pairs = {(a, b): n[a] * (n[a] + 1) // 2 if a == b else n[a] * n[b] for a in n for b in n if a <= b}
    flops = 0.0
    for (a, b), nab in pairs.items():
        if do_j:
            for (c, d), ncd in pairs.items():
                flops += nab * ncd * 2.0 * (2 * _nh(a + b + c + d + grad) + _nh(a + b + grad) * _nh(c + d))
        if do_k:
            for c, d in itertools.product(n, n):  # here (a, b) is the output pair, (c, d) the summed shells
                L = a + b + c + d + grad
                flops += nab * n[c] * n[d] * 2.0 * _nc(a) * _nc(b) * _nc(c) * _nc(d) * (L // 2 + 1) * (6 if grad else 1)
    naos = case["atoms"] * sum(case[x] * _nc(l) for l, x in enumerate("spdf"))
    prim_cart = {l: n[l] * _nc(l) for l in n}
    entries = sum(prim_cart[a] * prim_cart[b] for a in n for b in n if a <= b)
    return {"bytes": case["mols"] * 8.0 * (3 * naos * naos + 2 * entries), "flops": case["mols"] * flops}


# ------------------------------------------------------------------ the same results in 64 bits, plainly

def _boys(L, T):
    """F_0..F_L: the power series of F_L and downward recursion below T = 40, the asymptotic F_0 and upward above."""
    lo = T.clamp(max=40.0)
    term = torch.full_like(T, 1.0 / (2 * L + 1))
    tot = term.clone()
    for k in range(1, 180):
        term = term * (2.0 * lo / (2 * L + 2 * k + 1))
        tot = tot + term
    ex = torch.exp(-lo)
    F = [None] * (L + 1)
    F[L] = ex * tot
    for m in range(L - 1, -1, -1):
        F[m] = (2.0 * lo * F[m + 1] + ex) / (2 * m + 1)
    big = T.clamp(min=40.0)
    G = [0.5 * torch.sqrt(math.pi / big)]
    for m in range(L):
        G.append(((2 * m + 1) * G[m] - torch.exp(-big)) / (2.0 * big))
    return [torch.where(T < 40.0, f, g) for f, g in zip(F, G)]


def _hermite(la, lb, a, b, X):
    """E[i][j][t] of one direction, without the exponential prefactor; X = A - B."""
    p, one, zero = a + b, torch.ones_like(X), torch.zeros_like(X)
    PA, PB = -b / p * X, a / p * X
    E = {(0, 0, 0): one}
    g = lambda i, j, t: E.get((i, j, t), zero)  # noqa: E731
    for i in range(la + 1):
        for j in range(lb + 1):
            if i + j == 0:
                continue
            for t in range(i + j + 1):
                u, v, S = (i - 1, j, PA) if i else (i, j - 1, PB)
                E[i, j, t] = g(u, v, t - 1) / (2 * p) + S * g(u, v, t) + (t + 1) * g(u, v, t + 1)
    return E


class _Pairs:
    """All ordered primitive pairs of two contracted shell types: E coefficients per Cartesian component pair."""

    def __init__(self, prims, la, lb, comps_a, comps_b, factor_a=None):
        A, B = prims[la[1]], prims[lb[1]]
        na, nb = len(A["e"]), len(B["e"])
        self.i = torch.arange(na, device="cuda").repeat_interleave(nb)
        self.j = torch.arange(nb, device="cuda").repeat(na)
        a, b = A["e"][self.i], B["e"][self.j]
        RA, RB = A["R"][self.i], B["R"][self.j]
        self.p = a + b
        self.P = (a[:, None] * RA + b[:, None] * RB) / self.p[:, None]
        self.L = la[0] + lb[0]
        K = torch.exp(-a * b / self.p * (RA - RB).square().sum(1)) * A["c"][self.i] * B["c"][self.j]
        if factor_a is not None:
            K = K * factor_a(a)
        E = [_hermite(la[0], lb[0], a, b, RA[:, x] - RB[:, x]) for x in range(3)]
        self.tuv = [(t, u, v) for t in range(self.L + 1) for u in range(self.L + 1 - t)
                    for v in range(self.L + 1 - t - u)]
        z = torch.zeros_like(K)
        self.H = torch.stack([torch.stack([torch.stack([
            K * E[0].get((x[0], y[0], t), z) * E[1].get((x[1], y[1], u), z) * E[2].get((x[2], y[2], v), z)
            for (t, u, v) in self.tuv], -1) for y in comps_b], 1) for x in comps_a], 1)  # [pair][a][b][tuv]


def _integrals(bra, ket, omega):
    """[bra pair][ket pair][a][b][c][d], in blocks of bra pairs: yields (first pair, block)."""
    L = bra.L + ket.L
    nk = len(ket.p)
    step = max(1, 150000 // max(1, nk) if L > 4 else 600000 // max(1, nk))
    sign = torch.tensor([(-1.0) ** sum(t) for t in ket.tuv], dtype=torch.float64, device="cuda")
    for s in range(0, len(bra.p), step):
        p, q = bra.p[s:s + step, None], ket.p[None, :]
        d = bra.P[s:s + step, None, :] - ket.P[None, :, :]
        rho = p * q / (p + q)
        pre = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
        if omega > 0.0:
            f = omega * omega / (rho + omega * omega)
            pre, rho = pre * torch.sqrt(f), rho * f
        F = _boys(L, rho * d.square().sum(-1))
        R = {(0, 0, 0, m): pre * (-2.0 * rho) ** m * F[m] for m in range(L + 1)}
        for n in range(1, L + 1):
            for t in range(n + 1):
                for u in range(n - t + 1):
                    v = n - t - u
                    x = 0 if t else (1 if u else 2)
                    lo = [t, u, v]
                    lo[x] -= 1
                    lo2 = list(lo)
                    lo2[x] -= 1
                    for m in range(L - n + 1):
                        r = d[..., x] * R[(*lo, m + 1)]
                        if lo[x] > 0:
                            r = r + lo[x] * R[(*lo2, m + 1)]
                        R[t, u, v, m] = r
            for k in [k for k in R if sum(k[:3]) == n - 2 and k[3] > 0]:
                del R[k]
        M = torch.stack([torch.stack([R[e[0] + f[0], e[1] + f[1], e[2] + f[2], 0] for f in ket.tuv], -1)
                         for e in bra.tuv], -2)  # [bra][ket][e][f]
        half = torch.einsum("pabe,pqef->pqabf", bra.H[s:s + step], M * sign)
        yield s, torch.einsum("pqabf,qcdf->pqabcd", half, ket.H)


def _prims(mol):
    out = {}
    for l in sorted({sh.l for sh in mol.shells}):
        row = [(e, c, mol.coords[sh.atom], sh.ao0, sh.atom) for sh in mol.shells if sh.l == l
               for e, c in zip(sh.exps, sh.coefs)]
        t = lambda k: torch.tensor(np.array([r[k] for r in row]), device="cuda")  # noqa: E731
        out[l] = {"e": t(0), "c": t(1), "R": t(2), "ao": t(3), "atom": t(4)}
    return out


def _ao(prims, l, idx):
    return prims[l]["ao"][idx][:, None] + torch.arange(_nc(l), device="cuda")


def _fold(out, blk, ia, ib, jc, jd, n):
    """out[a, b, c, d] += block, by AO index."""
    k = ((ia[:, None, :, None, None, None] * n + ib[:, None, None, :, None, None]) * n
         + jc[None, :, None, None, :, None]) * n + jd[None, :, None, None, None, :]
    out.index_add_(0, k.reshape(-1), blk.reshape(-1))


def _ao_integrals(mol, omega):
    """The AO integrals (ab|cd), [n, n, n, n]."""
    prims, n = _prims(mol), mol.naos
    G = torch.zeros(n ** 4, dtype=torch.float64, device="cuda")
    ls = sorted(prims)
    pairs = {(a, b): _Pairs(prims, (a, a), (b, b), basis.CART[a], basis.CART[b]) for a in ls for b in ls if a <= b}
    keys = sorted(pairs)
    for x, ab in enumerate(keys):
        for cd in keys[x:]:
            bra, ket = pairs[ab], pairs[cd]
            for s, blk in _integrals(bra, ket, omega):
                e = s + blk.shape[0]
                _fold(G, blk, _ao(prims, ab[0], bra.i[s:e]), _ao(prims, ab[1], bra.j[s:e]), _ao(prims, cd[0], ket.i),
                      _ao(prims, cd[1], ket.j), n)
    G = G.view(n, n, n, n)
    l_of = torch.empty(n, dtype=torch.int64, device="cuda")
    for sh in mol.shells:
        l_of[sh.ao0:sh.ao0 + _nc(sh.l)] = sh.l
    # blocks of the pairs that were left out, by symmetry: a > b, c > d, then bra after ket
    up = l_of[:, None] <= l_of[None, :]
    G = torch.where(up[:, :, None, None], G, G.transpose(0, 1))
    G = torch.where(up[None, None], G, G.transpose(2, 3))
    lo, hi = torch.minimum(l_of[:, None], l_of[None]), torch.maximum(l_of[:, None], l_of[None])
    code = lo * 4 + hi
    return torch.where(code[:, :, None, None] <= code[None, None], G, G.permute(2, 3, 0, 1))


def _gradient(mol, D, exchange):
    """d/dR of half of Tr[D J] or Tr[D K]: four times the derivative of the first function's centre."""
    prims = _prims(mol)
    g = torch.zeros((mol.natoms, 3), dtype=torch.float64, device="cuda")
    ls = sorted(prims)
    kets = {(c, d): _Pairs(prims, (c, c), (d, d), basis.CART[c], basis.CART[d]) for c in ls for d in ls}
    for a, b in itertools.product(ls, ls):
        for x in range(3):
            up = [tuple(v + (k == x) for k, v in enumerate(w)) for w in basis.CART[a]]
            dn = [tuple(v - (k == x) for k, v in enumerate(w)) for w in basis.CART[a]]
            bra = _Pairs(prims, (a + 1, a), (b, b), up, basis.CART[b], lambda e: 2.0 * e)
            if a:  # the lowered functions share the raised ones' Hermite space
                low = _Pairs(prims, (a - 1, a), (b, b), [w if min(w) >= 0 else (0, 0, 0) for w in dn], basis.CART[b])
                for k, w in enumerate(basis.CART[a]):
                    for t, h in enumerate(low.tuv):
                        bra.H[:, k, :, bra.tuv.index(h)] -= w[x] * low.H[:, k, :, t]
            for (c, d), ket in kets.items():
                jc, jd = _ao(prims, c, ket.i), _ao(prims, d, ket.j)
                for s, blk in _integrals(bra, ket, 0.0):
                    e = s + blk.shape[0]
                    ia, ib = _ao(prims, a, bra.i[s:e]), _ao(prims, b, bra.j[s:e])
                    if exchange:
                        w1 = D[ia[:, None, :, None], jc[None, :, None, :]]
                        w2 = D[ib[:, None, :, None], jd[None, :, None, :]]
                        v = torch.einsum("pqabcd,pqac,pqbd->p", blk, w1, w2)
                    else:
                        w1 = D[ia[:, :, None], ib[:, None, :]]
                        w2 = D[jc[:, :, None], jd[:, None, :]]
                        v = torch.einsum("pqabcd,pab,qcd->p", blk, w1, w2)
                    g[:, x].index_add_(0, prims[a]["atom"][bra.i[s:e]], 2.0 * v)
    return g


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return None
    per_atom = {l: case[x] * case["degree"] for l, x in enumerate("spdf")}
    quartets = (case["atoms"] * sum(per_atom.values())) ** 4
    naos = case["atoms"] * sum(case[x] * _nc(l) for l, x in enumerate("spdf"))
    heavy = case["d"] or case["f"]
    if quartets > (1.0e7 if heavy else 4.0e7) or naos > 80 or (kind in ("gradj", "gradk") and quartets > 1.0e6):
        return None
    mol, D = _molecule(case, case["atoms"], seed)
    D = torch.from_numpy(np.ascontiguousarray(D)).cuda()
    if kind in ("gradj", "gradk"):
        return _gradient(mol, D, kind == "gradk")
    G = _ao_integrals(mol, case["omega"])
    if kind == "exchange":
        return {"K": torch.einsum("abcd,bd->ac", G, D)}
    use = torch.from_numpy(_difference(mol, seed)).cuda() if kind == "delta" else D
    J = torch.einsum("abcd,cd->ab", G, use)
    K = torch.einsum("abcd,bd->ac", G, use)
    if kind == "delta":
        g = torch.Generator(device="cuda").manual_seed(seed)
        J0, K0 = (torch.randn(D.shape, dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
        out = {"dJ": J, "dK": K, "J": J0 + J, "K": K0 + K}
        J, K = out["J"], out["K"]
    else:
        out = {"J": J, "K": K}
    dj, dk = (D * J).sum(), (D * K).sum()
    return {**out, "E": torch.stack([dj - 0.5 * dk, dj, dk])}
