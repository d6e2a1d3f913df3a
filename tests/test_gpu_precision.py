"""Results of quartets with tight and diffuse shells on centres far apart, where
a transfer of angular momentum between centres by differences cancels digits:
errors in units of the Schwarz bounds, against 50 digits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import helpers
import mp_integrals
from vlxb import basis, fock, lists
from vlxb._lib import lib

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53
CART = {l: [(l - s, s - z, z) for s in range(l + 1) for z in range(s + 1)] for l in range(4)}


def system(shells, alpha0, ratio, side, seed=5):
    """Two atoms `side` bohr apart, two primitives per shell, nothing screened."""
    lib().init(0)
    wl = basis.config_custom(2, max(side, 3.0), shells, 2, alpha0, ratio, 2, 1e-12, seed)
    wl.mol.coords[1] = wl.mol.coords[0] + side * np.array([0.48, 0.64, 0.6])
    return wl, lists.build_lists(wl.mol, wl.D, 0.0, helpers.oracle_schwarz_fn)


def prim(rl, l, idx):
    """(exponent, centre), exponents of a component, of a prim-cart index."""
    p, c = divmod(int(idx), len(CART[l]))
    info = rl.pd.info[l]
    return (info[0, p], tuple(info[2:5, p])), CART[l][c]


@pytest.mark.parametrize("alpha0,ratio,side", [(0.3, 2.5, 3.0), (0.05, 1000.0, 6.0), (0.1, 50.0, 2.0)])
def test_f_coulomb_keeps_its_digits(alpha0, ratio, side):
    """Three directions of at most 13 terms each, seven roots and one sum: 32
    roundings of the Schwarz bound per quartet leave room for all of them."""
    _, rl = system({0: 1, 3: 1}, alpha0, ratio, side)
    jl = rl.jlists["ff"]
    rng = np.random.default_rng(3)
    unlike = np.flatnonzero((jl.first // 10) % 2 != (jl.second // 10) % 2)  # a tight and a diffuse primitive
    pick = np.sort(np.concatenate([rng.choice(unlike, 5, replace=False), rng.choice(len(jl.first), 2, replace=False)]))
    for n in ("first", "second", "pdata", "Q", "D"):
        setattr(jl, n, np.ascontiguousarray(getattr(jl, n)[pick]))
    out = torch.zeros(len(pick), dtype=torch.float64, device="cuda")
    lib().coulomb("ffff", fock.coulomb_args(fock.to_device(rl), "ffff", out, torch.cuda.current_stream().cuda_stream))
    got = out.cpu().numpy()
    for e in range(len(pick)):
        exact, bound = mp_integrals.mp.mpf(0), 0.0
        for k in range(len(pick)):
            (A, a), (B, b) = prim(rl, 3, jl.first[e]), prim(rl, 3, jl.second[e])
            (C, c), (D, d) = prim(rl, 3, jl.first[k]), prim(rl, 3, jl.second[k])
            w = float(jl.D[k]) * (1.0 if jl.first[k] == jl.second[k] else 2.0)
            exact += float(jl.pdata[e]) * float(jl.pdata[k]) * w * mp_integrals.quartet([A, B, C, D])[0](a, b, c, d)
            bound += abs(w) * float(jl.Q[e]) * float(jl.Q[k])
        err = abs(float(exact - float(got[e])))
        assert bound > 0.0 and err <= 32 * EPS * bound, (e, got[e], err / (EPS * bound))


def thin(kp, per_row):
    """At most `per_row` seeded partners of every row of a partner list."""
    keep = []
    for i, (d, c) in enumerate(zip(kp.displs.astype(np.int64), kp.counts.astype(np.int64))):
        keep.append(np.sort(d + np.random.default_rng(i + 200).choice(c, min(per_row, c), replace=False)))
    kp.counts = np.array([len(k) for k in keep], dtype=kp.counts.dtype)
    kp.displs = np.concatenate([[0], np.cumsum(kp.counts[:-1].astype(np.int64))]).astype(kp.displs.dtype)
    for n in ("Dinds", "Q", "pdata"):
        setattr(kp, n, np.ascontiguousarray(getattr(kp, n)[np.concatenate(keep)]))


# limit: roundings of the bound, two to three times the largest of the same
# blocks by the Hermite recurrences (46, 4, 8 and 5)
@pytest.mark.parametrize("cls,alpha0,ratio,side,limit", [
    ("sdsd", 0.1, 50.0, 2.0, 128), ("dddd", 0.05, 1000.0, 6.0, 16), ("pddd", 0.05, 1000.0, 6.0, 24),
    ("dddd", 0.05, 2.5, 6.0, 16),
])
def test_exchange_gradient_keeps_its_digits(cls, alpha0, ratio, side, limit):
    """Blocks of one (i, k) entry and two partners a side; the bound of a
    derivative is the Schwarz bound of the raised and lowered functions."""
    from vlxb import gradient

    _, rl = system({0: 1, 1: 1, 2: 1}, alpha0, ratio, side)
    la, lb, lc, ld = (lists.LV[x] for x in cls)
    ac, kab, kcd = cls[0] + cls[2], rl.kpartners[cls[:2]], rl.kpartners[cls[2:]]
    thin(kab, 2)
    if kcd is not kab:
        thin(kcd, 2)
    dl = fock.to_device(rl)
    kq = rl.kpairs[ac]
    rows = np.random.default_rng(3).choice(len(kq.pair_i), 6, replace=False)
    ao = lambda l, idx: int(rl.pd.aoinds[l][int(idx) % len(CART[l]), int(idx) // len(CART[l])])  # noqa: E731
    root = lambda f, u, v: float(f(u, v, u, v)) ** 0.5  # noqa: E731
    worst = 0.0
    for r in rows:
        i, k = int(kq.pair_i[r]), int(kq.pair_k[r])
        dl.kpair[ac] = {n: torch.tensor([v], dtype=torch.int32, device="cuda") for n, v in (("i", i), ("k", k))}
        G = torch.zeros((6, 1), dtype=torch.float64, device="cuda")
        lib().exchange_grad(cls, gradient.kgrad_args(dl, cls, G, 0, 1, torch.cuda.current_stream().cuda_stream))
        got, exact, bound = G.cpu().numpy()[:, 0], [mp_integrals.mp.mpf(0)] * 6, np.zeros(6)
        wik = (1.0 if la == lc and i == k else 2.0) * rl.D_AO[ao(la, i), ao(lc, k)]
        for tj in range(int(kab.displs[i]), int(kab.displs[i]) + int(kab.counts[i])):
            for tl in range(int(kcd.displs[k]), int(kcd.displs[k]) + int(kcd.counts[k])):
                j, l = int(kab.Dinds[tj]), int(kcd.Dinds[tl])
                prims, comps = zip(prim(rl, la, i), prim(rl, lb, j), prim(rl, lc, k), prim(rl, ld, l))
                w = float(wik * rl.D_AO[ao(lb, j), ao(ld, l)] * kab.pdata[tj] * kcd.pdata[tl])
                grad = mp_integrals.quartet(prims)[1]
                for c in (0, 2):
                    f, o = (mp_integrals.quartet(prims[s:s + 2] * 2)[0] for s in (c, 2 - c))
                    other = root(o, *comps[2 - c:4 - c])
                    for x in range(3):
                        u = [tuple(v + s * (t == x) for t, v in enumerate(comps[c])) for s in (1, -1)]
                        s = 2.0 * float(prims[c][0]) * root(f, u[0], comps[c + 1])
                        if comps[c][x]:
                            s += comps[c][x] * root(f, u[1], comps[c + 1])
                        at = x if c == 0 else 3 + x
                        exact[at] += w * grad(c, x, *comps)
                        bound[at] += abs(w) * s * other
        for x in range(6):
            if bound[x] > 0.0:
                worst = max(worst, abs(float(exact[x] - float(got[x]))) / (EPS * bound[x]))
    assert 0.0 < worst <= limit, worst


@pytest.mark.parametrize("omega", [0.0, 0.4])
def test_exchange_gradient_per_component_path_on_either_centre(omega):
    """Records without a common S (the per-component path) whose pairs have a
    tighter shell on either centre, so that the recurrence is on b or d for some;
    FP64 bar of the suite, 1e-10 of the largest element."""
    from test_gpu_rys import close, system as rys_system
    from vlxb import gradient

    wl, rl = rys_system(2, 2, 2.0, 11, True)
    dl = fock.to_device(rl)
    g = gradient.ExchangeGradient(dl, wl.mol).compute(omega=omega).cpu().numpy()
    go, _ = helpers.oracle_exchange_gradient(rl, wl.mol.natoms, omega)
    assert float(np.abs(go).max()) > 1e-3 and close(g, go), float(np.abs(g - go).max())
