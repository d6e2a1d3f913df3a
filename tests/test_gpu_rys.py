"""Rys quadrature kernels against the FP64 oracle where they can go wrong:
output blocks with fewer quartets than lanes and with a ragged last batch,
partner records without a common S or with only some components present (the
per-component path), very short and very long distances (both branches of the
root tables), and range separation."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import helpers
from vlxb import basis, fock, lists
from vlxb._lib import lib

pytestmark = pytest.mark.gpu
RTOL = 1e-10  # the suite's FP64 bar: 1e-10 of the largest element


def close(got, exp):
    return not exp.size or float(np.abs(got - exp).max()) <= RTOL * float(np.abs(exp).max()) + 1e-14


def system(atoms, degree, side, seed, uneven, threshold=1e-12):
    """Two shells per type; `uneven`: S and Q differ between the components of
    a pair (so a pair splits into records with partial component masks)."""
    lib().init(0)
    wl = basis.config_custom(atoms, max(side, 3.0), {0: 1, 1: 1, 2: 1}, degree, 0.4, 3.0, max(1, atoms), threshold, seed)
    if atoms == 2:  # a fixed separation: `side` bohr along one diagonal
        wl.mol.coords[1] = wl.mol.coords[0] + side / np.sqrt(3.0)
    rl = lists.build_lists(wl.mol, wl.D, wl.threshold, fock.gpu_schwarz_fn())
    if uneven:
        for key, kp in rl.kpartners.items():
            na, nb = lists.NCART[lists.LV[key[0]]], lists.NCART[lists.LV[key[1]]]
            first = np.repeat(np.arange(len(kp.counts)), kp.counts.astype(np.int64))
            c = (first % na) * nb + kp.Dinds.astype(np.int64) % nb
            kp.pdata = kp.pdata * (1.0 + 0.05 * c)
            kp.Q = kp.Q * np.where(c % 3 == 1, 0.5, 1.0)
            order = np.lexsort((-kp.Q, first))
            kp.Dinds, kp.Q, kp.pdata = kp.Dinds[order], kp.Q[order].copy(), kp.pdata[order].copy()
        for key, jl in rl.jlists.items():
            na, nb = lists.NCART[lists.LV[key[0]]], lists.NCART[lists.LV[key[1]]]
            c = (jl.first.astype(np.int64) % na) * nb + jl.second.astype(np.int64) % nb
            jl.pdata = jl.pdata * (1.0 + 0.05 * c)
            jl.Q = jl.Q * np.where(c % 3 == 1, 0.5, 1.0)
            order = np.argsort(-np.abs(jl.Q * jl.D), kind="stable")
            for n in ("first", "second", "pdata", "Q", "D"):
                setattr(jl, n, np.ascontiguousarray(getattr(jl, n)[order]))
    return wl, rl


@pytest.mark.parametrize("atoms,degree,side,uneven,omega", [
    (1, 1, 2.0, False, 0.0),    # one quartet per block
    (1, 1, 2.0, True, 0.4),
    (2, 2, 1.2, True, 0.0),
    (2, 2, 30.0, False, 0.0),   # T beyond every root table
    (3, 3, 4.0, False, 0.33),   # 81 quartets per block: a ragged last batch for every root count
])
def test_exchange_rys_vs_oracle(atoms, degree, side, uneven, omega):
    wl, rl = system(atoms, degree, side, 3 + atoms, uneven)
    dl = fock.to_device(rl)
    runs = []
    for _ in range(2):
        _, matK = fock.build_jk(dl, do_j=False, omega=omega)
        torch.cuda.synchronize()
        runs.append({k: v.cpu().numpy() for k, v in matK.items()})
    _, oK = helpers.oracle_jk_all(rl, omega=omega)
    for k in oK:
        assert np.array_equal(runs[0][k], runs[1][k]), k
        assert close(runs[0][k], oK[k]), (k, float(np.abs(runs[0][k] - oK[k]).max()), float(np.abs(oK[k]).max()))


@pytest.mark.parametrize("atoms,degree,side,uneven,omega", [
    (2, 1, 2.0, True, 0.4),
    (2, 2, 4.0, False, 0.0),
    (3, 1, 4.0, True, 0.0),
])
def test_exchange_gradient_rys_vs_oracle(atoms, degree, side, uneven, omega):
    from vlxb import gradient

    wl, rl = system(atoms, degree, side, 3 + atoms, uneven)
    dl = fock.to_device(rl)
    eg = gradient.ExchangeGradient(dl, wl.mol)
    g = eg.compute(omega=omega).cpu().numpy()
    assert np.array_equal(g, eg.compute(omega=omega).cpu().numpy())
    go, _ = helpers.oracle_exchange_gradient(rl, wl.mol.natoms, omega)
    assert close(g, go), float(np.abs(g - go).max())


@pytest.mark.parametrize("atoms,degree,side,uneven,threshold", [
    (1, 1, 2.0, False, 1e-12),   # one ket per bra
    (2, 2, 1.2, True, 1e-12),
    (2, 2, 30.0, False, 1e-12),  # T beyond every root table
    (2, 3, 3.0, False, 1e-4),    # kets with some components screened out
    (3, 2, 4.0, True, 1e-5),
])
def test_coulomb_rys_vs_oracle(atoms, degree, side, uneven, threshold):
    from vlxb import gradient

    wl, rl = system(atoms, degree, side, 3 + atoms, uneven, threshold)
    dl = fock.to_device(rl)
    runs = []
    for _ in range(2):
        matJ, _ = fock.build_jk(dl, do_k=False)
        torch.cuda.synchronize()
        runs.append({k: v.cpu().numpy() for k, v in matJ.items()})
    oJ, _ = helpers.oracle_jk_all(rl)
    for k in oJ:
        assert np.array_equal(runs[0][k], runs[1][k]), k
        assert close(runs[0][k], oJ[k]), (k, float(np.abs(runs[0][k] - oJ[k]).max()), float(np.abs(oJ[k]).max()))
    g = gradient.CoulombGradient(dl, wl.mol).compute().cpu().numpy()
    go, _ = helpers.oracle_coulomb_gradient(rl, wl.mol.natoms)
    assert close(g, go), float(np.abs(g - go).max())


@pytest.mark.parametrize("atoms,omega,cut", [(1, 0.0, 0.0), (3, 0.3, 0.0), (3, 0.0, 1e-6)])
def test_one_call_build_equals_class_calls(atoms, omega, cut):
    """vlxb_fockBuild against the 36 + 54 class calls on the same lists: the
    same kernels on the same preparations, so the same bits."""
    L = lib()
    wl, rl = system(atoms, 3, 4.0, 9, False)
    dl = fock.to_device(rl)
    s = torch.cuda.current_stream().cuda_stream
    try:
        L.set_fp32_cut(cut)
        matJ, matK = fock.build_jk(dl, omega=omega)
        refJ, refK = fock.alloc_outputs(dl)
        for cls in lists.j_classes():
            L.coulomb(cls, fock.coulomb_args(dl, cls, refJ[cls[:2]], s))
        for cls in lists.k_classes():
            L.exchange(cls, fock.exchange_args(dl, cls, refK[cls[0] + cls[2]], s, omega))
        torch.cuda.synchronize()
    finally:
        L.set_fp32_cut(0.0)
    for a, b in ((matJ, refJ), (matK, refK)):
        for k in b:
            assert torch.equal(a[k], b[k]), k


@pytest.mark.parametrize("prims", [511, 512, 513, 700])
def test_long_partner_segments(prims):
    """Partner segments around the length of one tile of the segment sort: an
    s-only system of `prims` primitives on one list, a few (i, k) rows, the
    partner lists given in reverse order (the engine sorts them)."""
    L = lib()
    L.init(0)
    atoms = 7
    wl = basis.config_custom(atoms, 9.0, {0: 1}, 100, 0.02, 1.08, 3, 1e-12, 4)
    rl = lists.build_lists(wl.mol, wl.D, wl.threshold, fock.gpu_schwarz_fn())
    n = rl.pd.count[0]
    keep = np.arange(n) < prims
    kp = rl.kpartners["ss"]
    first = np.repeat(np.arange(n), kp.counts.astype(np.int64))
    m = keep[first] & keep[kp.Dinds.astype(np.int64)]
    kp.Dinds, kp.Q, kp.pdata, first = kp.Dinds[m], kp.Q[m], kp.pdata[m], first[m]
    kp.counts = np.bincount(first, minlength=n).astype(np.uint32)
    kp.displs = np.concatenate([[0], np.cumsum(kp.counts[:-1].astype(np.int64))]).astype(np.uint32)
    kq = rl.kpairs["ss"]
    rows = np.flatnonzero(keep[kq.pair_i.astype(np.int64)] & keep[kq.pair_k.astype(np.int64)])[::60000][:4]
    kq.pair_i, kq.pair_k = kq.pair_i[rows].copy(), kq.pair_k[rows].copy()
    exp = helpers.oracle_K(rl, "ssss")
    for name in ("Dinds", "Q", "pdata"):
        v = getattr(kp, name)
        setattr(kp, name, np.concatenate([v[d:d + c][::-1] for d, c in zip(kp.displs.astype(np.int64),
                                                                          kp.counts.astype(np.int64))]))
    dl = fock.to_device(rl)
    out = torch.zeros(len(rows), dtype=torch.float64, device="cuda")
    L.exchange("ssss", fock.exchange_args(dl, "ssss", out, torch.cuda.current_stream().cuda_stream, 0.0))
    torch.cuda.synchronize()
    assert int(kp.counts.max()) > 256 and close(out.cpu().numpy(), exp), (out.cpu().numpy(), exp)


def test_quartet_counts_do_not_depend_on_precision():
    """Every screened-in quartet is evaluated once, in FP64 or in FP32."""
    L = lib()
    wl, rl = system(3, 3, 4.0, 9, False)
    dl = fock.to_device(rl)
    counts = []
    try:
        for cut in (0.0, 1e-6, 1e30):
            L.set_fp32_cut(cut)
            L.reset_counters()
            fock.build_jk(dl)
            torch.cuda.synchronize()
            counts.append(L.quartet_counters())
    finally:
        L.set_fp32_cut(0.0)
    assert counts[0] == counts[1] == counts[2], counts


@pytest.mark.parametrize("prims", [63, 64, 65, 181, 182])
def test_short_scans(prims):
    """Occupancy tables around one round (64 x 64 entries) and around the bound
    (182 x 182 is above it) of the one-block scan: s primitives on one centre,
    sparse J and (i, k) lists that hold the first and the last pair."""
    L = lib()
    L.init(0)
    wl = basis.config_custom(1, 3.0, {0: 1}, prims, 0.02, 1.08, 1, 1e-12, 4)
    rl = lists.build_lists(wl.mol, wl.D, 0.0, fock.gpu_schwarz_fn())
    last = prims - 1
    jl, kq = rl.jlists["ss"], rl.kpairs["ss"]
    f, g = jl.first.astype(np.int64), jl.second.astype(np.int64)
    pick = np.flatnonzero((f * 7 + g) % 61 == 3)
    pick = np.unique(np.concatenate([pick, np.flatnonzero((f == 0) & (g == 0)), np.flatnonzero((f == last) & (g == last))]))
    for n in ("first", "second", "pdata", "Q", "D"):
        setattr(jl, n, np.ascontiguousarray(getattr(jl, n)[pick]))
    i, k = kq.pair_i.astype(np.int64), kq.pair_k.astype(np.int64)
    rows = np.flatnonzero(((i == 0) & (k == 0)) | ((i == last) & (k == last)) | ((i == 1) & (k == last)))
    kq.pair_i, kq.pair_k = kq.pair_i[rows].copy(), kq.pair_k[rows].copy()
    expJ, expK = helpers.oracle_J(rl, "ssss"), helpers.oracle_K(rl, "ssss")
    dl = fock.to_device(rl)
    matJ, matK = fock.build_jk(dl)
    torch.cuda.synchronize()
    assert len(rows) == 3 and len(pick) > 30
    assert close(matJ["ss"].cpu().numpy(), expJ), (matJ["ss"], expJ)
    assert close(matK["ss"].cpu().numpy(), expK), (matK["ss"], expK)


@pytest.mark.parametrize("kets", [1, 33, 511, 513, 4096, 4097])
def test_short_ket_sorts(kets):
    """Ket lists around the tile and the bound of the rank sort, in a shuffled
    order (the engine sorts them): seeded bra rows of (ss|ss)."""
    L = lib()
    L.init(0)
    wl = basis.config_custom(1, 3.0, {0: 1}, 100, 0.02, 1.08, 1, 1e-12, 4)
    rl = lists.build_lists(wl.mol, wl.D, 0.0, fock.gpu_schwarz_fn())
    rng = np.random.default_rng(kets)
    jl = rl.jlists["ss"]  # by descending |Q D|
    names = ("first", "second", "pdata", "Q", "D")
    pick = np.sort(rng.permutation(len(jl.first))[:kets])
    for n in names:
        setattr(jl, n, np.ascontiguousarray(getattr(jl, n)[pick]))
    rl.threshold = 0.5 * float(np.median(np.abs(jl.Q * jl.D)) * np.median(jl.Q))  # screens out some of the kets
    rows = rng.permutation(kets)[:5]
    exp = helpers.oracle_J(rl, "ssss", rows=rows)[rows]
    order = rng.permutation(kets)
    for n in names:
        setattr(jl, n, np.ascontiguousarray(getattr(jl, n)[order]))
    matJ, _ = fock.build_jk(fock.to_device(rl), do_k=False)
    got = np.empty(kets)
    got[order] = matJ["ss"].cpu().numpy()
    assert np.abs(exp).max() > 0.0 and close(got[rows], exp), (got[rows], exp)
