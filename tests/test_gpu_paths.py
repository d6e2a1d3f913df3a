"""Paths that no default call of the other tests takes: the kernels of a mixed
build's FP32 quartets with every quartet in FP32, the library sort of very long
partner segments, and the class calls that stand in for the one-call build."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import helpers
from vlxb import basis, fock, lists
from vlxb._lib import lib
from vlxb.batchfuse import FusedBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree,omega,threshold", [(1, 0.0, 1e-12), (3, 0.3, 1e-12), (3, 0.0, 1e-5)])
def test_every_exchange_class_in_fp32(degree, omega, threshold):
    """A cutoff above every bound, no error budget: each class's FP32 kernel
    (thread per quartet, column, packed column, contracted partners) evaluates
    all of its quartets.  FP32 carries 6e-8 a rounding; two hundred of them of
    the largest element, where a misplaced component would be of its order."""
    L = lib()
    L.init(0)
    wl = basis.config_custom(3, 4.0, {0: 2, 1: 1, 2: 1}, degree, 0.2, 2.5, 3, threshold, 17)
    rl = lists.build_lists(wl.mol, wl.D, wl.threshold, fock.gpu_schwarz_fn())
    dl = fock.to_device(rl)
    s = torch.cuda.current_stream().cuda_stream
    budget, bad, differ = L.get_fp32_budget(), [], 0
    try:
        L.set_fp32_cut(1e30)
        L.set_fp32_budget(0.0)
        for cls in lists.k_classes():
            out = torch.zeros(dl.kpair[cls[0] + cls[2]]["i"].numel(), dtype=torch.float64, device="cuda")
            L.exchange(cls, fock.exchange_args(dl, cls, out, s, omega))
            got, exp = out.cpu().numpy(), helpers.oracle_K(rl, cls, omega)
            scale = float(np.abs(exp).max())
            err = float(np.abs(got - exp).max())
            differ += err > 1e-13 * scale
            if err > 1.2e-5 * scale + 1e-14:
                bad.append((cls, err / scale))
    finally:
        L.set_fp32_cut(0.0)
        L.set_fp32_budget(budget)
    assert not bad and differ == len(lists.k_classes()), (bad, differ)


@pytest.mark.parametrize("prims", [455, 456])
def test_partner_segments_around_the_library_sort(prims):
    """Dense bounds of a partner segment below and above the 16384 records from
    which it is sorted by the library: d primitives on one centre with seven
    partner shells each, a few (i, k) rows, the lists in reverse order."""
    L = lib()
    L.init(0)
    wl = basis.config_custom(1, 3.0, {2: 1}, prims, 0.05, 1.01, 1, 1e-12, 4)
    pd = lists.prim_data(wl.mol)
    rng = np.random.default_rng(prims)
    partner = np.stack([np.sort(rng.choice(prims, 7, replace=False)) for _ in range(prims)])
    P, Q = np.repeat(np.arange(prims), 7), partner.reshape(-1)
    e, c = pd.info[2][0], pd.info[2][1]
    S = c[P] * c[Q] * (np.pi / (e[P] + e[Q])) ** 1.5
    q = np.abs(S) * fock.gpu_schwarz_fn()(2, 2, pd, np.minimum(P, Q), np.maximum(P, Q))
    order = np.argsort(-q.reshape(prims, 7), axis=1, kind="stable")
    sort = lambda a: np.take_along_axis(a.reshape(prims, 7), order, 1)  # noqa: E731
    expand = lambda a: np.repeat(np.repeat(a, 6, axis=1), 6, axis=0).reshape(-1)  # noqa: E731 (6 rows, 6 components)
    dinds = expand(sort(partner) * 6) + np.tile(np.arange(6), prims * 42)
    n = prims * 6
    kp = lists.KPartners((np.arange(n) * 42).astype(np.uint32), np.full(n, 42, dtype=np.uint32),
                         dinds.astype(np.uint32), expand(sort(q)), expand(sort(S)))
    kq = lists.KPairs(np.array([0, 1, n // 2, n - 1], dtype=np.uint32),
                      np.array([0, n - 1, n // 2 + 3, n - 1], dtype=np.uint32))
    rl = lists.ReferenceLists(pd, wl.mol.naos, wl.D, 1e-12, kpartners={"dd": kp}, kpairs={"dd": kq},
                              maxD={"dd": float(np.abs(wl.D).max())})
    exp = helpers.oracle_K(rl, "dddd")
    for name in ("Dinds", "Q", "pdata"):
        setattr(kp, name, np.ascontiguousarray(getattr(kp, name).reshape(n, 42)[:, ::-1].reshape(-1)))
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    dl = fock.to_device(rl)
    L.exchange("dddd", fock.exchange_args(dl, "dddd", out, torch.cuda.current_stream().cuda_stream, 0.0))
    got = out.cpu().numpy()
    assert np.abs(exp).max() > 0.0 and np.abs(got - exp).max() <= 1e-10 * np.abs(exp).max(), (got, exp)


@pytest.mark.parametrize("cut", [0.0, 1e-6])
def test_class_calls_of_a_batch_and_of_a_molecule(cut, monkeypatch):
    """What runs where the one-call build does not fit in memory has its bits."""
    L = lib()
    L.init(0)
    wls = [basis.config_custom(2 + t, 4.0, {0: 2, 1: 1, 2: 1}, 2, 0.2, 2.5, 2, 1e-12, 5 + t) for t in range(2)]
    dl = fock.to_device(lists.build_lists(wls[1].mol, wls[1].D, wls[1].threshold, fock.gpu_schwarz_fn()))
    fb = FusedBatch([w.mol for w in wls], [w.D for w in wls], 1e-12)
    runs = []
    try:
        L.set_fp32_cut(cut)
        for one_call in (True, False):
            if not one_call:
                monkeypatch.setattr(fb.L, "fock_build", lambda *a: False)
            fb.run()
            J, K = fock.build_jk(dl)
            torch.cuda.synchronize()
            runs.append([{k: v.clone() for k, v in d.items()} for d in (fb.matJ, fb.matK, J, K)])
    finally:
        L.set_fp32_cut(0.0)
    for a, b in zip(*runs):
        assert a and all(torch.equal(a[k], b[k]) and float(b[k].abs().max()) > 0.0 for k in b)
