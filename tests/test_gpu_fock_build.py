"""The build call and the class entry points beside stream capture and beside
other streams' work."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")

import helpers
from vlxb import basis, fock, gradient, lists
from vlxb._lib import lib

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))

# class calls of the kernels that read the root tables, each with its output
CALLS = {
    "exchange": lambda L, dl, out, s: L.exchange("dddd", fock.exchange_args(dl, "dddd", out, s, 0.0)),
    "coulomb": lambda L, dl, out, s: L.coulomb("dddd", fock.coulomb_args(dl, "dddd", out, s)),
    "gradient": lambda L, dl, out, s: L.coulomb_grad("dddd", gradient.grad_args(dl, "dddd", out, 0, out.shape[1], s)),
    "fshell": lambda L, dl, out, s: L.coulomb("ffff", fock.coulomb_args(dl, "ffff", out, s)),
}


def system(atoms, shells, degree=1):
    lib().init(0)
    wl = basis.config_custom(atoms, 3.0, shells, degree, 0.4, 3.0, atoms, 1e-12, 3)
    return wl, fock.to_device(lists.build_lists(wl.mol, wl.D, wl.threshold, fock.gpu_schwarz_fn()))


def capture_first_call(name):
    """In a process of its own: vlxb_init, then the library's first launch under
    capture; its replay has the bits of an eager call."""
    L = lib()
    L.init(0)
    shells = {0: 1, 1: 1, 3: 1} if name == "fshell" else {0: 1, 1: 1, 2: 1}
    wl = basis.config_custom(2, 3.0, shells, 1, 0.4, 3.0, 2, 1e-12, 3)
    dl = fock.to_device(lists.build_lists(wl.mol, wl.D, wl.threshold, helpers.oracle_schwarz_fn))
    key = "ff" if name == "fshell" else "dd"
    n = (dl.kpair[key]["i"] if name == "exchange" else dl.j[key]["first"]).numel()
    shape = (6, n) if name == "gradient" else (n,)
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        CALLS[name](L, dl, out, torch.cuda.current_stream().cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    ref = torch.zeros_like(out)
    CALLS[name](L, dl, ref, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert float(ref.abs().max()) > 0.0 and torch.equal(out, ref)


@pytest.mark.parametrize("name", sorted(CALLS))
def test_first_call_after_init_can_be_captured(name):
    code = (f"import sys; sys.path[:0] = [{HERE!r}, {os.path.dirname(HERE)!r}, "
            f"{os.path.join(os.path.dirname(HERE), 'vlx-twoe-ints_b200')!r}]; "
            f"import test_gpu_fock_build as t; t.capture_first_call({name!r})")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_calls_on_two_streams_do_not_wait_for_each_other():
    """A small build whose stream still has a long kernel before it holds up no
    build of another stream (both run their classes on side streams)."""
    _, dl = system(2, {0: 1, 1: 1, 2: 1})
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    for s in (busy, other):  # first calls load kernels, which may wait for the device
        with torch.cuda.stream(s):
            ref = fock.build_jk(dl)
    torch.cuda.synchronize()
    end = torch.cuda.Event()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(2_000_000_000)  # a second, ends by itself
        end.record()
        late = fock.build_jk(dl)
    with torch.cuda.stream(other):
        first = fock.build_jk(dl)
    other.synchronize()
    waited = end.query()
    torch.cuda.synchronize()
    assert not waited
    for out in (late, first):
        for part, r in zip(out, ref):
            assert all(torch.equal(part[k], r[k]) for k in r)


def test_f_shell_calls_take_no_stream_that_others_may_be_using():
    """f-shell class calls run on side streams while another thread captures: a
    stream of torch's pool, which hands the same 32 to everyone, may be the one
    that is being captured."""
    import threading

    _, dl = system(2, {0: 1, 3: 1})
    ref = fock.build_jk(dl)
    torch.cuda.synchronize()
    captured, mine = torch.cuda.Stream(), torch.cuda.Stream()
    outs, errors = [], []

    def builds():
        try:
            with torch.cuda.stream(mine):
                for _ in range(10):  # at four streams a build, more than the pool has
                    outs.append(fock.build_jk(dl))
                mine.synchronize()
        except Exception as e:  # noqa: BLE001 (handed to the test's thread)
            errors.append(e)

    x = torch.ones(8, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=captured, capture_error_mode="thread_local"):
        y = x + 1.0
        t = threading.Thread(target=builds)
        t.start()
        t.join()
    assert not errors, errors
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, x + 1.0) and len(outs) == 10
    for out in outs:
        for part, r in zip(out, ref):
            assert all(torch.equal(part[k], r[k]) for k in r)


@pytest.mark.parametrize("what", ["build", "coulomb gradient", "exchange gradient"])
def test_fresh_outputs_are_zeroed_before_another_stream_adds_to_them(what):
    """Outputs made by the call are zeroed on the current stream, here a late
    one, and added to on the stream that is asked for."""
    wl, dl = system(2, {0: 1, 1: 1, 2: 1})
    side = torch.cuda.Stream()
    cg, kg = gradient.CoulombGradient(dl, wl.mol), gradient.ExchangeGradient(dl, wl.mol)

    def call(stream):
        if what == "build":
            J, K = fock.build_jk(dl, stream=stream)
            return [J[k] for k in sorted(J)] + [K[k] for k in sorted(K)]
        if what == "coulomb gradient":
            return [gradient.pair_gradients(dl, cg.map, stream=stream)]
        return [gradient.exchange_pair_gradients(dl, kg.map, stream=stream)]

    ref = call(torch.cuda.current_stream())
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda._sleep(400_000_000)
        out = call(side)
    torch.cuda.synchronize()
    assert any(float(r.abs().max()) > 0.0 for r in ref)
    assert all(torch.equal(a, b) for a, b in zip(out, ref))
