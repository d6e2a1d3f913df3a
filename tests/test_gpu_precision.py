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
