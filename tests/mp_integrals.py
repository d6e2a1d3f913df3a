"""Component integrals of primitive Cartesian Gaussians to 50 digits (mpmath),
by the Obara-Saika recurrences, without the pair prefactors S_ab S_cd: the
reference of the precision tests, whose quartets cancel digits that a reference
in 64 bits would lose too."""
import mpmath as mp

from oracle import oracle


def quartet(prims, omega=0.0):
    """(bare, grad): functions of four exponent triples (ax, ay, az), ... for
    four primitives (alpha, centre): the integral, and its derivative on a
    centre's coordinate (of the integral with the pair prefactors, divided by
    them)."""
    with mp.workdps(50):
        al = [mp.mpf(float(a)) for a, _ in prims]
        R = [[mp.mpf(float(x)) for x in r] for _, r in prims]
        p, q = al[0] + al[1], al[2] + al[3]
        rho = p * q / (p + q)
        d2 = mp.mpf(omega) ** 2 / (rho + mp.mpf(omega) ** 2) if omega else mp.mpf(1)
        P = [(al[0] * x + al[1] * y) / p for x, y in zip(R[0], R[1])]
        Q = [(al[2] * x + al[3] * y) / q for x, y in zip(R[2], R[3])]
        T = rho * d2 * sum((x - y) ** 2 for x, y in zip(P, Q))
        F = oracle.boys_mpmath(16, T, 50)
        s = 2 * mp.sqrt(rho * d2 / mp.pi)
        base = [s * f * d2 ** m for m, f in enumerate(F)]
    memo = {}

    def vrr(n, m, k):  # [n|m]^(k) on the first centres
        if min(n) < 0 or min(m) < 0:
            return mp.mpf(0)
        if not sum(n) + sum(m):
            return base[k]
        key = (n, m, k)
        if key in memo:
            return memo[key]
        side = 0 if sum(n) else 1
        v = n if side == 0 else m
        x = max(i for i in range(3) if v[i])
        lo = tuple(c - (i == x) for i, c in enumerate(v))
        lo2 = tuple(c - 2 * (i == x) for i, c in enumerate(v))
        z, e, X, W = (p, q, P, R[0]) if side == 0 else (q, p, Q, R[2])
        g = (lambda a, kk: vrr(a, m, kk)) if side == 0 else (lambda a, kk: vrr(n, a, kk))
        r = (X[x] - W[x]) * g(lo, k) + e / (p + q) * ((Q[x] - P[x]) if side == 0 else (P[x] - Q[x])) * g(lo, k + 1)
        if lo[x]:
            r += lo[x] / (2 * z) * (g(lo2, k) - e / (p + q) * g(lo2, k + 1))
        w = m if side == 0 else n
        if w[x]:
            dn = tuple(c - (i == x) for i, c in enumerate(w))
            r += w[x] / (2 * (p + q)) * (vrr(lo, dn, k + 1) if side == 0 else vrr(dn, lo, k + 1))
        memo[key] = r
        return r

    def hrr(a, b, c, d):
        if min(min(v) for v in (a, b, c, d)) < 0:
            return mp.mpf(0)
        for x in range(3):
            if d[x]:
                dn = tuple(v - (i == x) for i, v in enumerate(d))
                return hrr(a, b, tuple(v + (i == x) for i, v in enumerate(c)), dn) + (R[2][x] - R[3][x]) * hrr(a, b, c, dn)
        for x in range(3):
            if b[x]:
                dn = tuple(v - (i == x) for i, v in enumerate(b))
                return hrr(tuple(v + (i == x) for i, v in enumerate(a)), dn, c, d) + (R[0][x] - R[1][x]) * hrr(a, dn, c, d)
        return vrr(a, c, 0)

    def bare(a, b, c, d):
        with mp.workdps(50):
            return hrr(a, b, c, d)

    def grad(centre, x, *comps):
        with mp.workdps(50):
            up, dn = list(comps), list(comps)
            up[centre] = tuple(v + (i == x) for i, v in enumerate(comps[centre]))
            dn[centre] = tuple(v - (i == x) for i, v in enumerate(comps[centre]))
            r = 2 * al[centre] * hrr(*up)
            return r - comps[centre][x] * hrr(*dn) if comps[centre][x] else r

    return bare, grad
