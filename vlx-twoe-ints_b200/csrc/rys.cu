// Host construction of the Rys root and weight tables (see rys.cuh).
#include <math.h>

#include <mutex>
#include <vector>

#include "engine.cuh"
#include "rys.cuh"

namespace vlxb {

namespace {

constexpr int NGL = 128;  // Gauss-Legendre points of the discretised inner product on t in [0, 1]

struct Legendre {
    long double x2[NGL], w[NGL];  // t^2 and weight
    Legendre()
    {
        const long double pi = acosl(-1.0L);
        for (int i = 0; i < NGL; i++) {
            long double z = cosl(pi * (i + 0.75L) / (NGL + 0.5L)), dp = 1.0L;
            for (int it = 0; it < 8; it++) {
                long double p0 = 1.0L, p1 = z;
                for (int k = 2; k <= NGL; k++) {
                    const long double p2 = ((2 * k - 1) * z * p1 - (k - 1) * p0) / k;
                    p0 = p1;
                    p1 = p2;
                }
                dp = NGL * (z * p1 - p0) / (z * z - 1.0L);
                z -= p1 / dp;
            }
            const long double t = 0.5L * (z + 1.0L);
            x2[i] = t * t;
            w[i] = 1.0L / ((1.0L - z * z) * dp * dp);
        }
    }
};

// Recurrence coefficients of the monic polynomials in x = t^2 orthogonal
// with weight exp(-T x): Stieltjes' procedure on the Legendre points.
void stieltjes(const Legendre& g, long double T, long double* al, long double* be)
{
    long double w[NGL], p[NGL], pm[NGL];
    for (int i = 0; i < NGL; i++) {
        w[i] = g.w[i] * expl(-T * g.x2[i]);
        p[i] = 1.0L;
        pm[i] = 0.0L;
    }
    long double prev = 1.0L;
    for (int k = 0; k < RYS_MAX; k++) {
        long double s0 = 0.0L, s1 = 0.0L;
        for (int i = 0; i < NGL; i++) {
            const long double v = w[i] * p[i] * p[i];
            s0 += v;
            s1 += v * g.x2[i];
        }
        al[k] = s1 / s0;
        be[k] = k ? s0 / prev : s0;
        prev = s0;
        for (int i = 0; i < NGL; i++) {
            const long double q = (g.x2[i] - al[k]) * p[i] - (k ? be[k] : 0.0L) * pm[i];
            pm[i] = p[i];
            p[i] = q;
        }
    }
}

long double monic(const long double* al, const long double* be, int n, long double x)
{
    long double q0 = 0.0L, q1 = 1.0L;
    for (int k = 0; k < n; k++) {
        const long double q2 = (x - al[k]) * q1 - (k ? be[k] : 0.0L) * q0;
        q0 = q1;
        q1 = q2;
    }
    return q1;
}

// Roots of every order up to RYS_MAX (those of order n separate those of
// order n + 1, so each bisection starts from a bracket) and the weights
// 1 / sum_k p_k(x)^2 / |p_k|^2.
void rules(const long double* al, const long double* be, long double x[][RYS_MAX], long double w[][RYS_MAX])
{
    for (int n = 1; n <= RYS_MAX; n++) {
        for (int r = 0; r < n; r++) {
            long double lo = r ? x[n - 1][r - 1] : 0.0L, hi = r < n - 1 ? x[n - 1][r] : 1.0L;
            const bool rising = (n - r) % 2 == 1;  // sign change at root r of a monic polynomial of degree n
            for (int it = 0; it < 90 && lo < hi; it++) {
                const long double mid = 0.5L * (lo + hi);
                if (mid <= lo || mid >= hi) break;
                if ((monic(al, be, n, mid) > 0.0L) == rising) hi = mid;
                else lo = mid;
            }
            const long double z = 0.5L * (lo + hi);
            long double q0 = 0.0L, q1 = 1.0L, nk = be[0], s = 0.0L;
            for (int k = 0; k < n; k++) {
                s += q1 * q1 / nk;
                const long double q2 = (z - al[k]) * q1 - (k ? be[k] : 0.0L) * q0;
                q0 = q1;
                q1 = q2;
                if (k + 1 < n) nk *= be[k + 1];
            }
            x[n][r] = z;
            w[n][r] = 1.0L / s;
        }
    }
}

}  // namespace

void rys_host_table(std::vector<double>& tab)
{
    const Legendre g;
    constexpr int NN = RYS_DEG + 1;
    const long double pi = acosl(-1.0L);
    tab.assign((size_t)rys_offset(RYS_MAX + 1), 0.0);
    long double al[RYS_MAX], be[RYS_MAX], x[RYS_MAX + 1][RYS_MAX], w[RYS_MAX + 1][RYS_MAX];
    const long double big = 110.0L;  // exp(-big) is far below one rounding: the half-range Hermite limit
    stieltjes(g, big, al, be);
    rules(al, be, x, w);
    for (int n = 1; n <= RYS_MAX; n++)
        for (int r = 0; r < n; r++) {
            tab[rys_offset(n) + 2 * r] = (double)(x[n][r] * big);
            tab[rys_offset(n) + 2 * r + 1] = (double)(w[n][r] * sqrtl(big));
        }
    // Chebyshev nodes of an interval, and the matrix from node values to
    // monomial coefficients in s in [-1, 1]
    long double node[NN], M[NN][NN];
    for (int i = 0; i < NN; i++) node[i] = cosl(pi * (i + 0.5L) / NN);
    for (int i = 0; i < NN; i++) {
        for (int m = 0; m < NN; m++) M[m][i] = 0.0L;
        long double t0[NN] = {1.0L}, t1[NN] = {0.0L, 1.0L};  // monomials of T_j and T_{j+1}
        for (int j = 0; j < NN; j++) {
            const long double c = (j ? 2.0L : 1.0L) / NN * cosl(j * pi * (i + 0.5L) / NN);
            for (int m = 0; m < NN; m++) M[m][i] += c * t0[m];
            long double t2[NN];
            for (int m = 0; m < NN; m++) t2[m] = (m ? 2.0L * t1[m - 1] : 0.0L) - t0[m];
            for (int m = 0; m < NN; m++) {
                t0[m] = t1[m];
                t1[m] = t2[m];
            }
        }
    }
    std::vector<long double> fx((size_t)NN * (RYS_MAX + 1) * RYS_MAX), fw(fx.size());
    for (int k = 0; k < rys_intervals(RYS_MAX); k++) {
        for (int i = 0; i < NN; i++) {
            stieltjes(g, ((long double)k + 0.5L + 0.5L * node[i]) * (long double)RYS_H, al, be);
            rules(al, be, x, w);
            for (int n = 1; n <= RYS_MAX; n++)
                for (int r = 0; r < n; r++) {
                    fx[((size_t)i * (RYS_MAX + 1) + n) * RYS_MAX + r] = x[n][r];
                    fw[((size_t)i * (RYS_MAX + 1) + n) * RYS_MAX + r] = w[n][r];
                }
        }
        for (int n = 1; n <= RYS_MAX; n++) {
            if (k >= rys_intervals(n)) continue;
            for (int m = 0; m < NN; m++)
                for (int r = 0; r < n; r++) {
                    long double sx = 0.0L, sw = 0.0L;
                    for (int i = 0; i < NN; i++) {
                        sx += M[m][i] * fx[((size_t)i * (RYS_MAX + 1) + n) * RYS_MAX + r];
                        sw += M[m][i] * fw[((size_t)i * (RYS_MAX + 1) + n) * RYS_MAX + r];
                    }
                    double* row = &tab[rys_offset(n) + 2 * n + ((size_t)k * NN + (NN - 1 - m)) * 2 * n + 2 * r];
                    row[0] = (double)sx;
                    row[1] = (double)sw;
                }
        }
    }
}

static std::mutex g_rys_mu;
static const double* g_rys_dev[64] = {nullptr};

const double* rys_table_device()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lk(g_rys_mu);
    if (g_rys_dev[dev]) return g_rys_dev[dev];
    static std::vector<double> host;
    if (host.empty()) rys_host_table(host);
    g_rys_dev[dev] = (const double*)upload_table(host.data(), host.size() * sizeof(double));
    return g_rys_dev[dev];
}

}  // namespace vlxb
