// J and K entry points of the classes with f shells.
//
// The reference's writer maps only p and d letters (eriwriter.py:44-62),
// although its ERI engine takes any number of Cartesian indices (eri.py:59
// labels angular momenta up to I); no f kernel is emitted.  These entry
// points are this library's own, with the argument conventions of the
// generated ones (gen_coulomb.py:74-93, gen_exchange.py:75-115) and the f
// components in the same order as d (x^3 first, then by decreasing y power:
// xxx, xxy, xxz, xyy, xyz, xzz, yyy, yyz, yzz, zzz).
//
// The s/p/d classes run generated straight-line shell-quartet code; doing
// the same for 170 f classes would multiply the library's size and build
// time.  The f classes run one generic kernel per kind instead, with the
// angular momenta as runtime arguments, at the reference's granularity: one
// Cartesian component quartet per work item, evaluated by Rys quadrature in
// registers (eri_component), rho' = rho for the Coulomb operator and
// rho w^2 / (rho + w^2) for the attenuated one.  Two atoms 1s1p1d1f (170 f class
// calls and the s/p/d ones): 209 ms with a Hermite box per component in local
// memory, 20.8 ms with a recurrence table per root and direction, 6.2 ms with
// the pairs' Hermite coefficients folded before the roots (eri_component).
// Screening is the reference's per-component predicate
// (|Q_ij Q_kl D_kl| > thr for J, |Q_ij Q_kl max_D| > thr for K), the J ket
// weights gen_coulomb.py:276-281, the K density gather gen_exchange.py:323.
// A CTA owns one output entry (J bra entry, K (i, k) entry); its threads
// stride over the kets / partner pairs and reduce in a fixed order, so
// results are bit-reproducible.  FP64 only; these classes are not counted
// by vlxb_quartetCounters.
#include "classes.cuh"
#include "md.cuh"
#include "rys.cuh"

namespace vlxb {

constexpr int FS_THREADS = 128;
constexpr int FS_WIDE = 512;                // threads per entry of lists too short to fill the device
constexpr int FS_LMAX = 3;                  // f
constexpr int FS_N = 2 * FS_LMAX + 1;     // 1-D Hermite coefficients of a pair: exponents 0..6
constexpr int FS_NR = RYS_MAX;            // roots of an (FF|FF) quartet

struct FPrim {
    double alpha, r[3];
    int c[3];  // Cartesian exponents of the component
};

// prim-cart index -> exponent, centre and component of a type-l primitive
// (prim_info [5][count]: row 0 exponent, rows 2..4 centre).
__device__ __forceinline__ FPrim fprim(const double* __restrict__ info, uint32_t count, int l, uint32_t idx)
{
    const int nc = ncart(l);
    const uint32_t p = idx / (uint32_t)nc;
    const int comp = (int)(idx % (uint32_t)nc);
    FPrim f;
    f.alpha = __ldg(info + p);
    f.r[0] = __ldg(info + p + 2 * (int64_t)count);
    f.r[1] = __ldg(info + p + 3 * (int64_t)count);
    f.r[2] = __ldg(info + p + 4 * (int64_t)count);
    const int yz = comp < 1 ? 0 : (comp < 3 ? 1 : (comp < 6 ? 2 : 3));  // y + z exponents (x^l first)
    f.c[2] = comp - yz * (yz + 1) / 2;
    f.c[1] = yz - f.c[2];
    f.c[0] = l - yz;
    return f;
}

// 1-D Hermite coefficients E^{ij}_t of one pair, t = 0..i + j (0 above), raised
// on the first centre, then on the second (md.cuh's recurrence; indices of
// arrays are constants throughout).
__device__ __forceinline__ void fs_hermite(int i, int j, double PA, double PB, double h, double* e)
{
#pragma unroll
    for (int t = 0; t < FS_N; t++) e[t] = t == 0 ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < FS_N - 1; k++) {
        if (k >= i + j) break;
        const double X = k < i ? PA : PB;
        double prev = 0.0;  // e[t - 1] before this step
#pragma unroll
        for (int t = 0; t <= k + 1; t++) {
            const double cur = e[t];
            double v = fma(h, prev, X * cur);
            if (t + 1 <= k) v = fma((double)(t + 1), e[t + 1], v);
            prev = cur;
            e[t] = v;
        }
    }
}

// (ab|cd) / (S_ab S_cd) of one Cartesian component quartet by Rys quadrature:
// per direction the integral at a root is sum_s G_s H_s, with the product of
// both pairs' Hermite coefficients G_{t+u} = sum E_t E'_u (-1)^u, which no root
// changes, and H_0 = 1, H_{s+1} = -2 rho x (PQ H_s + s H_{s-1}).  The pairs'
// centres enter through P - A and P - B as they are: a recurrence on A shifted
// to B by powers of A - B loses the digits of a tight b far from a diffuse a
// (5e-11 of the Schwarz bound, root mean square, for exponents 0.05 to 50 on
// two centres in a box of 6 bohr; this form 1.2e-16, a Hermite box 6e-16).
__device__ double eri_component(const FPrim& A, const FPrim& B, const FPrim& C, const FPrim& D, int nab, int ncd,
                                double omega, const double* __restrict__ rtab)
{
    const double p = A.alpha + B.alpha, q = C.alpha + D.alpha;
    const double ip = 1.0 / p, iq = 1.0 / q;
    const double rho = p * q / (p + q);
    const double d2 = omega != 0.0 ? omega * omega / (rho + omega * omega) : 1.0;
    const double rp = rho * d2;
    double PQ[3], r2 = 0.0;
#pragma unroll
    for (int x = 0; x < 3; x++) {
        PQ[x] = (A.r[x] - B.alpha * ip * (A.r[x] - B.r[x])) - (C.r[x] - D.alpha * iq * (C.r[x] - D.r[x]));
        r2 = fma(PQ[x], PQ[x], r2);
    }
    const int nr = (nab + ncd) / 2 + 1;
    double m2[FS_NR], prod[FS_NR];  // -2 rho x, and the product of the weight and the directions so far
#pragma unroll
    for (int r = 0; r < FS_NR; r++) {
        m2[r] = prod[r] = 0.0;
        if (r < nr) {
            rys_root_rt(nr, rp * r2, rtab, r, m2[r], prod[r]);
            m2[r] *= -2.0 * rp;
        }
    }
#pragma unroll
    for (int x = 0; x < 3; x++) {
        const double ab = A.r[x] - B.r[x], cd = C.r[x] - D.r[x];
        const int na = A.c[x] + B.c[x], nc = C.c[x] + D.c[x];
        double e[FS_N], f[FS_N], G[2 * FS_N - 1];
        fs_hermite(A.c[x], B.c[x], -B.alpha * ip * ab, A.alpha * ip * ab, 0.5 * ip, e);
        fs_hermite(C.c[x], D.c[x], -D.alpha * iq * cd, C.alpha * iq * cd, 0.5 * iq, f);
#pragma unroll
        for (int s = 0; s < 2 * FS_N - 1; s++) G[s] = 0.0;
#pragma unroll
        for (int u = 0; u < FS_N; u++) {
            if (u > nc) break;
            const double g = (u & 1) ? -f[u] : f[u];
#pragma unroll
            for (int t = 0; t < FS_N; t++)
                if (t <= na) G[t + u] = fma(e[t], g, G[t + u]);
        }
#pragma unroll
        for (int r = 0; r < FS_NR; r++) {
            if (r >= nr) break;
            double h = 1.0, h1 = m2[r] * PQ[x], s = G[0];  // H_{s-1}, H_s
#pragma unroll
            for (int n = 1; n < 2 * FS_N - 1; n++) {
                if (n > na + nc) break;
                s = fma(G[n], h1, s);
                const double h2 = m2[r] * fma(PQ[x], h1, n * h);
                h = h1;
                h1 = h2;
            }
            prod[r] *= s;
        }
    }
    double sum = 0.0;
#pragma unroll
    for (int r = 0; r < FS_NR; r++)
        if (r < nr) sum += prod[r];
    return 2.0 * sqrt(rp * INV_PI_D) * sum;
}

__device__ __forceinline__ double fs_block_sum(double v, double* red)
{
    v = warp_sum(v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += red[w];
    __syncthreads();
    return s;
}

struct FShellJ {
    int la, lb, lc, ld;
    const double* info[4];
    uint32_t count[4];
    const double *cd_D, *ab_Q, *cd_Q;
    const uint32_t *ab_first, *ab_second;
    const double* ab_pdata;
    uint32_t n_ab;
    const uint32_t *cd_first, *cd_second;
    const double* cd_pdata;
    uint32_t n_cd;
    double thr;
};

// 128 registers: four blocks of 128 threads per SM or one of 512 (the spills,
// 690 bytes here and 80 in the exchange kernel, are mostly the bra's
// coefficients, which no ket changes).
__global__ void __launch_bounds__(FS_WIDE, 1)
coulomb_fshell_kernel(FShellJ a, double* __restrict__ mat_J, const double* __restrict__ tab)
{
    __shared__ double red[FS_WIDE / 32];
    for (uint32_t ij = blockIdx.x; ij < a.n_ab; ij += gridDim.x) {
        const FPrim A = fprim(a.info[a.la], a.count[a.la], a.la, __ldg(a.ab_first + ij));
        const FPrim B = fprim(a.info[a.lb], a.count[a.lb], a.lb, __ldg(a.ab_second + ij));
        const double qij = __ldg(a.ab_Q + ij);
        double acc = 0.0;
        for (uint32_t kl = threadIdx.x; kl < a.n_cd; kl += blockDim.x) {
            const double dkl = __ldg(a.cd_D + kl);
            if (fabs(qij * __ldg(a.cd_Q + kl) * dkl) <= a.thr) continue;
            const uint32_t k = __ldg(a.cd_first + kl), l = __ldg(a.cd_second + kl);
            const FPrim C = fprim(a.info[a.lc], a.count[a.lc], a.lc, k);
            const FPrim D = fprim(a.info[a.ld], a.count[a.ld], a.ld, l);
            const double w = (a.lc != a.ld || k != l) ? 2.0 : 1.0;
            acc = fma(__ldg(a.cd_pdata + kl) * eri_component(A, B, C, D, a.la + a.lb, a.lc + a.ld, 0.0, tab), dkl * w, acc);
        }
        const double s = fs_block_sum(acc, red);
        if (threadIdx.x == 0) mat_J[ij] += __ldg(a.ab_pdata + ij) * s;
    }
}

struct FShellK {
    int la, lb, lc, ld;
    const uint32_t *pair_i, *pair_k;
    uint32_t n_ik;
    const double* info[4];
    const uint32_t* aoinds[4];
    uint32_t count[4];
    double maxD;
    const double* D;
    uint32_t naos;
    const double *Q_ab, *Q_cd;
    const uint32_t *Dinds_ab, *Dinds_cd, *displs_ab, *displs_cd, *counts_ab, *counts_cd;
    const double *pdata_ab, *pdata_cd;
    double omega, thr;
};

__global__ void __launch_bounds__(FS_WIDE, 1)
exchange_fshell_kernel(FShellK a, double* __restrict__ mat_K, const double* __restrict__ tab)
{
    __shared__ double red[FS_WIDE / 32];
    const int ncb = ncart(a.lb), ncd = ncart(a.ld);
    for (uint32_t ik = blockIdx.x; ik < a.n_ik; ik += gridDim.x) {
        const uint32_t i = __ldg(a.pair_i + ik), k = __ldg(a.pair_k + ik);
        const FPrim A = fprim(a.info[a.la], a.count[a.la], a.la, i);
        const FPrim C = fprim(a.info[a.lc], a.count[a.lc], a.lc, k);
        const uint32_t j0 = __ldg(a.displs_ab + i), nj = __ldg(a.counts_ab + i);
        const uint32_t l0 = __ldg(a.displs_cd + k), nl = __ldg(a.counts_cd + k);
        const uint64_t npair = (uint64_t)nj * nl;
        double acc = 0.0;
        for (uint64_t w = threadIdx.x; w < npair; w += blockDim.x) {
            const uint32_t pj = j0 + (uint32_t)(w / nl), pl = l0 + (uint32_t)(w % nl);
            if (fabs(__ldg(a.Q_ab + pj) * __ldg(a.Q_cd + pl) * a.maxD) <= a.thr) continue;
            const uint32_t jp = __ldg(a.Dinds_ab + pj), lp = __ldg(a.Dinds_cd + pl);
            const FPrim B = fprim(a.info[a.lb], a.count[a.lb], a.lb, jp);
            const FPrim D = fprim(a.info[a.ld], a.count[a.ld], a.ld, lp);
            const uint32_t jao = __ldg(a.aoinds[a.lb] + jp / (uint32_t)ncb + (int64_t)a.count[a.lb] * (jp % ncb));
            const uint32_t lao = __ldg(a.aoinds[a.ld] + lp / (uint32_t)ncd + (int64_t)a.count[a.ld] * (lp % ncd));
            const double eri = __ldg(a.pdata_ab + pj) * __ldg(a.pdata_cd + pl) * eri_component(A, B, C, D, a.la + a.lb, a.lc + a.ld, a.omega, tab);
            acc = fma(eri, __ldg(a.D + (int64_t)jao * a.naos + lao), acc);
        }
        const double s = fs_block_sum(acc, red);
        if (threadIdx.x == 0) mat_K[ik] += s;
    }
}

// Schwarz diagonal of primitive shell pairs with an f shell: the largest
// over components (a, b) of sqrt|(ab|ab)| / |S_ab| (vlxb_schwarzBareMax).
__global__ void __launch_bounds__(FS_THREADS)
schwarz_fshell_kernel(int la, int lb, const double* __restrict__ info_a, uint32_t cnt_a,
                      const double* __restrict__ info_b, uint32_t cnt_b, const uint32_t* __restrict__ P,
                      const uint32_t* __restrict__ Q, uint32_t n, double* __restrict__ out,
                      const double* __restrict__ tab)
{
    const int na = ncart(la), nb = ncart(lb);
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        double m = 0.0;
        for (int ca = 0; ca < na; ca++)
            for (int cb = 0; cb < nb; cb++) {
                const FPrim A = fprim(info_a, cnt_a, la, P[t] * (uint32_t)na + ca);
                const FPrim B = fprim(info_b, cnt_b, lb, Q[t] * (uint32_t)nb + cb);
                m = fmax(m, fabs(eri_component(A, B, A, B, la + lb, la + lb, 0.0, tab)));
            }
        out[t] = sqrt(m);
    }
}

// Pair prefactor S_PQ = c_P c_Q (pi / p)^(3/2) exp(-a b / p |A - B|^2) and
// Q_PQ = |S_PQ| sqrt(max bare diagonal) of pairs with an f shell
// (vlxb_shellPairData).
__global__ void __launch_bounds__(FS_THREADS)
shell_pair_fshell_kernel(int la, int lb, const double* __restrict__ info_a, uint32_t cnt_a,
                         const double* __restrict__ info_b, uint32_t cnt_b, const uint32_t* __restrict__ P,
                         const uint32_t* __restrict__ Q, uint32_t n, double* __restrict__ S_out,
                         double* __restrict__ q_out, const double* __restrict__ tab)
{
    const int na = ncart(la), nb = ncart(lb);
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const uint32_t i = P[t], j = Q[t];
        const FPrim A0 = fprim(info_a, cnt_a, la, i * (uint32_t)na);
        const FPrim B0 = fprim(info_b, cnt_b, lb, j * (uint32_t)nb);
        const double p = A0.alpha + B0.alpha, iz = 1.0 / p;
        double R2 = 0.0;
        for (int x = 0; x < 3; x++) R2 += (A0.r[x] - B0.r[x]) * (A0.r[x] - B0.r[x]);
        const double pi_p = 3.14159265358979323846 * iz;
        const double S = __ldg(info_a + i + (int64_t)cnt_a) * __ldg(info_b + j + (int64_t)cnt_b) * pi_p *
                         sqrt(pi_p) * exp(-A0.alpha * B0.alpha * iz * R2);
        double m = 0.0;
        for (int ca = 0; ca < na; ca++)
            for (int cb = 0; cb < nb; cb++) {
                const FPrim A = fprim(info_a, cnt_a, la, i * (uint32_t)na + ca);
                const FPrim B = fprim(info_b, cnt_b, lb, j * (uint32_t)nb + cb);
                m = fmax(m, fabs(eri_component(A, B, A, B, la + lb, la + lb, 0.0, tab)));
            }
        S_out[t] = S;
        q_out[t] = fabs(S) * sqrt(m);
    }
}

int run_shell_pair_f(int la, int lb, const double* info_a, uint32_t cnt_a, const double* info_b, uint32_t cnt_b,
                     const uint32_t* P, const uint32_t* Q, uint32_t n, double* S_out, double* q_out,
                     cudaStream_t st)
{
    const double* tab = rys_table_device();
    if (!tab) return VLXB_ECUDA;
    const uint32_t want = (n + FS_THREADS - 1) / FS_THREADS;
    const int grid = (int)(want < 148u * 64u ? want : 148u * 64u);
    shell_pair_fshell_kernel<<<grid, FS_THREADS, 0, st>>>(la, lb, info_a, cnt_a, info_b, cnt_b, P, Q, n, S_out, q_out,
                                                          tab);
    note_launches();
    VLXB_CHECK_CUDA(cudaGetLastError());
    return VLXB_OK;
}

int run_schwarz_f(int la, int lb, const double* info_a, uint32_t cnt_a, const double* info_b, uint32_t cnt_b,
                  const uint32_t* P, const uint32_t* Q, uint32_t n, double* out, cudaStream_t st)
{
    const double* tab = rys_table_device();
    if (!tab) return VLXB_ECUDA;
    const uint32_t want = (n + FS_THREADS - 1) / FS_THREADS;
    const int grid = (int)(want < 148u * 64u ? want : 148u * 64u);
    schwarz_fshell_kernel<<<grid, FS_THREADS, 0, st>>>(la, lb, info_a, cnt_a, info_b, cnt_b, P, Q, n, out, tab);
    note_launches();
    VLXB_CHECK_CUDA(cudaGetLastError());
    return VLXB_OK;
}

// Threads per output entry: with fewer entries than four blocks per SM the
// entry's partners are spread wider instead.
static int fs_threads(uint32_t entries) { return entries < 148u * 4u ? FS_WIDE : FS_THREADS; }

int run_coulomb_f(int la, int lb, int lc, int ld, const CoulombArgs& a, cudaStream_t st)
{
    if (a.n_ab == 0 || a.n_cd == 0) return VLXB_OK;
    if (!a.mat_J || !a.cd_D || !a.ab_Q || !a.cd_Q || !a.ab_first || !a.ab_second || !a.ab_pdata || !a.cd_first ||
        !a.cd_second || !a.cd_pdata)
        return VLXB_EINVAL;
    const int L4[4] = {la, lb, lc, ld};
    for (int t = 0; t < 4; t++)
        if (L4[t] < 0 || L4[t] > FS_LMAX || !a.info[L4[t]] || a.count[L4[t]] == 0) return VLXB_EINVAL;
    if (!(a.thr >= 0.0)) return VLXB_EINVAL;
    const double* tab = rys_table_device();
    if (!tab) return VLXB_ECUDA;
    FShellJ f{la, lb, lc, ld, {a.info[0], a.info[1], a.info[2], a.info[3]},
              {a.count[0], a.count[1], a.count[2], a.count[3]}, a.cd_D, a.ab_Q, a.cd_Q, a.ab_first, a.ab_second,
              a.ab_pdata, a.n_ab, a.cd_first, a.cd_second, a.cd_pdata, a.n_cd, a.thr};
    int grid = launch_grid_limit();
    if ((int64_t)grid > (int64_t)a.n_ab) grid = (int)a.n_ab;
    coulomb_fshell_kernel<<<grid, fs_threads(a.n_ab), 0, st>>>(f, a.mat_J, tab);
    note_launches();
    VLXB_CHECK_CUDA(cudaGetLastError());
    return VLXB_OK;
}

int run_exchange_f(int la, int lb, int lc, int ld, const ExchangeArgs& a, cudaStream_t st)
{
    if (a.n_ik == 0) return VLXB_OK;
    if (!a.mat_K || !a.pair_i || !a.pair_k || !a.D || !a.Q_ab || !a.Q_cd || !a.Dinds_ab || !a.Dinds_cd ||
        !a.displs_ab || !a.displs_cd || !a.counts_ab || !a.counts_cd || !a.pdata_ab || !a.pdata_cd || a.naos == 0)
        return VLXB_EINVAL;
    const int L4[4] = {la, lb, lc, ld};
    for (int t = 0; t < 4; t++)
        if (L4[t] < 0 || L4[t] > FS_LMAX || !a.info[L4[t]] || !a.aoinds[L4[t]] || a.count[L4[t]] == 0)
            return VLXB_EINVAL;
    if (!(a.thr >= 0.0) || !(a.omega >= 0.0)) return VLXB_EINVAL;
    const double* tab = rys_table_device();
    if (!tab) return VLXB_ECUDA;
    FShellK f{la, lb, lc, ld, a.pair_i, a.pair_k, a.n_ik, {a.info[0], a.info[1], a.info[2], a.info[3]},
              {a.aoinds[0], a.aoinds[1], a.aoinds[2], a.aoinds[3]}, {a.count[0], a.count[1], a.count[2], a.count[3]},
              a.maxD, a.D, a.naos, a.Q_ab, a.Q_cd, a.Dinds_ab, a.Dinds_cd, a.displs_ab, a.displs_cd, a.counts_ab,
              a.counts_cd, a.pdata_ab, a.pdata_cd, a.omega, a.thr};
    int grid = launch_grid_limit();
    if ((int64_t)grid > (int64_t)a.n_ik) grid = (int)a.n_ik;
    exchange_fshell_kernel<<<grid, fs_threads(a.n_ik), 0, st>>>(f, a.mat_K, tab);
    note_launches();
    VLXB_CHECK_CUDA(cudaGetLastError());
    return VLXB_OK;
}

}  // namespace vlxb
