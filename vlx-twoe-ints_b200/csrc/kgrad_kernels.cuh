// Exchange nuclear gradient by Rys quadrature (sm_100a).
//
// E_K = 1/2 Tr[D K] = 1/2 sum_{ijkl} D_ik D_jl (ij|kl) over all primitive
// Cartesian indices.  The sum is unchanged by (i <-> j, k <-> l) and by
// (ij) <-> (kl), so the derivatives on the centres of j and l equal those on
// i and k, and over the caller's (i, k) list (gen_exchange.py:139-342: i of
// type a, k of type c, i <= k for a == c)
//   dE_K/dR = sum_{(i,k) in list} w_ik D_ik sum_{jl} D_jl (d/dA + d/dC)(ij|kl),
// w_ik = 1 for i == k of a same-type list, else 2, d/dA acting on i's centre
// (credited to i's atom), d/dC on k's (credited to k's atom).  A Cartesian
// Gaussian differentiates as d/dA_x phi_a = 2 alpha phi_{a+1x} - a_x phi_{a-1x}
// (Obara-Saika 1986, Eq. 5; the reference generator's gradient='a' / 'c'
// terms, eri.py:85-152).
//
// One lane evaluates one root of one quartet (krys_kernels.cuh).  At a root
// the energy is E = sum Gam_abcd Ix Iy Iz with Gam = Dw_ac D_bd S_ab S_cd
// (Dw_ac = w_ik D_ik), so all six derivatives come from one reverse sweep:
// with the sensitivities  Xb(c, d) = dE / dIx(ax, bx; c, d)  of one (a, b),
//   gA_x += sum_cd Xb(c, d) (2 alpha I(ax + 1, bx; c, d) - ax I(ax - 1, ...))
//   gC_x += sum_cd Xb(c, d) (2 gamma I(ax, bx; c + 1, d) - c I(ax, bx; c - 1, d)).
// The sweep costs 24 multiply-adds per (a, b, c) for a d shell d (8 for the
// energy alone), against 6 x 2 per component and root for separate sums.
// Loops over b and a are not unrolled; the 27 sensitivities of one (a, b), the
// 1-D integrals and the six sums are all that a lane keeps in registers.  The
// VRR table in shared memory has one more row and column than the energy's.
// Bound: FP64 issue and the latency of dependent multiply-adds, with eight warps
// per SM (255 registers; seven for two d-d pairs): FP64 pipe 42 to 50 % busy, the
// shared-memory pipe 27 to 52 %.  5 atoms 4s3p2d, all 54 classes: 741 ms with the
// Hermite-table kernel it replaces (shared-memory bound at 91 %), 54.5 ms now.
//
// Layout follows the exchange kernels: one CTA per (i, k) primitive shell
// block, fixed-order reduction, no atomics on the output.  Screening is the K
// kernels' (|Q_ij Q_kl max_D| > thr), FP64.  The block's six values are added
// at the block's lowest (i, k) list position p, grad[x * gstride + p] (x = 0..2:
// i's centre, 3..5: k's); the block's other positions receive nothing (all of
// them share the two atoms).
#pragma once
#include "krys_kernels.cuh"

namespace vlxb {

template <int LA, int LB, int LC, int LD>
struct KGradShape {
    static constexpr int L = LA + LB + LC + LD;
    static constexpr int NR = (L + 1) / 2 + 1;
    static constexpr int QW = 32 / NR;
    // quartets set up together: as many as one pass takes, for shared memory's sake
    // (full batches up to L = 4: 4 atoms 4s3p2d, 3.9 and 5.9 ms for the classes of
    // L = 3 and 4 against 4.0 and 5.7); below L = 3 either way the same
    static constexpr int BATCH = L >= 3 ? QW : 32 / QW * QW;
    static constexpr int N1 = LA + LB + 2, M1 = LC + LD + 2;
    // two CTAs of four warps (255 registers); the tables of two d-d pairs leave
    // room for seven warps, taken as one CTA
    static constexpr int NW = N1 * M1 >= 36 ? 7 : 4;
    static constexpr int THREADS = NW * 32, MINB = NW == 7 ? 1 : (L >= 5 ? 2 : 3);
    static constexpr int SMEM = 3 * N1 * M1 * THREADS * 8;
};

// Shifts between the centres of a pair.  The recurrence is on the centre of the
// tighter shell: the exponent `near` on it and `far` on the other centre are
// sum_k binomial(far, k) R^(far - k) V(near + k), R = near centre - far centre,
// whose terms do not cancel as P is nearer to the near centre.  From a diffuse a
// to a tight b two shifts cancel: blocks of (SD|SD), exponents 0.1 and 5 at 2
// bohr, were 304 roundings off in units of the bound where the Hermite tables
// before were 16 (as here).  One shift costs no more than P - B = (P - A) + (A -
// B) does anyway ((PP|PP): 8 either way), so s and p shells b (d) keep a (c).
// 5 atoms 4s3p2d: 55 -> 59 ms.
//
// v[m], m < NM, for the exponents a and b; `swap`: the recurrence is on b.
template <int LA, int LB, int M1, int NM, int TH>
__device__ __forceinline__ void kgrad_shift(const double* V, bool swap, int a, int b, double R, double* v)
{
    // lanes of a warp mostly agree in `swap`: their quartets share the bra's record
    const int near = LB > 1 && swap ? b : a, far = LB > 1 && swap ? a : b;
    const double* p = V + near * M1 * TH;
    if (LB == 0 || far == 0) {
#pragma unroll
        for (int m = 0; m < NM; m++) v[m] = p[m * TH];
    } else if (LB == 1 || far == 1) {
#pragma unroll
        for (int m = 0; m < NM; m++) v[m] = fma(R, p[m * TH], p[(M1 + m) * TH]);
    } else if (LA < 2 || far == 2) {
        const double R2 = R * R, RR = R + R;
#pragma unroll
        for (int m = 0; m < NM; m++) v[m] = fma(R2, p[m * TH], fma(RR, p[(M1 + m) * TH], p[(2 * M1 + m) * TH]));
    } else {  // a + 1 = 3
        const double R3 = R * R * R, T2 = 3.0 * R * R, T1 = 3.0 * R;
#pragma unroll
        for (int m = 0; m < NM; m++)
            v[m] = fma(R3, p[m * TH], fma(T2, p[(M1 + m) * TH], fma(T1, p[(2 * M1 + m) * TH], p[(3 * M1 + m) * TH])));
    }
}

// h(c, d) from v[m], m <= LC + LD (shift_ket; `swap`: the recurrence is on d).
template <int LC, int LD>
__device__ __forceinline__ void kgrad_shift_ket(bool swap, double* v, double R, double* out)
{
    if (LD < 2 || !swap) {
        shift_ket<LC, LD>(v, R, out);
    } else {
#pragma unroll
        for (int c = 0; c <= LC; c++) {
#pragma unroll
            for (int d = 0; d <= LD; d++) out[c * (LD + 1) + d] = v[d];
            if (c < LC) {
#pragma unroll
                for (int d = 0; d < LC + LD - c; d++) v[d] = fma(R, v[d], v[d + 1]);
            }
        }
    }
}

// The two centres' derivative sums of one direction for sensitivities S(c, d)
// of the extended integrals H(c, d), c <= LC + 1.
template <int LA, int LB, int LC, int LD, int M1, int TH>
__device__ __forceinline__ void kgrad_direction(const double* V, int base, int ax, int bx, double R, double Rk,
                                                double al2, double ga2, const double* S, const double* H, double& gA, double& gC)
{
    constexpr int D1 = LD + 1, NM = LC + LD + 1;
    double p[NM], h[(LC + 1) * D1];
    kgrad_shift<LA, LB, M1, NM, TH>(V, base & 1, ax + 1, bx, R, p);
#pragma unroll
    for (int m = 0; m < NM; m++) p[m] *= al2;
    if (ax > 0) {
        double q[NM];
        kgrad_shift<LA, LB, M1, NM, TH>(V, base & 1, ax - 1, bx, R, q);
#pragma unroll
        for (int m = 0; m < NM; m++) p[m] = fma(-(double)ax, q[m], p[m]);
    }
    kgrad_shift_ket<LC, LD>(base & 2, p, Rk, h);
    double s1 = 0.0, s2 = 0.0;
#pragma unroll
    for (int c = 0; c <= LC; c++)
#pragma unroll
        for (int d = 0; d <= LD; d++) {
            gA = fma(S[c * D1 + d], h[c * D1 + d], gA);
            s1 = fma(S[c * D1 + d], H[(c + 1) * D1 + d], s1);
            if (c > 0) s2 = fma(-(double)c * S[c * D1 + d], H[(c - 1) * D1 + d], s2);
        }
    gC += fma(ga2, s1, s2);
}

// The six sums of one root with per-component S and component masks.
template <int LA, int LB, int LC, int LD>
__device__ __noinline__ void kgrad_masked(const KPartnerRecs& ab, const KPartnerRecs& cd, int jr, int lr, int base,
                                          const KDensity& dm, const double* Dw, const double* V, double al2,
                                          double ga2, double* g)
{
    constexpr int N1 = LA + LB + 2, M1 = LC + LD + 2, TH = KGradShape<LA, LB, LC, LD>::THREADS;
    const int spj = __ldg(ab.rec_sp + jr), spl = __ldg(cd.rec_sp + lr);
    const uint64_t mj = __ldg(ab.rec_mask + jr), ml = __ldg(cd.rec_mask + lr);
    const double suj = __ldg(ab.su + jr), sul = __ldg(cd.su + lr);
    const int jsh = __ldg(ab.partner + spj), lsh = __ldg(cd.partner + spl);
    double R[3], Rk[3];
    for (int x = 0; x < 3; x++) {
        R[x] = __ldg(ab.geo + (G_RX + x) * ab.sp_stride + spj);
        Rk[x] = __ldg(cd.geo + (G_RX + x) * cd.sp_stride + spl);
        if (base & 1) R[x] = -R[x];
        if (base & 2) Rk[x] = -Rk[x];
    }
    const bool sb = base & 1, sd = base & 2;
    auto value = [&](const double* Vx, int a, int b, int c, int d, int x) {
        return krys_value<M1, TH>(Vx, sb ? b : a, sb ? a : b, sd ? d : c, sd ? c : d, R[x], Rk[x]);
    };
    for (int ij = 0; ij < ncart(LA) * ncart(LB); ij++) {
        if (!((mj >> ij) & 1ull)) continue;
        const double Sij = isnan(suj) ? __ldg(ab.S + ij * ab.sp_stride + spj) : suj;
        const int ca = ij / ncart(LB), cb = ij % ncart(LB);
        int a[3], b[3], c[3], d[3];
        cart_exps(LA, ca, a[0], a[1], a[2]);
        cart_exps(LB, cb, b[0], b[1], b[2]);
        const uint32_t jao = __ldg(dm.b_aoinds + jsh + (int64_t)dm.b_count * cb);
        for (int kl = 0; kl < ncart(LC) * ncart(LD); kl++) {
            if (!((ml >> kl) & 1ull)) continue;
            const double Skl = isnan(sul) ? __ldg(cd.S + kl * cd.sp_stride + spl) : sul;
            const int cc = kl / ncart(LD), cdd = kl % ncart(LD);
            cart_exps(LC, cc, c[0], c[1], c[2]);
            cart_exps(LD, cdd, d[0], d[1], d[2]);
            const uint32_t lao = __ldg(dm.d_aoinds + lsh + (int64_t)dm.d_count * cdd);
            const double w = Dw[ca * ncart(LC) + cc] * Sij * Skl * __ldg(dm.D + (int64_t)jao * dm.naos + lao);
            double I[3], dA[3], dC[3];
            for (int x = 0; x < 3; x++) {
                const double* Vx = V + x * N1 * M1 * TH;
                I[x] = value(Vx, a[x], b[x], c[x], d[x], x);
                dA[x] = al2 * value(Vx, a[x] + 1, b[x], c[x], d[x], x);
                if (a[x] > 0) dA[x] -= a[x] * value(Vx, a[x] - 1, b[x], c[x], d[x], x);
                dC[x] = ga2 * value(Vx, a[x], b[x], c[x] + 1, d[x], x);
                if (c[x] > 0) dC[x] -= c[x] * value(Vx, a[x], b[x], c[x] - 1, d[x], x);
            }
            for (int x = 0; x < 3; x++) {
                const double o = w * I[(x + 1) % 3] * I[(x + 2) % 3];
                g[x] = fma(o, dA[x], g[x]);
                g[3 + x] = fma(o, dC[x], g[3 + x]);
            }
        }
    }
}

template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void kgrad_lane(const KPartnerRecs& ab, const KPartnerRecs& cd, const KWarpSetup<KGradShape<LA, LB, LC, LD>::BATCH>& st,
                                           int q, int root, const KDensity& dm, const double* Dw,
                                           const double* __restrict__ rtab, double* V, double* g)
{
    using S = KGradShape<LA, LB, LC, LD>;
    constexpr int N1 = S::N1, M1 = S::M1, TH = S::THREADS, NS = S::BATCH, VX = N1 * M1 * TH;
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    constexpr int D1 = LD + 1, CD = (LC + 1) * D1, CE = (LC + 2) * D1;
    const double* sc = st.sc + q;
    KVTable<N1 * M1, false, TH> Vx{V}, Vy{V + VX}, Vz{V + 2 * VX};
    krys_tables<S::NR, N1, M1, NS>(sc, root, rtab, Vx, Vy, Vz);
    const double al2 = 2.0 * sc[KF_AL * NS], ga2 = 2.0 * sc[KF_GA * NS];
    const int base = st.base[q];
    if (st.jr[q] < 0) {
        double h[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        kgrad_masked<LA, LB, LC, LD>(ab, cd, ~st.jr[q], st.lr[q], base, dm, Dw, V, al2, ga2, h);
#pragma unroll
        for (int x = 0; x < 6; x++) g[x] += h[x];
        return;
    }
    const int jsh = st.jsh[q], lsh = st.lsh[q];
    double R[3], Rk[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        R[k] = sc[(KF_AB + k) * NS];
        Rk[k] = sc[(KF_CD + k) * NS];
    }
    uint32_t lao[ND];
#pragma unroll
    for (int k = 0; k < ND; k++) lao[k] = __ldg(dm.d_aoinds + lsh + (int64_t)dm.d_count * k);
#pragma unroll 1
    for (int t = 0; t < NB; t++) {
        int bx, by, bz;
        krys_b<LB>(t, bx, by, bz);
        const uint32_t jao = __ldg(dm.b_aoinds + jsh + (int64_t)dm.b_count * cart_index(by, bz));
        const double* Drow = dm.D + (int64_t)jao * dm.naos;
        double Dv[ND];
#pragma unroll
        for (int k = 0; k < ND; k++) Dv[k] = __ldg(Drow + lao[k]);
#pragma unroll 1
        for (int a = 0; a < NA; a++) {
            int ax, ay, az;
            cart_exps(LA, a, ax, ay, az);
            double X[CE], Y[CE], Z[CE], v[M1];
            kgrad_shift<LA, LB, M1, M1, TH>(V, base & 1, ax, bx, R[0], v);
            kgrad_shift_ket<LC + 1, LD>(base & 2, v, Rk[0], X);
            kgrad_shift<LA, LB, M1, M1, TH>(V + VX, base & 1, ay, by, R[1], v);
            kgrad_shift_ket<LC + 1, LD>(base & 2, v, Rk[1], Y);
            kgrad_shift<LA, LB, M1, M1, TH>(V + 2 * VX, base & 1, az, bz, R[2], v);
            kgrad_shift_ket<LC + 1, LD>(base & 2, v, Rk[2], Z);
            double Xb[CD], Yb[CD], Zb[CD];
#pragma unroll
            for (int k = 0; k < CD; k++) Xb[k] = Yb[k] = Zb[k] = 0.0;
#pragma unroll
            for (int z = 0; z <= LC; z++) {
                double T1[ND], Tb[ND];
#pragma unroll
                for (int dy = 0; dy <= LD; dy++)
#pragma unroll
                    for (int dz = 0; dz <= LD - dy; dz++) {
                        const int k = cart_index(dy, dz);
                        T1[k] = Dv[k] * Z[z * D1 + dz];
                        Tb[k] = 0.0;
                    }
#pragma unroll
                for (int y = 0; y <= LC - z; y++) {
                    const int x = LC - z - y;
                    const double wc = Dw[a * NC + cart_index(y, z)];
#pragma unroll
                    for (int dx = 0; dx <= LD; dx++) {
                        const double xw = wc * X[x * D1 + dx];
                        double s = 0.0;
#pragma unroll
                        for (int dy = 0; dy <= LD - dx; dy++) {
                            const int k = cart_index(dy, LD - dx - dy);
                            s = fma(T1[k], Y[y * D1 + dy], s);
                            Yb[y * D1 + dy] = fma(xw, T1[k], Yb[y * D1 + dy]);
                            Tb[k] = fma(xw, Y[y * D1 + dy], Tb[k]);
                        }
                        Xb[x * D1 + dx] = fma(wc, s, Xb[x * D1 + dx]);
                    }
                }
#pragma unroll
                for (int dy = 0; dy <= LD; dy++)
#pragma unroll
                    for (int dz = 0; dz <= LD - dy; dz++) {
                        const int k = cart_index(dy, dz);
                        Zb[z * D1 + dz] = fma(Tb[k], Dv[k], Zb[z * D1 + dz]);
                    }
            }
            kgrad_direction<LA, LB, LC, LD, M1, TH>(V, base, ax, bx, R[0], Rk[0], al2, ga2, Xb, X, g[0], g[3]);
            kgrad_direction<LA, LB, LC, LD, M1, TH>(V + VX, base, ay, by, R[1], Rk[1], al2, ga2, Yb, Y, g[1], g[4]);
            kgrad_direction<LA, LB, LC, LD, M1, TH>(V + 2 * VX, base, az, bz, R[2], Rk[2], al2, ga2, Zb, Z, g[2], g[5]);
        }
    }
}

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__((KGradShape<LA, LB, LC, LD>::THREADS), (KGradShape<LA, LB, LC, LD>::MINB))
exchange_grad_kernel(KOutBlocks out, KPartnerRecs ab, KPartnerRecs cd, KDensity dm, KGradBlockD bd, double maxD,
                     double omega, double thr, double* __restrict__ grad, int64_t gstride,
                     const double* __restrict__ rtab)
{
    using S = KGradShape<LA, LB, LC, LD>;
    constexpr int NA = ncart(LA), NC = ncart(LC), NW = S::NW;
    extern __shared__ double krys_smem[];
    __shared__ int s_nl[K_JCHUNK], s_n64[K_JCHUNK], s_c64[K_JCHUNK + 1], s_c32[K_JCHUNK + 1];
    __shared__ double sDw[NA * NC];
    __shared__ double red[NW][6];
    __shared__ int s_pmin;
    __shared__ KWarpSetup<S::BATCH> s_set[NW];
    double* V = krys_smem + threadIdx.x;
    const KChunk ch{s_nl, s_n64, s_c64, s_c32};
    const int nout = *out.n;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int root = lane % S::NR, slot = lane / S::NR;
    KWarpSetup<S::BATCH>& set = s_set[warp];

    for (int o = blockIdx.x; o < nout; o += gridDim.x) {
        const int ish = __ldg(out.ish + o), ksh = __ldg(out.ksh + o);
        if (threadIdx.x == 0) s_pmin = INT32_MAX;
        __syncthreads();
        if (threadIdx.x < NA * NC) {
            const int ca = threadIdx.x / NC, cc = threadIdx.x % NC;
            const int32_t p = __ldg(out.idx + threadIdx.x * out.stride + o);
            double w = 0.0;
            if (p >= 0) {
                const uint32_t iao = __ldg(bd.a_aoinds + ish + (int64_t)bd.a_count * ca);
                const uint32_t kao = __ldg(bd.c_aoinds + ksh + (int64_t)bd.c_count * cc);
                const bool diag = bd.same_type && ish == ksh && ca == cc;
                w = (diag ? 1.0 : 2.0) * __ldg(dm.D + (int64_t)iao * dm.naos + kao);
                atomicMin(&s_pmin, (int)p);
            }
            sDw[threadIdx.x] = w;
        }
        __syncthreads();
        const int a0 = __ldg(ab.seg + ish), a1 = __ldg(ab.seg + ish + 1);
        const int c0 = __ldg(cd.seg + ksh), c1 = __ldg(cd.seg + ksh + 1);
        double g[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int jb = a0; jb < a1; jb += K_JCHUNK) {
            const int nj = min(K_JCHUNK, a1 - jb);
            k_chunk_scan(ab, cd, jb, nj, c0, c1, maxD, thr, 0.0, ch);
            const int total = s_c64[nj];
            const int batch = krys_batch(total, NW, S::QW, S::BATCH);
            int jj = 0;
            for (int w0 = warp * batch; w0 < total; w0 += NW * batch) {
                const int n = min(batch, total - w0), w = w0 + lane;
                if (lane < n) {
                    while (s_c64[jj + 1] <= w) jj++;
                    krys_setup<true, (LB > 1), (LD > 1)>(ab, cd, jb + jj, c0 + w - s_c64[jj], omega, set, lane);
                }
                __syncwarp();
                if (slot < S::QW)
                    for (int q = slot; q < n; q += S::QW)
                        kgrad_lane<LA, LB, LC, LD>(ab, cd, set, q, root, dm, sDw, rtab, V, g);
                __syncwarp();
            }
            __syncthreads();
        }
#pragma unroll
        for (int x = 0; x < 6; x++) {
            const double v = warp_sum(g[x]);
            if (lane == 0) red[warp][x] = v;
        }
        __syncthreads();
        if (threadIdx.x < 6 && s_pmin != INT32_MAX) {
            double s = red[0][threadIdx.x];
#pragma unroll
            for (int w = 1; w < NW; w++) s += red[w][threadIdx.x];
            grad[threadIdx.x * gstride + s_pmin] += s;
        }
        __syncthreads();
    }
}

template <int LA, int LB, int LC, int LD>
int launch_exchange_grad(int grid, cudaStream_t st, const KOutBlocks& out, const KPartnerRecs& ab,
                         const KPartnerRecs& cd, const KDensity& dm, const KGradBlockD& bd, double maxD, double omega,
                         double thr, double* grad, int64_t gstride)
{
    using S = KGradShape<LA, LB, LC, LD>;
    static std::atomic<unsigned long long> done;
    const double* tab = rys_table_device();
    if (!tab) return VLXB_ECUDA;
    const int rc = rys_prepare((const void*)exchange_grad_kernel<LA, LB, LC, LD>, S::SMEM, S::MINB, done);
    if (rc) return rc;
    exchange_grad_kernel<LA, LB, LC, LD><<<grid, S::THREADS, S::SMEM, st>>>(
        out, ab, cd, dm, bd, maxD, omega, thr, grad, gstride, tab + rys_offset(S::NR));
    VLXB_CHECK_CUDA(cudaGetLastError());
    return VLXB_OK;
}

}  // namespace vlxb
