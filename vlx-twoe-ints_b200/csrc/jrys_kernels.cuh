// Coulomb and its nuclear gradient by Rys quadrature over Hermite Gaussians
// (sm_100a).
//
// J_ab = S_ab sum_e E^{ab}_e X_e, X_e = sum over kets of sum_f R_{e+f} Dh_f
// (md.cuh).  At root r of the quadrature the Hermite Coulomb integral factors:
//   R_{tuv} = sum_r W_r Hx_t Hy_u Hz_v,  H_0 = 1,
//   H_{t+1} = -2 rho x_r (PQ H_t + t H_{t-1})
// (from R^{(n)}_{000} = (-2 rho)^n sum_r W_r x_r^n), so that X is a sum
// factorisation with no R table: per root
//   T[ez; fx fy] = sum_fz Hz[ez + fz] Dh[fx fy fz]
//   U[ey ez; fx] = sum_fy Hy[ey + fy] T[ez; fx fy]
//   X_e         += sum_fx Hx[ex + fx] U[ey ez; fx],
// 575 multiply-adds for a (DD|DD) quartet root against 1225 for R x Dh alone.
// One lane evaluates one root of one quartet and keeps the whole X of the bra
// in registers over all of the bra's kets: nothing is exchanged between lanes.
// A warp takes up to 32 kets at a time: one lane per ket sets up what does not
// depend on the root, the ket densities are copied to shared memory as one
// contiguous block and read back as broadcasts; a ket in the screening band
// (some components below the threshold) has its density rebuilt there by its
// lane with the exact per-component screen.
//
// Bound: FP64 issue (pipe 40 to 51 % busy, lane efficiency 30 of 32 at worst); for
// kets with two d shells the unrolled rebuilding of screened densities, which
// waits for instructions as often as for results.  10 atoms 4s3p2d, ms per class
// call: (DD|DD) 7.9 -> 1.8, (PD|DD) 9.8 -> 2.6, (DD|PD) 6.0 -> 1.7, (PD|PD) 5.5
// -> 2.8; the gradient of all classes 444 -> 78.
//
// G = 1: the bra-centre derivatives: the bra range grows by one level and the
// epilogue sums E^{a+-1,b} and E^{a,b+-1} against X:
//   dJ_ab/dA_x = S_ab sum_e (2 alpha E^{a+1x,b}_e - a_x E^{a-1x,b}_e) X_e,
// the same with beta = p - alpha on B (Obara-Saika 1986, Eq. 5; eri.py:85-129
// of the reference generator), written to out[k * gstride + o], k = 0..2 the
// A components, 3..5 the B components.  Quartet set, counters and FP32 pass
// are those of coulomb_kernel; results are accumulated with += in a fixed
// order (no atomics).
#pragma once
#include <atomic>
#include <type_traits>
#include <utility>

#include "engine.cuh"
#include "jk_kernels.cuh"
#include "launch.cuh"
#include "md.cuh"
#include "rys.cuh"

namespace vlxb {

template <int LA, int LB, int LC, int LD, int G>
struct JRysShape {
    static constexpr int LE = LA + LB + G, LF = LC + LD, L = LE + LF;
    static constexpr int NR = L / 2 + 1;
    static constexpr int QW = 32 / NR;  // kets per warp
    static constexpr int NW = J_THREADS / 32;
    static constexpr int NHB = nherm(LE), NHK = nherm(LF);
    static constexpr int BATCH = 32 / QW * QW;  // kets set up together
    // CTAs per SM: the NHB partials are the registers that count.  8 atoms 4s3p2d,
    // ms for the Coulomb classes / the gradient classes of one NHB with 2, 3 and 4
    // CTAs: NHB 10 5.1 4.3 4.1 / 9.2 7.9 7.2; 20 5.2 4.5 4.3 / 14.8 12.8 11.9;
    // 35 3.2 3.1 3.6 / 10.3 9.2 10.3; 56 (gradient) 6.3 7.8 11.3.
    static constexpr int MINB = NHB > 20 ? 2 : (NHB > 12 ? 3 : 4);
};

// Scalars of one quartet: field f of slot q at sc[f * 32 + q].
enum JField { JF_PQ = 0, JF_M2R = 3, JF_T, JF_W, JF_N };

template <int N, typename F, int... I>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, I...>)
{
    (f(std::integral_constant<int, I>{}), ...);
}
// f(integral_constant 0 .. N-1): loop indices that the body can use as constants.
template <int N, typename F>
__device__ __forceinline__ void static_for(F&& f)
{
    static_for_impl<N>(f, std::make_integer_sequence<int, N>{});
}

// E[t], t <= I + J, of the 1-D Hermite coefficients E^{IJ}_t.
template <int I, int J>
__device__ __forceinline__ void herm_one(double PA, double PB, double h, double (&e)[I + J + 1])
{
#pragma unroll
    for (int t = 0; t <= I + J; t++) e[t] = t == 0 ? 1.0 : 0.0;
    static_for<I + J>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        const double X = k < I ? PA : PB;
        double n[k + 2];
#pragma unroll
        for (int t = 0; t <= k + 1; t++) {
            double v = t <= k ? X * e[t] : 0.0;
            if (t > 0) v = fma(h, e[t - 1], v);
            if (t + 1 <= k) v = fma((double)(t + 1), e[t + 1], v);
            n[t] = v;
        }
#pragma unroll
        for (int t = 0; t <= k + 1; t++) e[t] = n[t];
    });
}

// Hermite density of a ket with the exact per-component screen (same product
// order as the reference: fabs(Q_ij * Q_kl * D_kl) <= thr -> skip); every index
// is a template constant, so that the sums stay in registers.
template <int LC, int LD, typename T>
__device__ __noinline__ void jrys_screened(const JKetPairs& ket, int kt, double qb, double thr, T* row)
{
    constexpr int ND = ncart(LD);
    const PairGeo k = load_geo(ket.geo, ket.stride, kt);
    double Dh[nherm(LC + LD)];
#pragma unroll
    for (int f = 0; f < nherm(LC + LD); f++) Dh[f] = 0.0;
    static_for<ncart(LC) * ND>([&](auto cdc) {
        constexpr int cd = decltype(cdc)::value, c = cd / ND, d = cd % ND;
        constexpr int cx = cart_x(LC, c), cy = cart_y(LC, c), cz = cart_z(LC, c);
        constexpr int dx = cart_x(LD, d), dy = cart_y(LD, d), dz = cart_z(LD, d);
        const double qk = __ldg(ket.Qc + cd * ket.stride + kt);
        const double dk = __ldg(ket.Dc + cd * ket.stride + kt);
        if (fabs(qb * qk * dk) > thr) {
            const double w = __ldg(ket.Dm + cd * ket.stride + kt);
            double ex[cx + dx + 1], ey[cy + dy + 1], ez[cz + dz + 1];
            herm_one<cx, dx>(k.Ax, k.Ax + k.Rx, k.i2z, ex);
            herm_one<cy, dy>(k.Ay, k.Ay + k.Ry, k.i2z, ey);
            herm_one<cz, dz>(k.Az, k.Az + k.Rz, k.i2z, ez);
            static_for<cx + dx + 1>([&](auto tc) {
                static_for<cy + dy + 1>([&](auto uc) {
                    static_for<cz + dz + 1>([&](auto vc) {
                        constexpr int t = decltype(tc)::value, u = decltype(uc)::value, v = decltype(vc)::value;
                        constexpr int f = herm_idx(t, u, v);
                        const double e = w * ex[t] * ey[u] * ez[v];
                        Dh[f] += ((t + u + v) & 1) ? -e : e;
                    });
                });
            });
        }
    });
#pragma unroll
    for (int f = 0; f < nherm(LC + LD); f++) row[f] = (T)Dh[f];
}

// Position of (x, y), x + y <= n, in a triangular table.
__host__ __device__ constexpr int cart_index2(int x, int y) { return (x + y) * (x + y + 1) / 2 + y; }

// One halving step of warp_fold: the upper half of v goes to the lanes with
// bit o set, the lower half to the others.
template <int N>
struct WarpFold {
    static __device__ __forceinline__ void run(double* v, int lane, int o)
    {
        constexpr int H = (N + 1) / 2;
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < H; i++) {
            const double hi = i + H < N ? v[i + H] : 0.0;
            const double send = up ? v[i] : hi, keep = up ? hi : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
};

// out[e] (shared memory) = sum of v[e] over the warp, in a fixed order.  Half
// of the array leaves each lane at every step: about N exchanges where N
// butterflies take 5 N.
template <int N>
__device__ __forceinline__ void warp_fold(double* v, int lane, double* out)
{
    constexpr int N1 = (N + 1) / 2, N2 = (N1 + 1) / 2, N3 = (N2 + 1) / 2, N4 = (N3 + 1) / 2, N5 = (N4 + 1) / 2;
    WarpFold<N>::run(v, lane, 16);
    WarpFold<N1>::run(v, lane, 8);
    WarpFold<N2>::run(v, lane, 4);
    WarpFold<N3>::run(v, lane, 2);
    WarpFold<N4>::run(v, lane, 1);
    // this lane now holds elements base .. base + lim - 1
    int base = 0, lim = N;
    const int half[5] = {N1, N2, N3, N4, N5};
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const bool up = (lane & (16 >> k)) != 0;
        if (up) base += half[k];
        lim = up ? lim - half[k] : min(lim, half[k]);
    }
#pragma unroll
    for (int i = 0; i < N5; i++)
        if (i < lim) out[base + i] = v[i];
}

template <int LA, int LB, int LC, int LD, int PM, int G>
__global__ void __launch_bounds__(J_THREADS, (JRysShape<LA, LB, LC, LD, G>::MINB))
coulomb_rys_kernel(JBraRecs bra, JKetPairs ket, double* __restrict__ mat_J, int64_t gstride, double thr,
                   const double* __restrict__ rtab, unsigned long long* __restrict__ qcount, double fp32_cut,
                   double fp32_budget)
{
    using S = JRysShape<LA, LB, LC, LD, G>;
    using T = typename std::conditional<PM == 0, double, float>::type;
    constexpr int LE = S::LE, LF = S::LF, L = S::L, NR = S::NR, QW = S::QW, NW = S::NW;
    constexpr int NHB = S::NHB, NHK = S::NHK;
    constexpr int NB = ncart(LB), NAB = ncart(LA) * NB;
    __shared__ T sDh[NW][S::BATCH * NHK];
    __shared__ double sSc[NW][JF_N * 32];
    __shared__ double sX[NW][NHB];
    __shared__ double sEb[3][(LA + G + 1) * (LB + G + 1) * (LA + LB + 2 * G + 1)];
    __shared__ int s_ncut, s_n64;
    const int nbra = *bra.n_rec;
    const int nket = *ket.n;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = lane / NR, root = lane % NR;

    for (int r = blockIdx.x; r < nbra; r += gridDim.x) {
        const int sp = __ldg(bra.rec_sp + r);
        const PairGeo b = load_geo(bra.geo, bra.sp_stride, sp);
        const double qb = __ldg(bra.rec_q + r);
        int k0 = 0, k1 = nket;
        if (bra.mol) {
            const int m = __ldg(bra.mol + r);
            k0 = __ldg(ket.seg + m);
            k1 = __ldg(ket.seg + m + 1);
        }
        if (threadIdx.x == 0) {
            int ncut, nexact, n64;
            ket_prefixes(ket, k0, k1, qb, thr, fp32_cut, fabs(qb) * pair_amp(b, LB), fp32_budget, ncut, nexact, n64);
            s_ncut = ncut;
            s_n64 = n64;
            if (qcount && PM == 0) atomicAdd(qcount, (unsigned long long)(nexact - k0));
        }
        __syncthreads();
        const int kb = PM == 0 ? k0 : s_n64, ke = PM == 0 ? s_n64 : s_ncut;
        if (PM == 1 && kb >= ke) {
            __syncthreads();
            continue;  // no FP32 quartets for this bra
        }

        double X[NHB];
#pragma unroll
        for (int e = 0; e < NHB; e++) X[e] = 0.0;
        const int share = (ke - kb + NW - 1) / NW;
        const int batch = min(S::BATCH, (share + QW - 1) / QW * QW);
        for (int base = kb + warp * batch; base < ke; base += NW * batch) {
            const int n = min(batch, ke - base);
            for (int i = lane; i < n * NHK; i += 32) sDh[warp][i] = (T)__ldg(ket.Dh + (int64_t)base * NHK + i);
            bool screened = false;
            if (lane < n) {
                const int kt = base + lane;
                screened = !(qb * __ldg(ket.tmin + kt) > thr * (1.0 + SCREEN_SLACK));
                const double kz = __ldg(ket.geo + G_Z * ket.stride + kt);
                const double rho = b.z * kz / (b.z + kz);
                const double PQ[3] = {b.Px - __ldg(ket.geo + G_PX * ket.stride + kt),
                                      b.Py - __ldg(ket.geo + G_PY * ket.stride + kt),
                                      b.Pz - __ldg(ket.geo + G_PZ * ket.stride + kt)};
                double* sc = sSc[warp] + lane;
#pragma unroll
                for (int k = 0; k < 3; k++) sc[(JF_PQ + k) * 32] = PQ[k];
                sc[JF_M2R * 32] = -2.0 * rho;
                sc[JF_T * 32] = rho * fma(PQ[0], PQ[0], fma(PQ[1], PQ[1], PQ[2] * PQ[2]));
                sc[JF_W * 32] = 2.0 * sqrt(rho * INV_PI_D);
            }
            __syncwarp();
            if (screened) jrys_screened<LC, LD, T>(ket, base + lane, qb, thr, sDh[warp] + lane * NHK);
            __syncwarp();
            for (int q = slot; slot < QW && q < n; q += QW) {
                const double* sc = sSc[warp] + q;
                double x, w;
                rys_root<NR>(sc[JF_T * 32], rtab, root, x, w);
                w *= sc[JF_W * 32];
                const double m2 = sc[JF_M2R * 32] * x;
                T H[3][L + 1];
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const T a = (T)m2, ap = (T)(m2 * sc[(JF_PQ + k) * 32]);
                    H[k][0] = k == 2 ? (T)w : (T)1;
                    if (L > 0) H[k][1] = ap * H[k][0];
#pragma unroll
                    for (int t = 1; t < L; t++) H[k][t + 1] = fma(ap, H[k][t], (T)t * a * H[k][t - 1]);
                }
                const T* Dh = sDh[warp] + q * NHK;
#pragma unroll
                for (int ez = 0; ez <= LE; ez++) {
                    T Tz[(LF + 1) * (LF + 2) / 2];
#pragma unroll
                    for (int fx = 0; fx <= LF; fx++)
#pragma unroll
                        for (int fy = 0; fy <= LF - fx; fy++) {
                            T s = H[2][ez] * Dh[herm_idx(fx, fy, 0)];
#pragma unroll
                            for (int fz = 1; fz <= LF - fx - fy; fz++)
                                s = fma(H[2][ez + fz], Dh[herm_idx(fx, fy, fz)], s);
                            Tz[cart_index2(fx, fy)] = s;
                        }
#pragma unroll
                    for (int ey = 0; ey <= LE - ez; ey++) {
                        T U[LF + 1];
#pragma unroll
                        for (int fx = 0; fx <= LF; fx++) {
                            T s = H[1][ey] * Tz[cart_index2(fx, 0)];
#pragma unroll
                            for (int fy = 1; fy <= LF - fx; fy++) s = fma(H[1][ey + fy], Tz[cart_index2(fx, fy)], s);
                            U[fx] = s;
                        }
#pragma unroll
                        for (int ex = 0; ex <= LE - ez - ey; ex++) {
                            if constexpr (PM == 0) {
#pragma unroll
                                for (int fx = 0; fx <= LF; fx++)
                                    X[herm_idx(ex, ey, ez)] = fma(H[0][ex + fx], U[fx], X[herm_idx(ex, ey, ez)]);
                            } else {
                                T s = H[0][ex] * U[0];
#pragma unroll
                                for (int fx = 1; fx <= LF; fx++) s = fma(H[0][ex + fx], U[fx], s);
                                X[herm_idx(ex, ey, ez)] += (double)s;
                            }
                        }
                    }
                }
            }
            __syncwarp();
        }
        warp_fold<NHB>(X, lane, sX[warp]);
        __syncthreads();
        for (int e = threadIdx.x; e < NHB; e += J_THREADS) {
            double s = sX[0][e];
#pragma unroll
            for (int w = 1; w < NW; w++) s += sX[w][e];
            sX[0][e] = s;
        }
        if (threadIdx.x < 3) {
            const double pa = threadIdx.x == 0 ? b.Ax : (threadIdx.x == 1 ? b.Ay : b.Az);
            const double ab = threadIdx.x == 0 ? b.Rx : (threadIdx.x == 1 ? b.Ry : b.Rz);
            herm_e1_flat<LA + G, LB + G>(pa, pa + ab, b.i2z, sEb[threadIdx.x]);
        }
        __syncthreads();
        const uint64_t mask = __ldg(bra.rec_mask + r);
        if (threadIdx.x < NAB && ((mask >> threadIdx.x) & 1ull)) {
            const int c = threadIdx.x;
            const int ai = c / NB, bi = c % NB;
            const int ax = cart_x(LA, ai), ay = cart_y(LA, ai), az = cart_z(LA, ai);
            const int bx = cart_x(LB, bi), by = cart_y(LB, bi), bz = cart_z(LB, bi);
            constexpr int LS = LA + LB + 2 * G + 1, NJ = LB + G + 1;
            // sum_e E^{(ix,iy,iz),(jx,jy,jz)}_e X_e over the product's Hermite box
            auto hsum = [&](int ix, int iy, int iz, int jx, int jy, int jz) {
                double acc = 0.0;
                for (int t = 0; t <= ix + jx; t++)
                    for (int u = 0; u <= iy + jy; u++) {
                        const double etu = sEb[0][(ix * NJ + jx) * LS + t] * sEb[1][(iy * NJ + jy) * LS + u];
                        for (int v = 0; v <= iz + jz; v++)
                            acc = fma(etu * sEb[2][(iz * NJ + jz) * LS + v], sX[0][herm_idx(t, u, v)], acc);
                    }
                return acc;
            };
            const int32_t o = __ldg(bra.entry + c * bra.sp_stride + sp);
            const double Sv = __ldg(bra.pdata + o);
            if constexpr (G == 0) {
                mat_J[o] += Sv * hsum(ax, ay, az, bx, by, bz);
            } else {
                const double al2 = 2.0 * __ldg(bra.geo + G_ALPHA * bra.sp_stride + sp);
                const double be2 = 2.0 * b.z - al2;
                const int av[3] = {ax, ay, az}, bv[3] = {bx, by, bz};
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    const int ex = d == 0, ey = d == 1, ez = d == 2;
                    double gA = al2 * hsum(ax + ex, ay + ey, az + ez, bx, by, bz);
                    if (av[d] > 0) gA -= av[d] * hsum(ax - ex, ay - ey, az - ez, bx, by, bz);
                    double gB = be2 * hsum(ax, ay, az, bx + ex, by + ey, bz + ez);
                    if (bv[d] > 0) gB -= bv[d] * hsum(ax, ay, az, bx - ex, by - ey, bz - ez);
                    mat_J[d * gstride + o] += Sv * gA;
                    mat_J[(3 + d) * gstride + o] += Sv * gB;
                }
            }
        }
        __syncthreads();
    }
}

template <int LA, int LB, int LC, int LD>
int launch_coulomb_rys(int grid, cudaStream_t st, const JBraRecs& bra, const JKetPairs& ket, double* mat_J, double thr,
                       unsigned long long* qc, double cut, double budget)
{
    const double* tab = rys_table_device();
    if (!tab) return VLXB_ECUDA;
    coulomb_rys_kernel<LA, LB, LC, LD, 0, 0><<<grid, J_THREADS, 0, st>>>(
        bra, ket, mat_J, 0, thr, tab + rys_offset(JRysShape<LA, LB, LC, LD, 0>::NR), qc, cut, budget);
    VLXB_CHECK_CUDA(cudaGetLastError());
    return VLXB_OK;
}

template <int LA, int LB, int LC, int LD>
int launch_coulomb_grad(int pm, int grid, cudaStream_t st, const JBraRecs& bra, const JKetPairs& ket, double* out,
                        int64_t gstride, double thr, double cut)
{
    const double* tab = rys_table_device();
    if (!tab) return VLXB_ECUDA;
    tab += rys_offset(JRysShape<LA, LB, LC, LD, 1>::NR);
    if (pm == 0)
        coulomb_rys_kernel<LA, LB, LC, LD, 0, 1><<<grid, J_THREADS, 0, st>>>(bra, ket, out, gstride, thr, tab, nullptr,
                                                                             cut, 0.0);
    else
        coulomb_rys_kernel<LA, LB, LC, LD, 1, 1><<<grid, J_THREADS, 0, st>>>(bra, ket, out, gstride, thr, tab, nullptr,
                                                                             cut, 0.0);
    VLXB_CHECK_CUDA(cudaGetLastError());
    return VLXB_OK;
}

}  // namespace vlxb
