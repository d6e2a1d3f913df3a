// Exchange by Rys quadrature with the density folded in (sm_100a).
//
// K_ac = sum over quartets, roots r and b, d of D_bd Ix(ax bx cx dx) Iy Iz,
// with Ix, Iy, Iz the 2-D integrals at root r (Dupuis, Rys and King 1976;
// recurrences of Rys, Dupuis and King 1983).  One lane evaluates one root of
// one primitive shell quartet: no lane idles except 32 mod NR, nothing is
// exchanged between lanes, and the K partials stay in its registers for the
// whole output block.  The components are never formed: for each b
//   T1[d]  = D_bd Iz(az bz cz dz)           per (az, cz)
//   T2[dx] = sum_dy T1 Iy(ay by cy dy)      per (az, cz, ay, cy)
//   K_ac  += sum_dx T2 Ix(ax bx cx dx),
// 9 multiply-adds per (a, b, c) for a d shell d, where the component integrals
// alone cost two per (a, b, c, d) and root.  All loops over components are
// unrolled and the VRR tables V(n, m), n <= LA + LB, m <= LC + LD, of the three
// directions stay in registers; the shifts to (a, b; c, d) are made when bx,
// by or bz changes (b runs through an order that changes bx and by least).
// What does not depend on the root (geometry, T, prefactor) is set up once per
// quartet by one lane for up to 32 quartets at a time and read back from
// shared memory by the lanes of the roots.
//
// Precision: the shift to the second centre loses digits from a diffuse to a
// tight shell, as a horizontal recurrence does, but fewer: 1.3e-15 of the Schwarz
// bound (root mean square over d-rich quartets, exponents 0.4 to 3, a box of 4
// bohr) against 4.6e-15 for VRR and HRR as in the thread and column kernels.
//
// Bound: FP64 issue.  (SD|DD) on 10 atoms 4s3p2d runs the FP64 pipe at 57 %
// ((PD|DP) 65 %), the rest being arithmetic latency that two warps per scheduler do not
// cover, with two CTAs of 128 threads per SM (registers); with the tables in shared
// memory the shared-memory pipe limits it (80 % busy, FP64 at 45 %).  Against
// the column kernels it replaces, ms per class call on that case: (DD|DD) 37.0
// -> 10.3, (PD|DD) 33.2 -> 9.6, (PD|DP) 31.8 -> 6.7, (DP|DD) 18.6 -> 5.8,
// (DD|DP) 18.4 -> 5.9, (SD|DD) 16.0 -> 5.4, (PD|PD) 15.9 -> 3.7, (PP|DD) 14.9
// -> 5.9, (DP|DP) 14.9 -> 3.4; thread per quartet: (SD|PD) 11.3 -> 4.5,
// (PP|DP) 9.2 -> 4.4, (SD|DP) 8.4 -> 3.9.
#pragma once
#include <atomic>

#include "common.cuh"
#include "engine.cuh"
#include "jk_kernels.cuh"
#include "launch.cuh"
#include "rys.cuh"

namespace vlxb {

constexpr int KR_THREADS = 128;

template <int LA, int LB, int LC, int LD>
struct KRysShape {
    static constexpr int L = LA + LB + LC + LD;
    static constexpr int NR = L / 2 + 1;        // roots
    static constexpr int QW = 32 / NR;          // quartets per warp
    static constexpr int BATCH = 32 / QW * QW;  // quartets a warp sets up together
    static constexpr int N1 = LA + LB + 1, M1 = LC + LD + 1;
    static constexpr int NAC = ncart(LA) * ncart(LC);
    // The VRR tables (3 N1 M1 values), the (a, c) partials and the x and y
    // slices stay in registers with the loop over b unrolled.  Where they do not
    // fit, (PD|DD), (DP|DD) and (DD|DP) spill 0.65 to 1.1 KB and are faster all
    // the same; (DD|DD), 4 KB, keeps the tables in shared memory, b not unrolled.
    // 10 atoms 4s3p2d, registers / shared memory, ms: (PD|DD) 9.2 / 11.7, (PD|PD)
    // 3.8 / 5.8, (DD|DP) 6.1 / 6.6, (DD|DD) 27.6 / 10.3.
    static constexpr bool REG = L < 8;
    static constexpr int SMEM_ROWS = REG ? 0 : 3 * N1 * M1;
    // values a lane keeps: up to 66 of them fit in the 168 registers of three
    // CTAs per SM ((SD|DP) 4.0 ms against 4.4 with two, (SD|DD) 5.8 against 5.6)
    static constexpr int KEPT = 3 * N1 * M1 + NAC + 2 * (LA + 1) * (LC + 1) * (LD + 1);
    static constexpr int MINB = KEPT <= 66 ? 3 : 2;
};

// Root-independent scalars of one quartet, set up once per quartet by one lane
// and read by the lanes of its roots: field f of slot q at sc[f * NS + q].
enum KField { KF_ZI = 0, KF_EI, KF_I2Z, KF_I2E, KF_HI, KF_PQ, KF_PA = KF_PQ + 3, KF_QC = KF_PA + 3,
              KF_AB = KF_QC + 3, KF_CD = KF_AB + 3, KF_T = KF_CD + 3, KF_W,
              KF_AL, KF_GA, KF_N };  // the exponents of a and c: gradient only

template <int NSLOT>
struct KWarpSetup {
    static constexpr int NS = NSLOT;
    double sc[KF_N * NS];
    int jsh[NS], lsh[NS];  // partner shells
    int jr[NS], lr[NS];    // records; jr < 0: no single S (per-component path)
    uint8_t base[NS];      // gradient only: bit 0 the bra's recurrence is on b, bit 1 the ket's on d
};

// SB, SD (gradient): the recurrence of a pair may be on b (d), its tighter shell;
// PA, AB (QC, CD) are then P - B, B - A (Q - D, D - C).
template <bool GRAD, bool SB, bool SD, typename ST>
__device__ __forceinline__ void krys_setup(const KPartnerRecs& ab, const KPartnerRecs& cd, int jr, int lr, double omega,
                                           ST& s, int q)
{
    constexpr int NS = ST::NS;
    const int spj = __ldg(ab.rec_sp + jr), spl = __ldg(cd.rec_sp + lr);
    const double suj = __ldg(ab.su + jr), sul = __ldg(cd.su + lr);
    const bool masked = isnan(suj) || isnan(sul);
    s.jsh[q] = __ldg(ab.partner + spj);
    s.lsh[q] = __ldg(cd.partner + spl);
    s.jr[q] = masked ? ~jr : jr;
    s.lr[q] = lr;
    if (GRAD) {
        s.sc[KF_AL * NS + q] = __ldg(ab.geo + G_ALPHA * ab.sp_stride + spj);
        s.sc[KF_GA * NS + q] = __ldg(cd.geo + G_ALPHA * cd.sp_stride + spl);
    }
    const PairGeo bg = load_geo(ab.geo, ab.sp_stride, spj);
    const PairGeo kg = load_geo(cd.geo, cd.sp_stride, spl);
    const double inv = 1.0 / (bg.z + kg.z);
    const double rho = bg.z * kg.z * inv;
    const double PQ[3] = {kg.Px - bg.Px, kg.Py - bg.Py, kg.Pz - bg.Pz};
    double d2 = 1.0;
    if (omega != 0.0) d2 = omega * omega / (rho + omega * omega);
    const double rd = rho * d2;
    double* sc = s.sc + q;
    sc[KF_ZI * NS] = kg.z * inv * d2;  // x d2 (rho / zeta), per root x
    sc[KF_EI * NS] = bg.z * inv * d2;
    sc[KF_I2Z * NS] = bg.i2z;
    sc[KF_I2E * NS] = kg.i2z;
    sc[KF_HI * NS] = 0.5 * inv * d2;
    double PA[3] = {bg.Ax, bg.Ay, bg.Az}, QC[3] = {kg.Ax, kg.Ay, kg.Az};
    double AB[3] = {bg.Rx, bg.Ry, bg.Rz}, CD[3] = {kg.Rx, kg.Ry, kg.Rz};
    if (GRAD) {
        const bool sb = SB && s.sc[KF_AL * NS + q] < 0.5 * bg.z, sd = SD && s.sc[KF_GA * NS + q] < 0.5 * kg.z;
        s.base[q] = (uint8_t)((sb ? 1 : 0) | (sd ? 2 : 0));
#pragma unroll
        for (int k = 0; k < 3; k++) {
            if (sb) {
                PA[k] += AB[k];
                AB[k] = -AB[k];
            }
            if (sd) {
                QC[k] += CD[k];
                CD[k] = -CD[k];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        sc[(KF_PQ + k) * NS] = PQ[k];
        sc[(KF_PA + k) * NS] = PA[k];
        sc[(KF_QC + k) * NS] = QC[k];
        sc[(KF_AB + k) * NS] = AB[k];
        sc[(KF_CD + k) * NS] = CD[k];
    }
    sc[KF_T * NS] = rd * fma(PQ[0], PQ[0], fma(PQ[1], PQ[1], PQ[2] * PQ[2]));
    sc[KF_W * NS] = 2.0 * sqrt(rd * INV_PI_D) * (masked ? 1.0 : suj * sul);
}

// Component index of (l - s, s - z, z) with s = y + z (the reference's order).
__host__ __device__ constexpr int cart_index(int y, int z) { return (y + z) * (y + z + 1) / 2 + z; }

// The b components in an order that changes (bx, by) least: packed bx, by, bz.
template <int LB>
__device__ __forceinline__ void krys_b(int t, int& bx, int& by, int& bz)
{
    if (LB == 0) {
        bx = by = bz = 0;
    } else if (LB == 1) {
        bx = t == 0;
        by = t == 1;
        bz = t == 2;
    } else {  // xx xz xy yz yy zz
        bx = t == 0 ? 2 : (t < 3 ? 1 : 0);
        by = t < 2 ? 0 : (t == 4 ? 2 : (t == 5 ? 0 : 1));
        bz = 2 - bx - by;
    }
}

// h(c, d) of the 1-D shift from v[m] (m <= LC + LD): h(c, d) = h(c+1, d-1) + R h(c, d-1).
template <int LC, int LD>
__device__ __forceinline__ void shift_ket(double* v, double R, double* out)
{
#pragma unroll
    for (int d = 0; d <= LD; d++) {
#pragma unroll
        for (int c = 0; c <= LC; c++) out[c * (LD + 1) + d] = v[c];
        if (d < LD) {
#pragma unroll
            for (int c = 0; c < LC + LD - d; c++) v[c] = fma(R, v[c], v[c + 1]);
        }
    }
}

// The VRR table of one direction of one lane, V(n, m) flattened: in registers
// or in shared memory (one column per thread, STRIDE threads).
template <int N, bool REG, int STRIDE>
struct KVTable {
    double p[N];
    __device__ __forceinline__ void bind(double*) {}
    __device__ __forceinline__ double get(int i) const { return p[i]; }
    __device__ __forceinline__ void set(int i, double v) { p[i] = v; }
};
template <int N, int STRIDE>
struct KVTable<N, false, STRIDE> {
    double* p;
    __device__ __forceinline__ void bind(double* smem) { p = smem; }
    __device__ __forceinline__ double get(int i) const { return p[i * STRIDE]; }
    __device__ __forceinline__ void set(int i, double v) { p[i * STRIDE] = v; }
};

// out[c, d] for one a and b exponent bx of one direction:
// the shift to b, sum_k binomial(bx, k) R^(bx - k) V(a + k, m), then to d.
template <int LB, int LC, int LD, typename VT>
__device__ __forceinline__ void krys_row(const VT& V, int a, int bx, double R, double Rk, double* out)
{
    constexpr int M1 = LC + LD + 1;
    const int i = a * M1;
    double v[M1];
    if (LB == 0 || bx == 0) {
#pragma unroll
        for (int m = 0; m < M1; m++) v[m] = V.get(i + m);
    } else if (LB == 1 || bx == 1) {
#pragma unroll
        for (int m = 0; m < M1; m++) v[m] = fma(R, V.get(i + m), V.get(i + M1 + m));
    } else {
        const double R2 = R * R, RR = R + R;
#pragma unroll
        for (int m = 0; m < M1; m++) v[m] = fma(R2, V.get(i + m), fma(RR, V.get(i + M1 + m), V.get(i + 2 * M1 + m)));
    }
    shift_ket<LC, LD>(v, Rk, out);
}

// V(n, m) of one direction from V(0, 0) = v0.
template <int N1, int M1, typename VT>
__device__ __forceinline__ void krys_vrr(double v0, double C, double D, double B10, double B01, double B00, VT& V)
{
    double p[N1], q[N1];  // columns m - 1 and m
    q[0] = v0;
    if (N1 > 1) q[1] = C * v0;
#pragma unroll
    for (int n = 2; n < N1; n++) q[n] = fma(C, q[n - 1], (n - 1) * B10 * q[n - 2]);
#pragma unroll
    for (int n = 0; n < N1; n++) {
        V.set(n * M1, q[n]);
        p[n] = 0.0;
    }
#pragma unroll
    for (int m = 1; m < M1; m++) {
        double t[N1];
#pragma unroll
        for (int n = 0; n < N1; n++) {
            double s = D * q[n];
            if (m > 1) s = fma((m - 1) * B01, p[n], s);
            if (n > 0) s = fma(n * B00, q[n - 1], s);
            t[n] = s;
        }
#pragma unroll
        for (int n = 0; n < N1; n++) {
            p[n] = q[n];
            q[n] = t[n];
            V.set(n * M1 + m, q[n]);
        }
    }
}

// The tables of the three directions at one root (weight, prefactor and S in z).
template <int NR, int N1, int M1, int NS, typename VT>
__device__ __forceinline__ void krys_tables(const double* sc, int root, const double* __restrict__ rtab, VT& Vx, VT& Vy,
                                            VT& Vz)
{
    double x, w;
    rys_root<NR>(sc[KF_T * NS], rtab, root, x, w);
    w *= sc[KF_W * NS];
    const double zx = sc[KF_ZI * NS] * x, ex = sc[KF_EI * NS] * x;  // (rho / zeta) t^2, (rho / eta) t^2
    const double B10 = sc[KF_I2Z * NS] * (1.0 - zx), B01 = sc[KF_I2E * NS] * (1.0 - ex);
    const double B00 = sc[KF_HI * NS] * x;
    double C[3], D[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double PQ = sc[(KF_PQ + k) * NS];
        C[k] = fma(zx, PQ, sc[(KF_PA + k) * NS]);
        D[k] = fma(-ex, PQ, sc[(KF_QC + k) * NS]);
    }
    krys_vrr<N1, M1>(1.0, C[0], D[0], B10, B01, B00, Vx);
    krys_vrr<N1, M1>(1.0, C[1], D[1], B10, B01, B00, Vy);
    krys_vrr<N1, M1>(w, C[2], D[2], B10, B01, B00, Vz);
}

// One exponent tuple of the 1-D table: sum over both binomial shifts (used
// only for records whose components do not share one S).
template <int M1, int STRIDE>
__device__ __forceinline__ double krys_value(const double* V, int a, int b, int c, int d, double R, double Rk)
{
    double s = 0.0;
    for (int k = 0; k <= b; k++) {
        double cb = (k == 0 || k == b) ? 1.0 : (double)b;  // binomial(b, k), b <= 3
        for (int j = 0; j < b - k; j++) cb *= R;
        for (int l = 0; l <= d; l++) {
            double cd = (l == 0 || l == d) ? cb : cb * (double)d;
            for (int j = 0; j < d - l; j++) cd *= Rk;
            s = fma(cd, V[((a + k) * M1 + c + l) * STRIDE], s);
        }
    }
    return s;
}

__device__ __forceinline__ void cart_exps(int l, int i, int& x, int& y, int& z)
{
    const int s = i < 1 ? 0 : (i < 3 ? 1 : 2);
    z = i - s * (s + 1) / 2;
    y = s - z;
    x = l - s;
}

// K_ac of one root with per-component S and component masks.
template <int LA, int LB, int LC, int LD, int STRIDE>
__device__ __noinline__ double krys_masked(const KPartnerRecs& ab, const KPartnerRecs& cd, int jr, int lr,
                                           const KDensity& dm, const double* V, int ca, int cc)
{
    constexpr int N1 = LA + LB + 1, M1 = LC + LD + 1;
    const int spj = __ldg(ab.rec_sp + jr), spl = __ldg(cd.rec_sp + lr);
    const uint64_t mj = __ldg(ab.rec_mask + jr), ml = __ldg(cd.rec_mask + lr);
    const int jsh = __ldg(ab.partner + spj), lsh = __ldg(cd.partner + spl);
    double R[3], Rk[3];
    for (int x = 0; x < 3; x++) {
        R[x] = __ldg(ab.geo + (G_RX + x) * ab.sp_stride + spj);
        Rk[x] = __ldg(cd.geo + (G_RX + x) * cd.sp_stride + spl);
    }
    int a[3], c[3], b[3], d[3];
    cart_exps(LA, ca, a[0], a[1], a[2]);
    cart_exps(LC, cc, c[0], c[1], c[2]);
    double acc = 0.0;
    for (int cb = 0; cb < ncart(LB); cb++) {
        const int ij = ca * ncart(LB) + cb;
        if (!((mj >> ij) & 1ull)) continue;
        const double Sij = __ldg(ab.S + ij * ab.sp_stride + spj);
        const uint32_t jao = __ldg(dm.b_aoinds + jsh + (int64_t)dm.b_count * cb);
        cart_exps(LB, cb, b[0], b[1], b[2]);
        double s = 0.0;
        for (int cdd = 0; cdd < ncart(LD); cdd++) {
            const int kl = cc * ncart(LD) + cdd;
            if (!((ml >> kl) & 1ull)) continue;
            const uint32_t lao = __ldg(dm.d_aoinds + lsh + (int64_t)dm.d_count * cdd);
            cart_exps(LD, cdd, d[0], d[1], d[2]);
            double v = __ldg(cd.S + kl * cd.sp_stride + spl);
            for (int x = 0; x < 3; x++)
                v *= krys_value<M1, STRIDE>(V + x * N1 * M1 * STRIDE, a[x], b[x], c[x], d[x], R[x], Rk[x]);
            s = fma(v, __ldg(dm.D + (int64_t)jao * dm.naos + lao), s);
        }
        acc = fma(s, Sij, acc);
    }
    return acc;
}

template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void krys_lane(const KPartnerRecs& ab, const KPartnerRecs& cd, const KWarpSetup<32>& st, int q,
                                          int root, const KDensity& dm, const double* __restrict__ rtab, double* smem,
                                          double* Kacc)
{
    using S = KRysShape<LA, LB, LC, LD>;
    constexpr int N1 = S::N1, M1 = S::M1;
    constexpr int NB = ncart(LB), ND = ncart(LD), D1 = LD + 1, CD = (LC + 1) * (LD + 1);
    constexpr int NT = N1 * M1;
    KVTable<NT, S::REG, KR_THREADS> Vx, Vy, Vz;
    Vx.bind(smem);
    Vy.bind(smem + NT * KR_THREADS);
    Vz.bind(smem + 2 * NT * KR_THREADS);
    const double* sc = st.sc + q;
    krys_tables<S::NR, N1, M1, 32>(sc, root, rtab, Vx, Vy, Vz);
    if (st.jr[q] < 0) {
        const int jr = ~st.jr[q], lr = st.lr[q];
        if constexpr (S::REG) {
            double copy[3 * NT];
#pragma unroll
            for (int i = 0; i < NT; i++) {
                copy[i] = Vx.get(i);
                copy[NT + i] = Vy.get(i);
                copy[2 * NT + i] = Vz.get(i);
            }
#pragma unroll
            for (int x = 0; x < S::NAC; x++)
                Kacc[x] += krys_masked<LA, LB, LC, LD, 1>(ab, cd, jr, lr, dm, copy, x / ncart(LC), x % ncart(LC));
        } else {
#pragma unroll
            for (int x = 0; x < S::NAC; x++)
                Kacc[x] += krys_masked<LA, LB, LC, LD, KR_THREADS>(ab, cd, jr, lr, dm, smem, x / ncart(LC),
                                                                      x % ncart(LC));
        }
        return;
    }
    const int jsh = st.jsh[q], lsh = st.lsh[q];
    double R[3], Rk[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        R[k] = sc[(KF_AB + k) * 32];
        Rk[k] = sc[(KF_CD + k) * 32];
    }
    uint32_t lao[ND];
#pragma unroll
    for (int k = 0; k < ND; k++) lao[k] = __ldg(dm.d_aoinds + lsh + (int64_t)dm.d_count * k);

    double X[(LA + 1) * CD], Y[(LA + 1) * CD];
    int px = -1, py = -1;
#pragma unroll (S::REG ? NB : 1)
    for (int t = 0; t < NB; t++) {
        int bx, by, bz;
        krys_b<LB>(t, bx, by, bz);
        const uint32_t jao = __ldg(dm.b_aoinds + jsh + (int64_t)dm.b_count * cart_index(by, bz));
        const double* Drow = dm.D + (int64_t)jao * dm.naos;
        double Dv[ND];
#pragma unroll
        for (int k = 0; k < ND; k++) Dv[k] = __ldg(Drow + lao[k]);
        if (bx != px) {
            px = bx;
#pragma unroll
            for (int a = 0; a <= LA; a++) krys_row<LB, LC, LD>(Vx, a, bx, R[0], Rk[0], X + a * CD);
        }
        if (by != py) {
            py = by;
#pragma unroll
            for (int a = 0; a <= LA; a++) krys_row<LB, LC, LD>(Vy, a, by, R[1], Rk[1], Y + a * CD);
        }
#pragma unroll
        for (int az = 0; az <= LA; az++) {
            double Z[CD];
            krys_row<LB, LC, LD>(Vz, az, bz, R[2], Rk[2], Z);
#pragma unroll
            for (int cz = 0; cz <= LC; cz++) {
                double T1[ND];
#pragma unroll
                for (int dy = 0; dy <= LD; dy++)
#pragma unroll
                    for (int dz = 0; dz <= LD - dy; dz++) {
                        const int k = cart_index(dy, dz);
                        T1[k] = Dv[k] * Z[cz * D1 + dz];
                    }
#pragma unroll
                for (int ay = 0; ay <= LA - az; ay++) {
                    const int ax = LA - az - ay;
#pragma unroll
                    for (int cy = 0; cy <= LC - cz; cy++) {
                        const int cx = LC - cz - cy;
                        const int o = cart_index(ay, az) * ncart(LC) + cart_index(cy, cz);
                        double acc = Kacc[o];
#pragma unroll
                        for (int dx = 0; dx <= LD; dx++) {
                            double s = 0.0;
#pragma unroll
                            for (int dy = 0; dy <= LD - dx; dy++) {
                                const int k = cart_index(dy, LD - dx - dy);
                                s = dy == 0 ? T1[k] * Y[ay * CD + cy * D1] : fma(T1[k], Y[ay * CD + cy * D1 + dy], s);
                            }
                            acc = fma(s, X[ax * CD + cx * D1 + dx], acc);
                        }
                        Kacc[o] = acc;
                    }
                }
            }
        }
    }
}

// Quartets a warp sets up together: whole passes of qw quartets, at most
// `most`, and few enough that every warp gets a share.
__device__ __forceinline__ int krys_batch(int total, int warps, int qw, int most)
{
    const int share = (total + warps - 1) / warps;
    return min(most, (share + qw - 1) / qw * qw);
}

// The FP64 quartets (all of them without an FP32 cutoff).
template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(KR_THREADS, (KRysShape<LA, LB, LC, LD>::MINB))
exchange_rys_kernel(KOutBlocks out, KPartnerRecs ab, KPartnerRecs cd, KGroups gab, KGroups gcd, KDensity dm,
                    double maxD, double omega,
                    double thr, double* __restrict__ mat_K, const double* __restrict__ rtab,
                    unsigned long long* __restrict__ qcount, double fp32_cut, double fp32_budget)
{
    using S = KRysShape<LA, LB, LC, LD>;
    constexpr int NAC = S::NAC, NW = KR_THREADS / 32;
    extern __shared__ double krys_smem[];
    __shared__ int s_nl[K_JCHUNK], s_n64[K_JCHUNK], s_c64[K_JCHUNK + 1], s_c32[K_JCHUNK + 1];
    __shared__ double red[NW][NAC];
    __shared__ KWarpSetup<32> s_set[NW];
    double* V = krys_smem + threadIdx.x;
    const KChunk ch{s_nl, s_n64, s_c64, s_c32};
    const int nout = *out.n;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int root = lane % S::NR, slot = lane / S::NR;
    KWarpSetup<32>& set = s_set[warp];
    const bool grouped = gab.of_rec != nullptr;

    for (int o = blockIdx.x; o < nout; o += gridDim.x) {
        const int ish = __ldg(out.ish + o), ksh = __ldg(out.ksh + o);
        const double mD = out.maxD ? __ldg(out.maxD + o) : maxD;
        const int a0 = __ldg(ab.seg + ish), a1 = __ldg(ab.seg + ish + 1);
        const int c0 = __ldg(cd.seg + ksh), c1 = __ldg(cd.seg + ksh + 1);
        const int gc0 = grouped ? __ldg(gcd.seg + ksh) : 0, gc1 = grouped ? __ldg(gcd.seg + ksh + 1) : 0;
        const int gnj = grouped ? __ldg(gab.seg + ish + 1) - __ldg(gab.seg + ish) : 0;
        double Kacc[NAC];
#pragma unroll
        for (int x = 0; x < NAC; x++) Kacc[x] = 0.0;

        for (int jb = a0; jb < a1; jb += K_JCHUNK) {
            const int nj = min(K_JCHUNK, a1 - jb);
            k_chunk_scan(ab, cd, jb, nj, c0, c1, mD, thr, grouped ? 0.0 : fp32_cut, ch, a1 - a0, fp32_budget);
            const int total = s_c64[nj];
            // the contracted kernels count their own FP32 quartets
            if (qcount && !grouped && threadIdx.x == 0) atomicAdd(qcount, (unsigned long long)(total + s_c32[nj]));
            if (grouped) {
                // first FP32 group of l for every j record (the split of exchange_colc_kernel)
                for (int t = threadIdx.x; t < nj; t += KR_THREADS) {
                    const int g = __ldg(gab.of_rec + jb + t);
                    int nl;
                    k_prefixes(__ldg(gab.q + g), gab.qa ? __ldg(gab.qa + g) : 0.0, gcd.q, gab.qa ? gcd.qpre : nullptr,
                               gc0, gc1, mD, thr, fp32_cut, gnj, fp32_budget, nl, s_n64[t]);
                    s_n64[t] += gc0;
                }
                __syncthreads();
            }
            const int batch = krys_batch(total, NW, S::QW, S::BATCH);
            int jj = 0;
            for (int w0 = warp * batch; w0 < total; w0 += NW * batch) {
                const int w = w0 + lane;
                bool mine = lane < min(batch, total - w0);
                int l = 0;
                if (mine) {
                    while (s_c64[jj + 1] <= w) jj++;  // w ascends; s_c64[nj] = total > w
                    l = c0 + w - s_c64[jj];
                    if (grouped) mine = __ldg(gcd.of_rec + l) < s_n64[jj];
                }
                const unsigned taken = __ballot_sync(0xffffffffu, mine);
                const int n = __popc(taken);
                if (grouped && qcount && lane == 0) atomicAdd(qcount, (unsigned long long)n);
                if (mine)
                    krys_setup<false, false, false>(ab, cd, jb + jj, l, omega, set, __popc(taken & ((1u << lane) - 1)));
                __syncwarp();
                if (slot < S::QW)
                    for (int q = slot; q < n; q += S::QW)
                        krys_lane<LA, LB, LC, LD>(ab, cd, set, q, root, dm, rtab, V, Kacc);
                __syncwarp();
            }
            __syncthreads();
        }

#pragma unroll
        for (int x = 0; x < NAC; x++) {
            const double v = warp_sum(Kacc[x]);
            if (lane == 0) red[warp][x] = v;
        }
        __syncthreads();
        if (threadIdx.x < NAC) {
            double s = red[0][threadIdx.x];
#pragma unroll
            for (int w = 1; w < NW; w++) s += red[w][threadIdx.x];
            const int32_t p = __ldg(out.idx + threadIdx.x * out.stride + o);
            if (p >= 0) mat_K[p] += s;
        }
        __syncthreads();
    }
}

// Raise the dynamic shared memory limit of a kernel and ask for the carve-out
// that lets `ctas` of its CTAs be resident (once per device: `done` is a
// static of the caller).
inline int rys_prepare(const void* kernel, int smem, int ctas, std::atomic<unsigned long long>& done)
{
    int dev = 0;
    VLXB_CHECK_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return VLXB_OK;
    cudaFuncAttributes at;
    VLXB_CHECK_CUDA(cudaFuncGetAttributes(&at, kernel));
    VLXB_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    int pct = (int)((ctas * (smem + (int)at.sharedSizeBytes + 1024) * 100ll + 228 * 1024 - 1) / (228 * 1024));
    VLXB_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         pct > 100 ? 100 : pct));
    done.fetch_or(bit, std::memory_order_acq_rel);
    return VLXB_OK;
}

template <int LA, int LB, int LC, int LD>
int launch_exchange_rys(int grid, cudaStream_t st, const KOutBlocks& out, const KPartnerRecs& ab,
                        const KPartnerRecs& cd, const KGroups& gab, const KGroups& gcd, const KDensity& dm, double maxD, double omega, double thr,
                        double* mat_K, unsigned long long* qk, double cut, double budget)
{
    using S = KRysShape<LA, LB, LC, LD>;
    static std::atomic<unsigned long long> done;
    const double* tab = rys_table_device();
    if (!tab) return VLXB_ECUDA;
    const int smem = S::SMEM_ROWS * KR_THREADS * (int)sizeof(double);
    const int rc = rys_prepare((const void*)exchange_rys_kernel<LA, LB, LC, LD>, smem, S::MINB, done);
    if (rc) return rc;
    exchange_rys_kernel<LA, LB, LC, LD><<<grid, KR_THREADS, smem, st>>>(
        out, ab, cd, gab, gcd, dm, maxD, omega, thr, mat_K, tab + rys_offset(S::NR), qk, cut, budget);
    VLXB_CHECK_CUDA(cudaGetLastError());
    return VLXB_OK;
}

}  // namespace vlxb
