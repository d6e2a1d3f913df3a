// Kernel launchers of one class.  The class drivers (classes.cuh) call them;
// they are defined next to their kernels and instantiated in the translation
// units of generated/ (cls_<abcd>_j.cu, cls_<abcd>_k.cu, krys_<ab>.cu), so that
// a kernel's change rebuilds only the units that hold it.
#pragma once
#include "jk_kernels.cuh"

namespace vlxb {

// Exchange kernel of a class.  The thread-per-quartet kernel shares a quartet's
// set-up and recurrences among all its components and wins while its
// straight-line code fits in registers; the Rys kernel repeats part of them per
// root.  10 atoms 4s3p2d, thread / Rys, ms per class call: (PP|PP) 1.3 / 1.8,
// (SD|DS) 2.2 / 2.9, (SP|PD) 2.5 / 3.3 (L = 4); (DP|DS) 2.10 / 2.15, (PD|DS)
// 3.8 / 3.7, (SP|DD) 4.8 / 3.4, (PP|DP) 9.2 / 4.4, (SD|PD) 11.3 / 4.5 (L = 5);
// (DS|DD) 7.2 / 2.6 (L = 6).
__host__ __device__ constexpr bool k_rys(int la, int lb, int lc, int ld) { return la + lb + lc + ld >= 5; }

// FP64 kernel of a Coulomb class: Rys where the thread-per-quartet kernel's
// registers limit it and both Hermite ranges are wide enough to repay the
// set-up per root.  10 atoms 4s3p2d, thread / Rys, ms per class call: (SD|SD)
// 2.0 / 2.1, (PP|PP) 0.72 / 0.78 (L = 4); (SP|DD) 1.7 / 2.5, (DD|SP) 1.18 / 1.27,
// (PD|PP) 1.7 / 1.3, (SD|PD) 3.2 / 2.5 (L = 5); (PP|DD) 1.9 / 1.5, (PD|PD) 5.5 /
// 2.8, (DD|PD) 6.0 / 1.7.
__host__ __device__ constexpr bool j_rys(int la, int lb, int lc, int ld)
{
    return la + lb >= 2 && lc + ld >= 2 && la + lb + lc + ld >= 5;
}

// Pass pm: 0 = FP64, 1 = FP32 quartets; launch_exchange_rys evaluates the FP64
// and launch_exchange_mixed the FP32 quartets of a class.  variant as
// vlxb_setSchedule.
template <int LA, int LB, int LC, int LD>
int launch_coulomb(int variant, int pm, int grid, cudaStream_t st, const JBraRecs& bra, const JKetPairs& ket,
                   double* mat_J, double thr, const BoysTabs& tab, unsigned long long* qc, double cut, double budget);

template <int LA, int LB, int LC, int LD>
int launch_coulomb_rys(int grid, cudaStream_t st, const JBraRecs& bra, const JKetPairs& ket, double* mat_J, double thr,
                       unsigned long long* qc, double cut, double budget);

// out[k * gstride + o], k = 0..5: bra-centre derivatives.
template <int LA, int LB, int LC, int LD>
int launch_coulomb_grad(int pm, int grid, cudaStream_t st, const JBraRecs& bra, const JKetPairs& ket, double* out,
                        int64_t gstride, double thr, double cut);

// Partner groups of a contracted kernel: the records of one first primitive
// shell whose partners belong to one contracted shell.
struct KGroups {
    const int* seg;          // [n_first + 1] group offsets by first primitive shell
    const double* q;         // max member q, descending inside a segment
    const int32_t* beg;      // first member
    const int32_t* cnt;      // member count
    const int32_t* msp;      // member shell pair
    const double* mq;        // member q
    const double* msu;       // member uniform S, or NaN (member alone in its group)
    const uint64_t* mmask;   // member component mask
    const double* qa;        // sum over members of |q| times HRR growth (FP32 error budget), or null
    const double* qpre;      // inclusive prefix sum of qa, or null
    const int32_t* of_rec;   // group of every record
};

template <int LA, int LB, int LC, int LD>
int launch_exchange_thread(int pm, int grid, cudaStream_t st, const KOutBlocks& out, const KPartnerRecs& ab,
                           const KPartnerRecs& cd, const KDensity& dm, double maxD, double omega, double thr,
                           double* mat_K, const BoysTabs& tab, unsigned long long* qk, double cut, double budget);

// Kernel of a Rys class's FP32 quartets: 0 thread per quartet, else a column
// kernel (1 = plan kind 0, 7 = packed kind 4; 3 / 4 = contracted partners,
// kinds 0 / 1), each class's fastest there.  They keep their FP32 arithmetic:
// a mixed-precision result carries the rounding of its FP32 quartets (2e-9 of
// K on 8 atoms), which another evaluation order would replace by a different
// one of the same size.  The contracted kernels split FP64 from FP32 by partner
// groups; the Rys kernel then leaves out the quartets of their FP32 groups.
__host__ __device__ constexpr int k_mixed(int la, int lb, int lc, int ld)
{
    switch (la * 1000 + lb * 100 + lc * 10 + ld) {
        case 2222: return 1;
        case 1222: case 2122: case 1122: case 2121: return 3;
        case 2221: case 2220: return 4;
        case 1221: case 222: case 1212: return 7;
        default: return 0;
    }
}
__host__ __device__ constexpr bool k_contracted(int la, int lb, int lc, int ld)
{
    return k_mixed(la, lb, lc, ld) == 3 || k_mixed(la, lb, lc, ld) == 4;
}

template <int LA, int LB, int LC, int LD>
int launch_exchange_mixed(int grid, cudaStream_t st, const KOutBlocks& out, const KPartnerRecs& ab,
                          const KPartnerRecs& cd, const KGroups& gab, const KGroups& gcd, const KDensity& dm,
                          double maxD, double omega, double thr, double* mat_K, const BoysTabs& tab,
                          unsigned long long* qk, double cut, double budget);

template <int LA, int LB, int LC, int LD>
int launch_exchange_rys(int grid, cudaStream_t st, const KOutBlocks& out, const KPartnerRecs& ab,
                        const KPartnerRecs& cd, const KGroups& gab, const KGroups& gcd, const KDensity& dm,
                        double maxD, double omega, double thr, double* mat_K, unsigned long long* qk, double cut,
                        double budget);

// D_ik per (i, k) block of the exchange gradient: rows / columns of the (i, k)
// components in the AO density (single-molecule calls).
struct KGradBlockD {
    const uint32_t* a_aoinds;
    uint32_t a_count;
    const uint32_t* c_aoinds;
    uint32_t c_count;
    int same_type;  // a == c: the diagonal entries i == k have weight 1
};

template <int LA, int LB, int LC, int LD>
int launch_exchange_grad(int grid, cudaStream_t st, const KOutBlocks& out, const KPartnerRecs& ab,
                         const KPartnerRecs& cd, const KDensity& dm, const KGradBlockD& bd, double maxD, double omega,
                         double thr, double* grad, int64_t gstride);

}  // namespace vlxb
