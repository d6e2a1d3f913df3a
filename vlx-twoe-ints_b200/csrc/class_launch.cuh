// Launchers of the generated (straight-line) kernels of one class.
#pragma once
#include <atomic>

#include "col_kernels.cuh"
#include "engine.cuh"
#include "jtma_kernels.cuh"
#include "launch.cuh"
#include "md_kernels.cuh"

namespace vlxb {

// The staged Coulomb kernel's shared memory exceeds the 48 KB default for
// kets with d functions: raise the limit once per device for each
// instantiation.
template <int LA, int LB, int LC, int LD, int PM>
int jtma_prepare_launch()
{
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    VLXB_CHECK_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return VLXB_OK;
    VLXB_CHECK_CUDA(cudaFuncSetAttribute(coulomb_tma_kernel<LA, LB, LC, LD, PM>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)JTmaShape<LC, LD>::SMEM));
    done.fetch_or(bit, std::memory_order_acq_rel);
    return VLXB_OK;
}

template <int LA, int LB, int LC, int LD, int PM>
int launch_coulomb_pass(int variant, int grid, cudaStream_t st, const JBraRecs& bra, const JKetPairs& ket,
                        double* mat_J, double thr, const BoysTabs& tab, unsigned long long* qc, double cut,
                        double budget)
{
    if (variant == 2) {
        coulomb_md_kernel<LA, LB, LC, LD, PM><<<grid, MD_THREADS, 0, st>>>(bra, ket, mat_J, thr, tab, qc, cut, budget);
    } else if (variant == 3) {
        unsigned long long* kerr = kernel_errors_device();
        if (!kerr) return VLXB_ECUDA;
        const int rc = jtma_prepare_launch<LA, LB, LC, LD, PM>();
        if (rc) return rc;
        coulomb_tma_kernel<LA, LB, LC, LD, PM><<<grid, JT_TILE, JTmaShape<LC, LD>::SMEM, st>>>(
            bra, ket, mat_J, thr, tab, qc, cut, budget, kerr);
    } else if (variant == 1) {
        coulomb_col_kernel<LA, LB, LC, LD, PM><<<grid, J_THREADS, 0, st>>>(bra, ket, mat_J, thr, tab, qc, cut, budget);
    } else {
        coulomb_kernel<LA, LB, LC, LD, PM><<<grid, J_THREADS, 0, st>>>(bra, ket, mat_J, thr, tab, qc, cut, budget);
    }
    VLXB_CHECK_CUDA(cudaGetLastError());
    return VLXB_OK;
}

template <int LA, int LB, int LC, int LD>
int launch_coulomb(int variant, int pm, int grid, cudaStream_t st, const JBraRecs& bra, const JKetPairs& ket,
                   double* mat_J, double thr, const BoysTabs& tab, unsigned long long* qc, double cut, double budget)
{
    if (pm == 1)
        return launch_coulomb_pass<LA, LB, LC, LD, 1>(variant, grid, st, bra, ket, mat_J, thr, tab, qc, cut, budget);
    if constexpr (j_rys(LA, LB, LC, LD))
        return VLXB_EINVAL;  // launch_coulomb_rys
    else
        return launch_coulomb_pass<LA, LB, LC, LD, 0>(variant, grid, st, bra, ket, mat_J, thr, tab, qc, cut, budget);
}

template <int LA, int LB, int LC, int LD>
int launch_exchange_thread(int pm, int grid, cudaStream_t st, const KOutBlocks& out, const KPartnerRecs& ab,
                           const KPartnerRecs& cd, const KDensity& dm, double maxD, double omega, double thr,
                           double* mat_K, const BoysTabs& tab, unsigned long long* qk, double cut, double budget)
{
    if (pm == 0)
        exchange_kernel<LA, LB, LC, LD, 0><<<grid, K_THREADS, 0, st>>>(out, ab, cd, dm, maxD, omega, thr, mat_K, tab,
                                                                       qk, cut, budget);
    else
        exchange_kernel<LA, LB, LC, LD, 1><<<grid, K_THREADS, 0, st>>>(out, ab, cd, dm, maxD, omega, thr, mat_K, tab,
                                                                       qk, cut, budget);
    VLXB_CHECK_CUDA(cudaGetLastError());
    return VLXB_OK;
}

template <int LA, int LB, int LC, int LD>
int launch_exchange_mixed(int grid, cudaStream_t st, const KOutBlocks& out, const KPartnerRecs& ab,
                          const KPartnerRecs& cd, const KGroups& gab, const KGroups& gcd, const KDensity& dm,
                          double maxD, double omega, double thr, double* mat_K, const BoysTabs& tab,
                          unsigned long long* qk, double cut, double budget)
{
    constexpr int V = k_mixed(LA, LB, LC, LD);
    if constexpr (V == 3 || V == 4)
        exchange_colc_kernel<LA, LB, LC, LD, V - 3><<<grid, K_THREADS, 0, st>>>(
            out, ab, cd, gab, gcd, dm, maxD, omega, thr, mat_K, tab, qk, cut, budget);
    else if constexpr (V != 0)
        exchange_col_kernel<LA, LB, LC, LD, (V == 7 ? 4 : 0)><<<grid, K_THREADS, 0, st>>>(
            out, ab, cd, dm, maxD, omega, thr, mat_K, tab, cut, budget);
    else
        exchange_kernel<LA, LB, LC, LD, 1><<<grid, K_THREADS, 0, st>>>(out, ab, cd, dm, maxD, omega, thr, mat_K, tab,
                                                                       qk, cut, budget);
    VLXB_CHECK_CUDA(cudaGetLastError());
    return VLXB_OK;
}

}  // namespace vlxb
