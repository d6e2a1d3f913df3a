// One call for the class calls of a whole J / K build (or of its nuclear
// gradient).  A class call regroups its lists on the device before its
// integral kernel; the 90 classes of a build do that 225 times for only 27
// distinct lists.  Here every list is prepared once: two atoms 1s1p1d, 4735
// device operations and 22 ms per build become 284 and 1.1 ms.
#include <algorithm>

#include "classes.cuh"
#include "fork.cuh"
#include "rys.cuh"
#include "../../include/vlxb.h"

namespace vlxb {

int dispatch_coulomb(int cls, bool grad, const CoulombArgs& a, int64_t gstride, cudaStream_t st);
int dispatch_exchange(int cls, bool grad, const ExchangeArgs& a, int64_t gstride, cudaStream_t st);

constexpr int pair_ab[6][2] = {{0, 0}, {0, 1}, {0, 2}, {1, 1}, {1, 2}, {2, 2}};

// Whether a batch names the molecules that its classes ask for (as
// vlxb_coulombBatch and vlxb_exchangeBatch; an empty Coulomb list asks for none).
static bool batch_complete(const VlxbFockBuild& b)
{
    for (int x = 0; x < 6; x++) {
        const int la = pair_ab[x][0], lb = pair_ab[x][1];
        for (int y = 0; y < 6; y++) {
            const int lc = pair_ab[y][0], ld = pair_ab[y][1];
            if (((b.j_classes >> (x * 6 + y)) & 1ull) && b.j_count[la * 3 + lb] && b.j_count[lc * 3 + ld] &&
                (!b.prim_mol[la] || !b.prim_mol[lc]))
                return false;
        }
        for (int bd = 0; bd < 9; bd++)
            if (((b.k_classes >> (x * 9 + bd)) & 1ull) && (!b.prim_mol[la] || !b.maxD_mol[bd])) return false;
    }
    return true;
}

static int run_build(const VlxbFockBuild& b, PrepShare& share, Fork* fork, cudaStream_t stream)
{
    const bool batched = b.n_mol > 0;
    int bit = 0;
    for (int x = 0; x < 6; x++)
        for (int y = 0; y < 6; y++, bit++) {
            if (!((b.j_classes >> bit) & 1ull)) continue;
            const cudaStream_t st = fork ? fork->at(x) : stream;
            const int la = pair_ab[x][0], lb = pair_ab[x][1], lc = pair_ab[y][0], ld = pair_ab[y][1];
            const int p = la * 3 + lb, q = lc * 3 + ld;
            CoulombArgs A{};
            A.mat_J = b.mat_J[p];
            for (int l = 0; l < 3; l++) {
                A.info[l] = b.prim_info[l];
                A.count[l] = b.prim_count[l];
            }
            A.ab_first = b.j_first[p]; A.ab_second = b.j_second[p]; A.ab_pdata = b.j_pdata[p]; A.ab_Q = b.j_Q[p];
            A.n_ab = b.j_count[p];
            A.cd_first = b.j_first[q]; A.cd_second = b.j_second[q]; A.cd_pdata = b.j_pdata[q]; A.cd_Q = b.j_Q[q];
            A.cd_D = b.j_D[q];
            A.n_cd = b.j_count[q];
            A.thr = b.thr;
            if (batched) {
                A.prim_mol_a = b.prim_mol[la];
                A.prim_mol_c = b.prim_mol[lc];
                A.n_mol = b.n_mol;
            }
            A.share = &share;
            const int rc = dispatch_coulomb(la * 27 + lb * 9 + lc * 3 + ld, b.gradient != 0, A, (int64_t)b.grad_stride, st);
            if (rc) return rc;
        }
    bit = 0;
    for (int x = 0; x < 6; x++)
        for (int bd = 0; bd < 9; bd++, bit++) {
            if (!((b.k_classes >> bit) & 1ull)) continue;
            const cudaStream_t st = fork ? fork->at(x + 2) : stream;
            const int la = pair_ab[x][0], lc = pair_ab[x][1], lb = bd / 3, ld = bd % 3;
            const int o = la * 3 + lc, p = la * 3 + lb, q = lc * 3 + ld;
            ExchangeArgs A{};
            A.mat_K = b.mat_K[o];
            A.pair_i = b.k_i[o];
            A.pair_k = b.k_k[o];
            A.n_ik = b.k_count[o];
            for (int l = 0; l < 3; l++) {
                A.info[l] = b.prim_info[l];
                A.aoinds[l] = b.prim_aoinds[l];
                if (batched) A.aoinds_col[l] = b.prim_aocols[l];
                A.count[l] = b.prim_count[l];
            }
            A.maxD = b.maxD[bd];
            A.D = b.D;
            A.naos = b.naos;
            if (batched) A.D_stride = b.D_stride;
            A.Q_ab = b.kp_Q[p]; A.pdata_ab = b.kp_pdata[p]; A.Dinds_ab = b.kp_Dinds[p];
            A.displs_ab = b.kp_displs[p]; A.counts_ab = b.kp_counts[p];
            A.Q_cd = b.kp_Q[q]; A.pdata_cd = b.kp_pdata[q]; A.Dinds_cd = b.kp_Dinds[q];
            A.displs_cd = b.kp_displs[q]; A.counts_cd = b.kp_counts[q];
            A.omega = b.omega;
            A.thr = b.thr;
            if (batched) {
                A.prim_mol_a = b.prim_mol[la];
                A.maxD_mol = b.maxD_mol[bd];
            }
            A.share = &share;
            const int rc = dispatch_exchange(la * 27 + lb * 9 + lc * 3 + ld, b.gradient != 0, A, (int64_t)b.grad_stride, st);
            if (rc) return rc;
        }
    return VLXB_OK;
}

// Scratch of the shared preparations, from the sizes of the lists' dense bounds:
// a partner list reserves its whole (shell, shell, component) table.  A class
// call holds two such lists at a time, a shared build nine, which grows with
// the square of the primitive count: 14 atoms 4s3p2d 0.1 GB, but a union of 64
// molecules of 3 to 8 atoms 53 GB in FP64 and 157 GB in mixed precision.
static uint64_t share_bytes(const VlxbFockBuild& b, const Fp32Settings& fp32)
{
    bool kp[9] = {}, j[9] = {};
    for (int x = 0; x < 6; x++) {
        for (int y = 0; y < 6; y++)
            if ((b.j_classes >> (x * 6 + y)) & 1ull)
                j[pair_ab[x][0] * 3 + pair_ab[x][1]] = j[pair_ab[y][0] * 3 + pair_ab[y][1]] = true;
        for (int bd = 0; bd < 9; bd++)
            if ((b.k_classes >> (x * 9 + bd)) & 1ull)
                kp[pair_ab[x][0] * 3 + bd / 3] = kp[pair_ab[x][1] * 3 + bd % 3] = true;
    }
    uint64_t bytes = 0;
    for (int p = 0; p < 9; p++) {
        const int la = p / 3, lb = p % 3;
        const uint64_t nxy = (uint64_t)ncart(la) * ncart(lb), ntab = (uint64_t)b.prim_count[la] * b.prim_count[lb];
        if (kp[p]) {
            uint64_t rec = 60;  // records before and after the sort, S, list positions
            if (fp32.cut > 0.0) rec += (k_pair_contracted(la, lb) ? 150 : 0) + (fp32.budget > 0.0 ? 32 : 0);
            bytes += ntab * (130 + rec * nxy);
        }
        if (j[p]) bytes += ntab * 8 + std::min<uint64_t>(b.j_count[p], ntab) * (250 + 16 * (4 * nxy + 35));
    }
    return bytes;
}

// Above this (of 180 GB) a build goes class by class: its integral kernels take
// minutes, beside which the repeated preparations are nothing.
constexpr uint64_t SHARE_MAX_BYTES = 40ull << 30;

}  // namespace vlxb

extern "C" int vlxb_fockBuild(const VlxbFockBuild* b, void* stream)
{
    if (!b || b->n_mol < 0 || b->grad_stride > (uint64_t)INT64_MAX || (b->gradient && b->n_mol > 0)) return VLXB_EINVAL;
    if (b->n_mol > 0 && !vlxb::batch_complete(*b)) return VLXB_EINVAL;
    const vlxb::Fp32Settings fp32 = vlxb::fp32_settings();
    if (vlxb::share_bytes(*b, fp32) > vlxb::SHARE_MAX_BYTES) return VLXB_ENOMEM;
    if (!vlxb::rys_table_device()) return VLXB_ECUDA;  // uploaded before any kernel of the build is queued
    const cudaStream_t st = (cudaStream_t)stream;
    vlxb::PrepShare share(st, fp32);
    share.prepare_only = true;  // every list first: a call short of memory then leaves the outputs as they were
    int rc = vlxb::run_build(*b, share, nullptr, st);
    if (rc) return rc;
    share.prepare_only = false;
    uint64_t outputs = 0;
    for (int p = 0; p < 9; p++) outputs += (uint64_t)b->j_count[p] + b->k_count[p];
    vlxb::Fork fork(st, outputs);  // joined before the preparations are handed back on `st`
    rc = vlxb::run_build(*b, share, &fork, st);
    const int jc = fork.join();
    if (!rc) rc = jc;
    // a launch may fail for memory too (a kernel's code or stack): outputs have
    // been added to by then, so it must not read as "nothing done"
    return rc == VLXB_ENOMEM ? VLXB_ECUDA : rc;
}
