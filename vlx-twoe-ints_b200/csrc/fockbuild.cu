// One call for the class calls of a whole J / K build (or of its nuclear
// gradient).  A class call regroups its lists on the device before its
// integral kernel; the 90 classes of a build do that 225 times for only 27
// distinct lists.  Here every list is prepared once: two atoms 4s3p2d, 4735
// device operations and 25.5 ms per build become about 700 and 4.0 ms.
#include "classes.cuh"
#include "../../include/vlxb.h"

namespace vlxb {

int dispatch_coulomb(int cls, bool grad, const CoulombArgs& a, int64_t gstride, cudaStream_t st);
int dispatch_exchange(int cls, bool grad, const ExchangeArgs& a, int64_t gstride, cudaStream_t st);

static int run_build(const VlxbFockBuild& b, PrepShare& share, cudaStream_t st)
{
    static const int pair_ab[6][2] = {{0, 0}, {0, 1}, {0, 2}, {1, 1}, {1, 2}, {2, 2}};
    const bool batched = b.n_mol > 0;
    int bit = 0;
    for (int x = 0; x < 6; x++)
        for (int y = 0; y < 6; y++, bit++) {
            if (!((b.j_classes >> bit) & 1ull)) continue;
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
                A.aoinds_col[l] = b.prim_aocols[l];
                A.count[l] = b.prim_count[l];
            }
            A.maxD = b.maxD[bd];
            A.D = b.D;
            A.naos = b.naos;
            A.D_stride = b.D_stride;
            A.Q_ab = b.kp_Q[p]; A.pdata_ab = b.kp_pdata[p]; A.Dinds_ab = b.kp_Dinds[p];
            A.displs_ab = b.kp_displs[p]; A.counts_ab = b.kp_counts[p];
            A.Q_cd = b.kp_Q[q]; A.pdata_cd = b.kp_pdata[q]; A.Dinds_cd = b.kp_Dinds[q];
            A.displs_cd = b.kp_displs[q]; A.counts_cd = b.kp_counts[q];
            A.omega = b.omega;
            A.thr = b.thr;
            if (batched) {
                A.prim_mol_a = b.prim_mol[la];
                A.maxD_mol = b.maxD_mol[bd];
                if (!A.prim_mol_a || !A.maxD_mol) return VLXB_EINVAL;
            }
            A.share = &share;
            const int rc = dispatch_exchange(la * 27 + lb * 9 + lc * 3 + ld, b.gradient != 0, A, (int64_t)b.grad_stride, st);
            if (rc) return rc;
        }
    return VLXB_OK;
}

}  // namespace vlxb

extern "C" int vlxb_fockBuild(const VlxbFockBuild* b, void* stream)
{
    if (!b || b->n_mol < 0 || b->grad_stride > (uint64_t)INT64_MAX || (b->gradient && b->n_mol > 0)) return VLXB_EINVAL;
    vlxb::PrepShare share((cudaStream_t)stream);
    share.prepare_only = true;  // every list first: a call short of memory then leaves the outputs as they were
    int rc = vlxb::run_build(*b, share, (cudaStream_t)stream);
    if (rc) return rc;
    share.prepare_only = false;
    return vlxb::run_build(*b, share, (cudaStream_t)stream);
}
