// Per-class host drivers: regroup the caller's lists on the device, then
// launch the class's integral kernel, all on the caller's stream.
#pragma once
#include "engine.cuh"
#include "launch.cuh"

namespace vlxb {

struct CoulombArgs {
    double* mat_J;
    const double* info[4];  // prim_info by angular momentum (s, p, d, f)
    uint32_t count[4];      // prim_count by angular momentum
    const double* cd_D;
    const double* ab_Q;
    const double* cd_Q;
    const uint32_t* ab_first;
    const uint32_t* ab_second;
    const double* ab_pdata;
    uint32_t n_ab;
    const uint32_t* cd_first;
    const uint32_t* cd_second;
    const double* cd_pdata;
    uint32_t n_cd;
    double thr;
    // batched calls over several molecules (null / 0 for a class call): the
    // molecule of every primitive of types a and c; a bra pairs only with
    // kets of its own molecule
    const int32_t* prim_mol_a;
    const int32_t* prim_mol_c;
    int n_mol;
    PrepShare* share;  // preparations shared with the other classes of a build, or null
};

struct ExchangeArgs {
    double* mat_K;
    const uint32_t* pair_i;
    const uint32_t* pair_k;
    uint32_t n_ik;
    const double* info[4];
    const uint32_t* aoinds[4];
    uint32_t count[4];
    double maxD;
    const double* D;
    uint32_t naos;
    const double *Q_ab, *Q_cd;
    const uint32_t *Dinds_ab, *Dinds_cd;
    const uint32_t *displs_ab, *displs_cd;
    const uint32_t *counts_ab, *counts_cd;
    const double *pdata_ab, *pdata_cd;
    double omega;
    double thr;
    // batched calls over several molecules (all null / 0 for a class call):
    const uint32_t* aoinds_col[4];  // density column index per prim component (default: aoinds)
    uint32_t D_stride;              // row stride of D (default: naos)
    uint32_t key_naos;              // bound on the AO indices in aoinds (default: naos)
    const int32_t* prim_mol_a;      // molecule of every type-a primitive
    const double* maxD_mol;         // [molecules] max |D| bound of each molecule
    PrepShare* share;               // as for CoulombArgs
};

// The list of type pair (LA, LB) grouped by shell pair.
template <int LA, int LB>
int group_jlist(Arena& ar, PrepShare* sh, const CoulombArgs& a, const uint32_t* first, const uint32_t* second,
                uint32_t n, PairGroups& g)
{
    constexpr int P = LA * 3 + LB;
    if (!sh || !sh->has_jgrp[P]) {
        const int rc = group_flat(ar, ncart(LA), ncart(LB), (int)a.count[LA], (int)a.count[LB], first, second, n,
                                  a.info[LA], a.count[LA], a.info[LB], a.count[LB], g);
        if (rc) return rc;
        if (sh) {
            sh->jgrp[P] = g;
            sh->has_jgrp[P] = true;
        }
    } else {
        g = sh->jgrp[P];
    }
    return VLXB_OK;
}

// Bra records of a Coulomb class (mol: molecule of every record, batched calls).
template <int LA, int LB>
int prepare_jbra(Arena& ar, const CoulombArgs& a, bool batched, PairGroups& g, int32_t*& mol)
{
    constexpr int P = LA * 3 + LB;
    PrepShare* sh = a.share;
    if (sh && sh->has_jbra[P]) {
        g = sh->jbra[P];
        mol = sh->jmol[P];
        return VLXB_OK;
    }
    int rc = group_jlist<LA, LB>(ar, sh, a, a.ab_first, a.ab_second, a.n_ab, g);
    if (rc) return rc;
    rc = make_records(ar, ncart(LA) * ncart(LB), g, a.ab_Q, a.n_ab);
    if (rc) return rc;
    mol = nullptr;
    if (batched) {
        rc = bra_record_mol(ar, g, a.prim_mol_a, &mol);
        if (rc) return rc;
    }
    if (sh) {
        sh->jbra[P] = g;
        sh->jmol[P] = mol;
        sh->has_jbra[P] = true;
    }
    return VLXB_OK;
}

// Sorted kets of a Coulomb class.
template <int LC, int LD>
int prepare_jket(Arena& ar, const CoulombArgs& a, bool batched, bool hermite, bool budget, JKetData& kd)
{
    constexpr int P = LC * 3 + LD;
    PrepShare* sh = a.share;
    if (sh && sh->has_jket[P]) {
        kd = sh->jket[P];
        return VLXB_OK;
    }
    PairGroups g;
    int rc = group_jlist<LC, LD>(ar, sh, a, a.cd_first, a.cd_second, a.n_cd, g);
    if (rc) return rc;
    rc = jket_prepare<LC, LD>(ar, g, a.cd_first, a.cd_second, a.cd_D, a.cd_Q, a.cd_pdata, kd,
                              batched ? a.prim_mol_c : nullptr, batched ? a.n_mol : 0, hermite || sh != nullptr);
    if (rc) return rc;
    if (budget) {
        rc = budget_prefix_kets(ar, kd, LD);
        if (rc) return rc;
    }
    if (sh) {
        sh->jket[P] = kd;
        sh->has_jket[P] = true;
    }
    return VLXB_OK;
}

// Coulomb class call on a given arena (pool, static or measuring) with given
// Boys tables and quartet counter (may be null).  G = 1: the bra-centre
// derivatives of J instead, written to a.mat_J[k * gstride + o], k = 0..5.
template <int LA, int LB, int LC, int LD, int G = 0>
int run_coulomb_impl(const CoulombArgs& a, cudaStream_t st, Arena& ar, const BoysTabs& tab,
                     unsigned long long* qc, const Fp32Settings& fp32, int64_t gstride = 0)
{
    if (a.n_ab == 0 || a.n_cd == 0) return VLXB_OK;
    if (!a.mat_J || !a.cd_D || !a.ab_Q || !a.cd_Q || !a.ab_first || !a.ab_second || !a.ab_pdata || !a.cd_first ||
        !a.cd_second || !a.cd_pdata)
        return VLXB_EINVAL;
    const int L4[4] = {LA, LB, LC, LD};
    for (int t = 0; t < 4; t++)
        if (!a.info[L4[t]] || a.count[L4[t]] == 0) return VLXB_EINVAL;
    if (!(a.thr >= 0.0)) return VLXB_EINVAL;
    if (G && gstride < (int64_t)a.n_ab) return VLXB_EINVAL;
    if (!tab.f64 || !tab.f32) return VLXB_ECUDA;
    const bool batched = a.prim_mol_a && a.prim_mol_c && a.n_mol > 0;
    const int jvar = schedule_get(0, LA, LB, LC, LD);
    // the Rys and McMurchie-Davidson kernels read the Hermite ket density
    const bool hermite = G || j_rys(LA, LB, LC, LD) || jvar == 2;
    const double cut = fp32.cut, budget = G ? 0.0 : fp32.budget;
    PairGroups gb;
    JKetData kd;
    int32_t* bmol = nullptr;
    int rc = prepare_jbra<LA, LB>(ar, a, batched, gb, bmol);
    if (rc) return rc;
    rc = prepare_jket<LC, LD>(ar, a, batched, hermite, budget > 0.0, kd);
    if (rc) return rc;
    if (ar.failed()) return VLXB_ENOMEM;
    if (ar.measuring() || (a.share && a.share->prepare_only)) return VLXB_OK;
    JBraRecs bra{gb.rec_sp, gb.rec_q, gb.rec_mask, gb.n_rec, gb.geo, gb.entry, gb.sp_stride, a.ab_pdata, bmol};
    JKetPairs ket{kd.geo, kd.tmax, kd.tmin, kd.Dpp, kd.Dm, kd.Qc, kd.Dc, kd.stride, kd.n, batched ? kd.seg : nullptr,
                  kd.Dh, kd.tpre};
    int grid = launch_grid_limit();
    if ((int64_t)grid > (int64_t)a.n_ab) grid = (int)a.n_ab;
    for (int pm = 0; pm < (cut > 0.0 ? 2 : 1); pm++) {
        if constexpr (G == 1)
            rc = launch_coulomb_grad<LA, LB, LC, LD>(pm, grid, st, bra, ket, a.mat_J, gstride, a.thr, cut);
        else if (j_rys(LA, LB, LC, LD) && pm == 0) {
            if constexpr (j_rys(LA, LB, LC, LD))
                rc = launch_coulomb_rys<LA, LB, LC, LD>(grid, st, bra, ket, a.mat_J, a.thr, qc, cut, budget);
        } else {
            rc = launch_coulomb<LA, LB, LC, LD>(jvar, pm, grid, st, bra, ket, a.mat_J, a.thr, tab, qc, cut, budget);
        }
        if (rc) return rc;
        note_launches();
    }
    return VLXB_OK;
}

template <int LA, int LB, int LC, int LD>
int run_coulomb(const CoulombArgs& a, cudaStream_t st)
{
    if (a.n_ab == 0 || a.n_cd == 0) return VLXB_OK;
    int rc = ensure_pool_configured();
    if (rc) return rc;
    const BoysTabs tab{boys_table_device(), boys_table32_device()};
    if (!tab.f64 || !tab.f32) return VLXB_ECUDA;
    if (a.share)
        return run_coulomb_impl<LA, LB, LC, LD>(a, st, a.share->ar, tab, quartet_counters_device(), a.share->fp32);
    Arena ar(st);
    return run_coulomb_impl<LA, LB, LC, LD>(a, st, ar, tab, quartet_counters_device(), fp32_settings());
}

// Bra-centre derivatives of one Coulomb class: grad[k * gstride + o] +=
// d mat_J[o] / d (A_x, A_y, A_z, B_x, B_y, B_z)[k], ket held fixed.
template <int LA, int LB, int LC, int LD>
int run_coulomb_grad(const CoulombArgs& a, int64_t gstride, cudaStream_t st)
{
    if (a.n_ab == 0 || a.n_cd == 0) return VLXB_OK;
    int rc = ensure_pool_configured();
    if (rc) return rc;
    const BoysTabs tab{boys_table_device(), boys_table32_device()};
    if (!tab.f64 || !tab.f32) return VLXB_ECUDA;
    if (a.share)
        return run_coulomb_impl<LA, LB, LC, LD, 1>(a, st, a.share->ar, tab, nullptr, a.share->fp32, gstride);
    Arena ar(st);
    return run_coulomb_impl<LA, LB, LC, LD, 1>(a, st, ar, tab, nullptr, fp32_settings(), gstride);
}

// Whether a pair of types is a side of some class whose FP32 quartets run on a
// contracted kernel.
constexpr bool k_pair_contracted(int la, int lb)
{
    for (int x = 0; x < 3; x++)
        for (int y = 0; y < 3; y++)
            if ((la <= x && k_contracted(la, lb, x, y)) || (x <= la && k_contracted(x, y, la, lb))) return true;
    return false;
}

// Partner records of type pair (LX, LY) from its CSR list; with FP32 on, the
// partner groups where a class needs them and the error budget's prefix sums.
template <int LX, int LY>
int prepare_kpart(Arena& ar, const ExchangeArgs& a, const uint32_t* displs, const uint32_t* counts,
                  const uint32_t* Dinds, const double* Q, const double* pdata, const Fp32Settings& fp32,
                  bool contracted, PairGroups& g)
{
    constexpr int P = LX * 3 + LY, NX = ncart(LX), NY = ncart(LY);
    PrepShare* sh = a.share;
    if (sh && sh->has_kpart[P]) {
        g = sh->kpart[P];
        return VLXB_OK;
    }
    const int npx = (int)a.count[LX], npy = (int)a.count[LY];
    int rc = group_csr(ar, NX, NY, npx, npy, displs, counts, Dinds, (int64_t)npx * npy, a.info[LX], a.count[LX],
                       a.info[LY], a.count[LY], g);
    if (rc) return rc;
    rc = make_records(ar, NX * NY, g, Q, (int64_t)npx * npy * NX * NY);
    if (rc) return rc;
    rc = segment_records(ar, NX * NY, npx, npy, g, pdata);
    if (rc) return rc;
    if (fp32.cut > 0.0 && (sh ? k_pair_contracted(LX, LY) : contracted)) {
        rc = contract_groups(ar, npx, g, a.aoinds[LY], a.key_naos ? a.key_naos : a.naos);
        if (rc) return rc;
    }
    if (fp32.budget > 0.0) {
        // after contract_groups: groups get their amplified sums too
        rc = budget_prefix_records(ar, g, npx, LY);
        if (rc) return rc;
    }
    if (sh) {
        sh->kpart[P] = g;
        sh->has_kpart[P] = true;
    }
    return VLXB_OK;
}

// Output blocks and both sides' partner records of an exchange class.
template <int LA, int LB, int LC, int LD>
int prepare_exchange(Arena& ar, const ExchangeArgs& a, const Fp32Settings& fp32, KOutData& ko, PairGroups& gab,
                     PairGroups& gcd)
{
    constexpr int P = LA * 3 + LC;
    constexpr bool CONTRACTED = k_rys(LA, LB, LC, LD) && k_contracted(LA, LB, LC, LD);
    PrepShare* sh = a.share;
    int rc;
    if (sh && sh->has_kout[P]) {
        ko = sh->kout[P];
    } else {
        rc = kout_prepare(ar, ncart(LA), ncart(LC), (int)a.count[LA], (int)a.count[LC], a.pair_i, a.pair_k, a.n_ik, ko);
        if (rc) return rc;
        if (sh) {
            sh->kout[P] = ko;
            sh->has_kout[P] = true;
        }
    }
    rc = prepare_kpart<LA, LB>(ar, a, a.displs_ab, a.counts_ab, a.Dinds_ab, a.Q_ab, a.pdata_ab, fp32, CONTRACTED, gab);
    if (rc) return rc;
    if (LA == LC && LB == LD && a.Q_ab == a.Q_cd && a.Dinds_ab == a.Dinds_cd && a.displs_ab == a.displs_cd &&
        a.counts_ab == a.counts_cd && a.pdata_ab == a.pdata_cd) {
        gcd = gab;
        return VLXB_OK;
    }
    return prepare_kpart<LC, LD>(ar, a, a.displs_cd, a.counts_cd, a.Dinds_cd, a.Q_cd, a.pdata_cd, fp32, CONTRACTED, gcd);
}

template <int LA, int LB, int LC, int LD>
int run_exchange(const ExchangeArgs& a, cudaStream_t st)
{
    if (a.n_ik == 0) return VLXB_OK;
    if (!a.mat_K || !a.pair_i || !a.pair_k || !a.D || !a.Q_ab || !a.Q_cd || !a.Dinds_ab || !a.Dinds_cd ||
        !a.displs_ab || !a.displs_cd || !a.counts_ab || !a.counts_cd || !a.pdata_ab || !a.pdata_cd || a.naos == 0)
        return VLXB_EINVAL;
    const int L4[4] = {LA, LB, LC, LD};
    for (int t = 0; t < 4; t++)
        if (!a.info[L4[t]] || !a.aoinds[L4[t]] || a.count[L4[t]] == 0) return VLXB_EINVAL;
    if (!(a.thr >= 0.0) || !(a.omega >= 0.0)) return VLXB_EINVAL;
    int rc = ensure_pool_configured();
    if (rc) return rc;
    const BoysTabs tab{boys_table_device(), boys_table32_device()};
    if (!tab.f64 || !tab.f32) return VLXB_ECUDA;
    const Fp32Settings fp32 = a.share ? a.share->fp32 : fp32_settings();
    const double cut = fp32.cut, budget = fp32.budget;
    Arena local(st);
    Arena& ar = a.share ? a.share->ar : local;
    KOutData ko;
    PairGroups gab, gcd;
    rc = prepare_exchange<LA, LB, LC, LD>(ar, a, fp32, ko, gab, gcd);
    if (rc) return rc;
    [[maybe_unused]] KGroups kgab{}, kgcd{};
    if (k_rys(LA, LB, LC, LD) && k_contracted(LA, LB, LC, LD) && cut > 0.0) {
        kgab = KGroups{gab.gseg, gab.gq, gab.gbeg, gab.gcnt, gab.msp, gab.mq, gab.msu, gab.mmask, gab.gqa, gab.gqpre,
                       gab.rec_grp};
        kgcd = KGroups{gcd.gseg, gcd.gq, gcd.gbeg, gcd.gcnt, gcd.msp, gcd.mq, gcd.msu, gcd.mmask, gcd.gqa, gcd.gqpre,
                       gcd.rec_grp};
    }
    double* blk_maxD = a.share ? a.share->maxd[LA * 3 + LC][LB * 3 + LD] : nullptr;
    if (a.prim_mol_a && a.maxD_mol && !blk_maxD) {
        rc = kout_block_maxd(ar, ko, a.prim_mol_a, a.maxD_mol, &blk_maxD);
        if (rc) return rc;
        if (a.share) a.share->maxd[LA * 3 + LC][LB * 3 + LD] = blk_maxD;
    }
    if (ar.failed()) return VLXB_ENOMEM;
    if (a.share && a.share->prepare_only) return VLXB_OK;
    KOutBlocks out{ko.ish, ko.ksh, ko.idx, ko.stride, ko.n, blk_maxD};
    KPartnerRecs rab{gab.rec_sp, gab.rec_q, gab.rec_mask, gab.seg, gab.geo, gab.S, gab.sp_j, gab.sp_stride, gab.su,
                     gab.rec_qa, gab.rec_qpre};
    KPartnerRecs rcd{gcd.rec_sp, gcd.rec_q, gcd.rec_mask, gcd.seg, gcd.geo, gcd.S, gcd.sp_j, gcd.sp_stride, gcd.su,
                     gcd.rec_qa, gcd.rec_qpre};
    int grid = launch_grid_limit();
    if ((int64_t)grid > (int64_t)a.n_ik) grid = (int)a.n_ik;
    unsigned long long* qc = quartet_counters_device();
    unsigned long long* qk = qc ? qc + 1 : nullptr;
    const KDensity dm{a.aoinds[LB], a.count[LB], a.aoinds_col[LD] ? a.aoinds_col[LD] : a.aoinds[LD], a.count[LD],
                      a.D, a.D_stride ? a.D_stride : a.naos};
    for (int pm = 0; pm < (cut > 0.0 ? 2 : 1); pm++) {
        if constexpr (!k_rys(LA, LB, LC, LD))
            rc = launch_exchange_thread<LA, LB, LC, LD>(pm, grid, st, out, rab, rcd, dm, a.maxD, a.omega, a.thr,
                                                        a.mat_K, tab, qk, cut, budget);
        else if (pm == 1)
            rc = launch_exchange_mixed<LA, LB, LC, LD>(grid, st, out, rab, rcd, kgab, kgcd, dm, a.maxD, a.omega, a.thr,
                                                       a.mat_K, tab, qk, cut, budget);
        else
            rc = launch_exchange_rys<LA, LB, LC, LD>(grid, st, out, rab, rcd, kgab, kgcd, dm, a.maxD, a.omega, a.thr,
                                                     a.mat_K, qk, cut, budget);
        if (rc) return rc;
        note_launches();
    }
    return VLXB_OK;
}

// Energy-weighted centre derivatives of one exchange class (see
// exchange_grad_kernel): grad[x * gstride + p] += ..., p the lowest (i, k)
// list position of each primitive shell block.  FP64, single-molecule calls.
template <int LA, int LB, int LC, int LD>
int run_exchange_grad(const ExchangeArgs& a, int64_t gstride, cudaStream_t st)
{
    if (a.n_ik == 0) return VLXB_OK;
    if (!a.mat_K || !a.pair_i || !a.pair_k || !a.D || !a.Q_ab || !a.Q_cd || !a.Dinds_ab || !a.Dinds_cd ||
        !a.displs_ab || !a.displs_cd || !a.counts_ab || !a.counts_cd || !a.pdata_ab || !a.pdata_cd || a.naos == 0)
        return VLXB_EINVAL;
    const int L4[4] = {LA, LB, LC, LD};
    for (int t = 0; t < 4; t++)
        if (!a.info[L4[t]] || !a.aoinds[L4[t]] || a.count[L4[t]] == 0) return VLXB_EINVAL;
    if (!(a.thr >= 0.0) || !(a.omega >= 0.0)) return VLXB_EINVAL;
    if (gstride < (int64_t)a.n_ik) return VLXB_EINVAL;
    int rc = ensure_pool_configured();
    if (rc) return rc;
    Arena local(st);
    Arena& ar = a.share ? a.share->ar : local;
    KOutData ko;
    PairGroups gab, gcd;
    rc = prepare_exchange<LA, LB, LC, LD>(ar, a, Fp32Settings{}, ko, gab, gcd);
    if (rc) return rc;
    if (ar.failed()) return VLXB_ENOMEM;
    if (a.share && a.share->prepare_only) return VLXB_OK;
    KOutBlocks out{ko.ish, ko.ksh, ko.idx, ko.stride, ko.n, nullptr};
    KPartnerRecs rab{gab.rec_sp, gab.rec_q, gab.rec_mask, gab.seg, gab.geo, gab.S, gab.sp_j, gab.sp_stride, gab.su,
                     nullptr, nullptr};
    KPartnerRecs rcd{gcd.rec_sp, gcd.rec_q, gcd.rec_mask, gcd.seg, gcd.geo, gcd.S, gcd.sp_j, gcd.sp_stride, gcd.su,
                     nullptr, nullptr};
    const KDensity dm{a.aoinds[LB], a.count[LB], a.aoinds[LD], a.count[LD], a.D, a.naos};
    const KGradBlockD bd{a.aoinds[LA], a.count[LA], a.aoinds[LC], a.count[LC], LA == LC ? 1 : 0};
    int grid = launch_grid_limit();
    if ((int64_t)grid > (int64_t)a.n_ik) grid = (int)a.n_ik;
    rc = launch_exchange_grad<LA, LB, LC, LD>(grid, st, out, rab, rcd, dm, bd, a.maxD, a.omega, a.thr, a.mat_K,
                                              gstride);
    if (rc) return rc;
    note_launches();
    return VLXB_OK;
}

}  // namespace vlxb
