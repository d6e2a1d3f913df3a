// Host side of vlxb_fockBuild without a device: fockbuild.cu and the class
// drivers as they are, the list preparations and the kernel launchers replaced
// by fakes that record what they are given.  (PD|DD) exchange and (PD|DD)
// Coulomb stand for their kinds.  Arguments: the scenario and its number; prints
// "name value" lines.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "../vlx-twoe-ints_b200/csrc/fockbuild.cu"
#include "../vlx-twoe-ints_b200/csrc/fork.cu"

namespace vlxb {

static double g_cut[2], g_budget[2];  // the settings before and after another thread changes them,
static int g_change_at = 1 << 30;     // which it does when they have been read this often
static int g_reads;
static int g_fail_at = -1, g_fail_rc;  // the launch that fails, and how
static int g_launches, g_null_groups, g_null_sums, g_launch_cut_differs, g_col_index, g_stride;
static char g_buffer[64];

double fp32_cut_get() { return g_cut[g_reads++ >= g_change_at]; }
double fp32_budget_get() { return g_budget[g_reads++ >= g_change_at]; }
int ensure_pool_configured() { return VLXB_OK; }
const double* boys_table_device() { return (const double*)g_buffer; }
const float* boys_table32_device() { return (const float*)g_buffer; }
const double* rys_table_device() { return (const double*)g_buffer; }
unsigned long long* quartet_counters_device() { return nullptr; }
int launch_grid_limit() { return 1; }
int schedule_get(int, int, int, int, int) { return 0; }
void note_launches(int) {}

int group_flat(Arena&, int, int, int, int, const uint32_t*, const uint32_t*, int64_t, const double*, uint32_t,
               const double*, uint32_t, PairGroups&) { return VLXB_OK; }
int group_csr(Arena&, int, int, int, int, const uint32_t*, const uint32_t*, const uint32_t*, int64_t, const double*,
              uint32_t, const double*, uint32_t, PairGroups&) { return VLXB_OK; }
static int g_prepared, g_short_at = -1;  // the preparation that runs out of memory
int make_records(Arena&, int, PairGroups&, const double*, int64_t)
{
    return g_prepared++ == g_short_at ? VLXB_ENOMEM : VLXB_OK;
}
int segment_records(Arena&, int, int, int, PairGroups&, const double*) { return VLXB_OK; }
int bra_record_mol(Arena&, const PairGroups&, const int32_t*, int32_t** mol)
{
    *mol = (int32_t*)g_buffer;
    return VLXB_OK;
}
int budget_prefix_records(Arena&, PairGroups& g, int, int)
{
    g.rec_qa = g.rec_qpre = (double*)g_buffer;
    return VLXB_OK;
}
int budget_prefix_kets(Arena&, JKetData& kd, int)
{
    kd.tpre = (double*)g_buffer;
    return VLXB_OK;
}
int contract_groups(Arena&, int, PairGroups& g, const uint32_t*, uint32_t)
{
    g.gseg = g.rec_grp = (int*)g_buffer;
    return VLXB_OK;
}
int kout_prepare(Arena&, int, int, int, int, const uint32_t*, const uint32_t*, int64_t, KOutData&) { return VLXB_OK; }
int kout_block_maxd(Arena&, const KOutData&, const int32_t*, const double*, double** out)
{
    *out = (double*)g_buffer;
    return VLXB_OK;
}
template <int LC, int LD>
int jket_prepare(Arena&, const PairGroups&, const uint32_t*, const uint32_t*, const double*, const double*,
                 const double*, JKetData& out, const int32_t*, int, bool)
{
    out = JKetData{};
    return VLXB_OK;
}

static double g_first_cut = -1.0;
static int launched(double cut)
{
    if (g_first_cut < 0.0) g_first_cut = cut;
    g_launch_cut_differs += cut != g_first_cut;
    return g_launches++ == g_fail_at ? g_fail_rc : VLXB_OK;
}

template <int LA, int LB, int LC, int LD>
int launch_coulomb(int, int, int, cudaStream_t, const JBraRecs&, const JKetPairs& ket, double*, double, const BoysTabs&,
                   unsigned long long*, double cut, double budget)
{
    g_null_sums += budget > 0.0 && !ket.tpre;
    return launched(cut);
}
template <int LA, int LB, int LC, int LD>
int launch_coulomb_rys(int, cudaStream_t, const JBraRecs&, const JKetPairs& ket, double*, double, unsigned long long*,
                       double cut, double budget)
{
    g_null_sums += budget > 0.0 && !ket.tpre;
    return launched(cut);
}
template <int LA, int LB, int LC, int LD>
int launch_exchange_mixed(int, cudaStream_t, const KOutBlocks&, const KPartnerRecs& ab, const KPartnerRecs&,
                          const KGroups& gab, const KGroups& gcd, const KDensity&, double, double, double, double*,
                          const BoysTabs&, unsigned long long*, double cut, double budget)
{
    g_null_groups += !gab.seg || !gcd.seg;
    g_null_sums += budget > 0.0 && !ab.qa;
    return launched(cut);
}
template <int LA, int LB, int LC, int LD>
int launch_exchange_rys(int, cudaStream_t, const KOutBlocks&, const KPartnerRecs&, const KPartnerRecs&, const KGroups&,
                        const KGroups&, const KDensity& dm, double, double, double, double*, unsigned long long*,
                        double cut, double)
{
    g_col_index = (int)((const char*)dm.d_aoinds - g_buffer);
    g_stride = (int)dm.naos;
    return launched(cut);
}

int dispatch_coulomb(int, bool, const CoulombArgs& a, int64_t, cudaStream_t st) { return run_coulomb<1, 2, 2, 2>(a, st); }
int dispatch_exchange(int, bool, const ExchangeArgs& a, int64_t, cudaStream_t st) { return run_exchange<1, 2, 2, 2>(a, st); }

}  // namespace vlxb

int main(int argc, char** argv)
{
    using namespace vlxb;
    const char* what = argc > 1 ? argv[1] : "";
    const int number = argc > 2 ? atoi(argv[2]) : 0;
    VlxbFockBuild b;
    memset(&b, 0, sizeof b);
    void* p = g_buffer;
    for (int l = 0; l < 3; l++) {
        b.prim_info[l] = (const double*)p;
        b.prim_aoinds[l] = (const uint32_t*)p;
        b.prim_count[l] = 2;
    }
    for (int t = 0; t < 9; t++) {
        b.mat_J[t] = b.mat_K[t] = (double*)p;
        b.j_first[t] = b.j_second[t] = b.k_i[t] = b.k_k[t] = (const uint32_t*)p;
        b.j_pdata[t] = b.j_Q[t] = b.j_D[t] = b.kp_Q[t] = b.kp_pdata[t] = (const double*)p;
        b.kp_displs[t] = b.kp_counts[t] = b.kp_Dinds[t] = (const uint32_t*)p;
        b.j_count[t] = b.k_count[t] = 4;
    }
    b.D = (const double*)p;
    b.naos = 5;
    b.j_classes = 1ull << 29;           // (PD|DD): bra pair 4, ket pair 5
    b.k_classes = 1ull << (4 * 9 + 8);  // (PD|DD): (a, c) = (p, d), (b, d) = (d, d)
    if (!strcmp(what, "cutoff set")) {
        g_change_at = number;
        g_cut[1] = 1e-6;
    } else if (!strcmp(what, "cutoff reset")) {
        g_change_at = number;
        g_cut[0] = 1e-6;
    } else if (!strcmp(what, "budget set")) {
        g_change_at = number;
        g_cut[0] = g_cut[1] = 1e-6;
        g_budget[1] = 0.2;
    } else if (!strcmp(what, "launch fails")) {
        g_cut[0] = g_cut[1] = 1e-6;
        g_fail_at = number;
        g_fail_rc = VLXB_ENOMEM;
    } else if (!strcmp(what, "preparation fails")) {
        g_short_at = number;
    } else if (!strcmp(what, "batch")) {  // number: bits of what is missing
        b.n_mol = 2;
        if (!(number & 1)) b.prim_mol[1] = (const int32_t*)p;
        if (!(number & 2)) b.prim_mol[2] = (const int32_t*)p;
        if (!(number & 4)) b.maxD_mol[8] = (const double*)p;
        if (number & 8) b.k_classes = 0;
        if (number & 16) b.j_count[1 * 3 + 2] = 0;
    } else if (!strcmp(what, "columns")) {  // number: n_mol
        b.n_mol = number;
        for (int l = 0; l < 3; l++) {
            b.prim_mol[l] = (const int32_t*)p;
            b.prim_aocols[l] = (const uint32_t*)(g_buffer + 8);
        }
        b.maxD_mol[8] = (const double*)p;
        b.D_stride = 3;
    }
    const int rc = vlxb_fockBuild(&b, nullptr);
    printf("prepared %d\n", g_prepared);
    printf("rc %d\nlaunches %d\nnull_groups %d\nnull_sums %d\ncut_differs %d\n", rc, g_launches, g_null_groups,
           g_null_sums, g_launch_cut_differs);
    printf("col_index %d\nstride %d\n", g_col_index, g_stride);
    return 0;
}
