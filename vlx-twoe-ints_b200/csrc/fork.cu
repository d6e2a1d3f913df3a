// Side streams of small builds (fork.cuh).  Class kernels of a small build leave
// most of the device idle, and those of different output lists share no output.
//
// A set of streams serves one call at a time and is handed out again to the same
// caller's stream, whose order the calls then keep, or when its work has ended:
// calls on different streams never queue behind one another in a side stream.
// Sets are made on demand, SIDE_SETS per device at most; a call that finds none
// stays on its own stream, as does one that is being captured.
#include "fork.cuh"

#include <mutex>
#include <new>
#include <vector>

#include "engine.cuh"
#include "../../include/vlxb.h"

namespace vlxb {

// Calls of at most this many output entries fork: on one stream / forked, 2 atoms
// 4s3p2d (22000 entries) 2.78 / 1.98 ms, 5 atoms (135000) 17.0 / 14.7, 8 atoms
// (336000) 75.4 / 70.0.  The gain shrinks but does not end at the bound (10 atoms,
// 520000: 169 / 159; 14 atoms, 1.0 million: 567 / 543): 4 to 10 % are still to be
// had above it.
constexpr uint64_t FORK_ENTRIES = 400000;
// More callers' streams than a server keeps in flight.
constexpr size_t SIDE_SETS = 32;

static std::mutex g_sets_mu;
static std::vector<SideStreams*> g_sets[64];

// While another thread captures in global mode, calls such as cudaEventQuery are
// refused to every thread that does not ask for the relaxed mode.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

static void destroy(SideStreams* w)
{
    for (int k = 0; k < FORK_STREAMS; k++) {
        if (w->s[k]) cudaStreamDestroy(w->s[k]);
        if (w->done[k]) cudaEventDestroy(w->done[k]);
    }
    if (w->start) cudaEventDestroy(w->start);
    delete w;
    cudaGetLastError();
}

static SideStreams* create()
{
    SideStreams* w = new (std::nothrow) SideStreams;
    if (!w) return nullptr;
    bool ok = cudaEventCreateWithFlags(&w->start, cudaEventDisableTiming) == cudaSuccess;
    for (int k = 0; ok && k < FORK_STREAMS; k++)
        ok = cudaStreamCreateWithFlags(&w->s[k], cudaStreamNonBlocking) == cudaSuccess &&
             cudaEventCreateWithFlags(&w->done[k], cudaEventDisableTiming) == cudaSuccess;
    if (ok) return w;
    destroy(w);
    return nullptr;
}

static bool idle(SideStreams* w)
{
    for (int k = 0; k < FORK_STREAMS; k++)
        if (w->used[k]) {
            if (cudaEventQuery(w->done[k]) != cudaSuccess) {
                cudaGetLastError();  // cudaErrorNotReady stays set otherwise
                return false;
            }
            w->used[k] = false;
        }
    return true;
}

static SideStreams* take(cudaStream_t st)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    const RelaxedCapture relaxed;
    std::lock_guard<std::mutex> lk(g_sets_mu);
    std::vector<SideStreams*>& sets = g_sets[dev];
    SideStreams* w = nullptr;
    if (st != cudaStreamPerThread)  // one handle, a stream for every thread
        for (SideStreams* c : sets)
            if (!c->taken && c->caller == st) {
                w = c;
                break;
            }
    if (!w)
        for (SideStreams* c : sets)
            if (!c->taken && idle(c)) {
                w = c;
                break;
            }
    if (!w && sets.size() < SIDE_SETS) {
        w = create();
        if (w) sets.push_back(w);
    }
    if (w) {
        w->taken = true;
        w->caller = st;
    }
    return w;
}

static void give_back(SideStreams* w)
{
    std::lock_guard<std::mutex> lk(g_sets_mu);
    w->taken = false;
}

Fork::Fork(cudaStream_t st, uint64_t outputs) : st_(st)
{
    if (outputs > FORK_ENTRIES) return;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return;
    }
    set_ = take(st);
    if (set_ && cudaEventRecord(set_->start, st) != cudaSuccess) {
        cudaGetLastError();
        give_back(set_);
        set_ = nullptr;
    }
}

cudaStream_t Fork::at(int g)
{
    if (!set_) return st_;
    const int k = g % FORK_STREAMS;
    if (!open_[k]) {
        if (cudaStreamWaitEvent(set_->s[k], set_->start, 0) != cudaSuccess) {
            cudaGetLastError();
            return st_;
        }
        open_[k] = true;
    }
    return set_->s[k];
}

int Fork::join()
{
    int rc = VLXB_OK;
    for (int k = 0; k < FORK_STREAMS; k++)
        if (open_[k]) {
            set_->used[k] = true;
            if (cudaEventRecord(set_->done[k], set_->s[k]) != cudaSuccess ||
                cudaStreamWaitEvent(st_, set_->done[k], 0) != cudaSuccess) {
                // never leave work behind that the caller's stream does not wait for
                cudaGetLastError();
                cudaStreamSynchronize(set_->s[k]);
                rc = VLXB_ECUDA;
            }
            open_[k] = false;
        }
    return rc;
}

Fork::~Fork()
{
    join();
    if (set_) give_back(set_);
}

}  // namespace vlxb

extern "C" void* vlxb_forkBegin(void* stream, uint64_t outputs)
{
    vlxb::Fork* f = new (std::nothrow) vlxb::Fork((cudaStream_t)stream, outputs);
    if (f && f->forked()) return f;
    delete f;
    return nullptr;
}

extern "C" void* vlxb_forkStream(void* fork, int list)
{
    return fork && list >= 0 ? (void*)((vlxb::Fork*)fork)->at(list) : nullptr;
}

extern "C" int vlxb_forkJoin(void* fork)
{
    if (!fork) return VLXB_EINVAL;
    const int rc = ((vlxb::Fork*)fork)->join();
    delete (vlxb::Fork*)fork;
    return rc;
}
