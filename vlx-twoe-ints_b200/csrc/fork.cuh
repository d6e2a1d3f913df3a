// Side streams of one call: kernels that write different output lists run
// beside one another between a fork and a join on the caller's stream.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace vlxb {

constexpr int FORK_STREAMS = 4;

// Streams and events that one call at a time uses (of the current device).
struct SideStreams {
    cudaStream_t s[FORK_STREAMS] = {};
    cudaEvent_t start = nullptr, done[FORK_STREAMS] = {};
    bool used[FORK_STREAMS] = {};   // since they were last known to be idle
    cudaStream_t caller = nullptr;  // stream of the last call
    bool taken = false;
};

class Fork {
  public:
    // outputs: entries of all output lists of the call (FORK_ENTRIES).
    Fork(cudaStream_t st, uint64_t outputs);
    // Stream of output list g: the calls of one list keep their order, so
    // results do not depend on it.
    cudaStream_t at(int g);
    // The caller's stream continues after every forked kernel.
    int join();
    bool forked() const { return set_ != nullptr; }
    ~Fork();
    Fork(const Fork&) = delete;
    Fork& operator=(const Fork&) = delete;

  private:
    cudaStream_t st_;
    SideStreams* set_ = nullptr;
    bool open_[FORK_STREAMS] = {};  // forked and not joined
};

}  // namespace vlxb
