// report_wait.cuh — the host's wait for a round's counts in pinned memory.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace dmtz {

// Waits until *at is seq: the last kernel of a round writes it, behind the round's
// counts.  query() is the state of the stream that the kernel runs on.  A stream that
// is idle without having written it (a launch failed) ends the wait with
// cudaErrorUnknown, an error of the stream with that error.
template <class Query>
cudaError_t wait_report(const volatile unsigned long long *at, unsigned long long seq, Query &&query) {
    for (unsigned spin = 1; *at != seq; spin++) {
        if (spin % 4096) continue;
        const cudaError_t q = query();
        if (q == cudaErrorNotReady) continue;
        if (q != cudaSuccess) return q;
        if (*at != seq) return cudaErrorUnknown;
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    return cudaSuccess;
}

}  // namespace dmtz
