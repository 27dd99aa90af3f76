// alloc_retry.cuh with an allocator that is played by functions.
#include <cstdio>

#include "../../dmtz_gb300/csrc/alloc_retry.cuh"

int main() {
    int bad = 0, allocs = 0, released = 0;
    auto run = [&](int full, int kept, cudaError_t error) {  // full: failing calls until something is released
        allocs = released = 0;
        return dmtz::alloc_retry(
            [&]() {
                allocs++;
                return full && !released ? error : cudaSuccess;
            },
            [&]() {
                released = kept;
                return kept != 0;
            });
    };
    bad += run(0, 1, cudaErrorMemoryAllocation) != cudaSuccess || allocs != 1 || released;
    bad += run(1, 1, cudaErrorMemoryAllocation) != cudaSuccess || allocs != 2;
    bad += run(1, 0, cudaErrorMemoryAllocation) != cudaErrorMemoryAllocation || allocs != 1;
    bad += run(1, 1, cudaErrorIllegalState) != cudaErrorIllegalState || allocs != 1 || released;
    printf("%d wrong\n", bad);
    return bad != 0;
}
