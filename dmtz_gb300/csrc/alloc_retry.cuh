// alloc_retry.cuh — an allocation that may give something up first.
#pragma once
#include <cuda_runtime.h>

namespace dmtz {

// alloc(); where it is out of memory and release() gave some back, once more
template <class Alloc, class Release>
cudaError_t alloc_retry(Alloc &&alloc, Release &&release) {
    const cudaError_t e = alloc();
    return e == cudaErrorMemoryAllocation && release() ? alloc() : e;
}

}  // namespace dmtz
