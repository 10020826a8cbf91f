// Places that a large call carries past the width of the integers they are
// made from.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace rsg {

// The place of a thread's warp in its launch.  In 64 bits: a launch with a warp
// for each of 2^27 things has 2^32 threads, and the product of 32-bit block and
// thread numbers starts again at zero there.
__host__ __device__ __forceinline__ int64_t warp_index(unsigned block, unsigned threads,
                                                       unsigned thread) {
    return ((int64_t)block * threads + thread) >> 5;
}

}  // namespace rsg
