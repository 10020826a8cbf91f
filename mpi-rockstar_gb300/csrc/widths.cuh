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

// Whether a place that a counter handed out lies in a pool of `cap`.  The
// counter also counts what finds no room, past 2^31 for the lists of very dense
// snapshots: as an int such a place is negative and below every cap.
__host__ __device__ __forceinline__ bool has_place(unsigned place, int cap) {
    return cap > 0 && place < (unsigned)cap;
}

}  // namespace rsg
