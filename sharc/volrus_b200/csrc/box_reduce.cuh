// Bounding box of integer coordinates over a whole grid, for sort keys that
// hold only the bits a grid's extent needs.
#pragma once
#include <climits>

namespace vlr {

// box[a] = max over ~c_a, box[3 + a] = max over c_a (so ~box[a] is the
// minimum): six maxima, cleared to kBoxClear bytes (below any leaf
// coordinate).  Every thread of the block calls it once; a block does six
// atomics (one warp each of a wide grid doing six took 37 us at 40k points).
constexpr int kBoxClear = 0x80;

__device__ __forceinline__ void block_box(const int lo[3], const int hi[3], int* __restrict__ box) {
    __shared__ int s_box[6];
    if (threadIdx.x < 6) s_box[threadIdx.x] = INT_MIN;
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int l = __reduce_max_sync(0xffffffffu, ~lo[a]), h = __reduce_max_sync(0xffffffffu, hi[a]);
        if ((threadIdx.x & 31) == 0) {
            atomicMax(&s_box[a], l);
            atomicMax(&s_box[3 + a], h);
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) atomicMax(&box[threadIdx.x], s_box[threadIdx.x]);
}

// Bits that hold values 0..ext.
inline int bits_for(long long ext) {
    int b = 0;
    while (b < 62 && (1ll << b) <= ext) ++b;
    return b;
}

}  // namespace vlr
