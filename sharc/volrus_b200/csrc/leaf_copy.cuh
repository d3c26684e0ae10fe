// Moves of whole leaf records between a level set's pool (f16 or f32, voxel
// units, 16-byte aligned) and f32 leaf arrays, shared by uploads, downloads
// and host steps.  One warp moves one leaf: a lane holds four groups of four
// consecutive values, so every load is in flight before the first store and
// each store instruction of the warp covers whole 128-byte lines.
//
// Bound: HBM (an f16 leaf moves 1 KB + 2 KB).  One value per thread and load
// kept only ~2 bytes per thread in flight: 312k f16 leaves took 466 us to
// read out and 552 us to load (2.1 and 1.7 TB/s); one warp per leaf takes 166
// and 160 us (5.9 and 6.0 TB/s, against 6.5 TB/s of a plain copy).
#pragma once
#include "method.cuh"

namespace vlr {

// Four consecutive pool values as f32 (8 bytes of f16, 16 of f32).
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __half* p) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&r.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__half* p, float4 v) {
    __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<unsigned*>(&a), *reinterpret_cast<unsigned*>(&b));
}

// Pool values of one leaf -> 512 f32 at dst, by one warp.  vec: dst is
// 16-byte aligned (a caller's device buffer need not be).
template <typename T>
__device__ __forceinline__ void leaf_out(const T* __restrict__ src, float* __restrict__ dst, bool vec, int lane) {
    if (vec) {
        float4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = load4(src + 4 * (q * 32 + lane));
#pragma unroll
        for (int q = 0; q < 4; ++q) store4(dst + 4 * (q * 32 + lane), v[q]);
    } else {
#pragma unroll 8
        for (int t = lane; t < kLeafVoxels; t += 32) dst[t] = to_f(src[t]);
    }
}

// 512 f32 at src -> the pool values of one leaf, by one warp.
template <typename T>
__device__ __forceinline__ void leaf_in(const float* __restrict__ src, T* __restrict__ dst, bool vec, int lane) {
    if (vec) {
        float4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = load4(src + 4 * (q * 32 + lane));
#pragma unroll
        for (int q = 0; q < 4; ++q) store4(dst + 4 * (q * 32 + lane), v[q]);
    } else {
#pragma unroll 8
        for (int t = lane; t < kLeafVoxels; t += 32) dst[t] = from_f<T>(src[t]);
    }
}

__host__ __device__ inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace vlr
