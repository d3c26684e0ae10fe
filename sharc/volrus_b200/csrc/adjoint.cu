// Differentiable advection: frozen-band semi-Lagrangian steps through a dense
// staggered velocity field, with a hand-written adjoint.
//
// Forward, K steps (t_k = t0 + k dt, c_k = cos(pi t_{k+1} / T)):
//   phi_{k+1}(x) = trilinear(phi_k)(x - dt c_k u(x))        for band voxels x
// where u(x) is the trilinear upsample of a staggered (MAC) field V of n^3
// cells of H voxels (component a lives on the faces normal to axis a) and
// every non-band voxel keeps its initial value (+-hw; unallocated leaves read
// the clamped-sign rule).  The map phi_0 -> phi_K is affine on the band, so
// the gradient is exact (up to rounding) wherever floor() does not jump.
//
// Backward, given lambda_K = dL/dphi_K on the band:
//   lambda_k(c) = sum_x lambda_{k+1}(x) w_c(p_k(x))     (transpose of the blend)
//   G(x)      += lambda_{k+1}(x) (-dt c_k) grad trilinear(phi_k)(p_k(x))
//   dL/dphi_0 = lambda_0,  dL/dV = upsample^T G
// The lambda transpose is a gather over the band voxels whose foot cell can
// hold the corner (a window of at most (2R+2)^3 voxels, R the per-step reach),
// summed in a fixed order.  upsample^T depends on the geometry alone: its
// entries are sorted by node once at creation (stable radix sort) and a
// backward pass sums each node's entries in that order.  No float atomics:
// deterministic results.  The trilinear gradient of phi_k at every foot comes
// from recomputing phi_k between checkpoints taken every C steps (sqrt(K)),
// by the forward kernel itself, which reads the same eight corners.  A level
// set's displacement is fixed and its map is linear in lambda with constant
// feet, so its backward pass needs neither phi_k nor checkpoints.
//
// State lives in leaf pools (512 values a leaf); band voxels are listed in
// leaf order, and the step kernels take the list in chunks of up to 32 voxels
// of one leaf, one warp a chunk: the leaf's 27 neighbour slots sit in the
// warp's lanes (one shuffle per lookup instead of a load) and its candidate
// window is uniform over the warp.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include "box_reduce.cuh"
#include "method_state.hpp"
#include "sort_reduce.hpp"

struct vlr_adjoint {
    vlr_ctx* ctx = nullptr;
    int n_leaves = 0;
    int n_band = 0;
    float hw = 3.0f;
    int4* origin = nullptr;
    int* nbr = nullptr;
    uint64_t* hkey = nullptr;
    int* hval = nullptr;
    int hcap = 0;
    long long base[3] = {0, 0, 0};
    float* phi[2] = {nullptr, nullptr};  // leaf-major, 512 per leaf; phi[0] holds phi_0 layout template
    float* phi_init = nullptr;           // initial full leaves (non-band values are constants)
    int* bidx = nullptr;                 // slot*512 + off -> band index or -1
    int* bvox = nullptr;                 // band index -> slot*512 + off
    float3* ub = nullptr;                // upsampled velocity at band voxels
    float* vel = nullptr;                // staggered field 3 x n^3
    int n_stag = 0;
    double H = 1.0;                      // staggered cell size in voxels
    double dt = 0.0, t0 = 0.0, period = 1.0;
    int steps = 0, chk_every = 1;
    char* block = nullptr;               // staggered: holds checkpoints, segment, G and the feet
    bool block_pooled = false;           // from the context's pool
    float* checkpoints = nullptr;        // (steps / chk_every + 1) x n_band
    float3* segment = nullptr;           // chk_every x n_band (gradients of the recomputed states at the feet)
    float* lam[2] = {nullptr, nullptr};  // band order: [1] lambda_K (and phi_K), [0] lambda_0
    float* lam_final = nullptr;          // lam buffer holding dL/dphi_0 after the last backward pass
    // the forward and backward step loops captured as CUDA graphs (dropped
    // when the velocity, hence the reach, changes)
    cudaGraphExec_t fwd_exec = nullptr, bwd_exec = nullptr;
    float* gvel = nullptr;               // dL/dV, 3 x n^3
    float3* G = nullptr;
    int reach = 1;                       // displacement bound per step, voxels (ceil of dt max|V|)
    int gather = 0;                      // transpose kernel: 0 by band size and reach, 1 windowed, 2 quad
    int disp = 0;                        // 1: ub holds each band voxel's fixed backtrace displacement
                                         // (a level set's time-independent velocity), step factor 1
    int* lstart = nullptr;               // n_leaves + 1: first band index of each leaf
    int2* chunks = nullptr;              // up to 32 band voxels of one leaf: see load_chunk
    int n_chunks = 0;
    float* urange = nullptr;             // per leaf: min and max of ub per axis over its band voxels (6 floats)
    float* nrange = nullptr;             // the same over the leaf's 27-leaf neighbourhood
    // feet of the band voxels by pool voxel, ping-pong over the steps (one
    // buffer for a fixed displacement): packed offsets (0 off the band) and
    // (wx, wy, wz, lambda); a fixed displacement keeps lambda in lam_pool
    unsigned* foot_pk[2] = {nullptr, nullptr};
    float4* foot_w[2] = {nullptr, nullptr};
    float* lam_pool[2] = {nullptr, nullptr};
    // upsample^T: entry e adds ent_w[e] G[ent_b[e]] (G as 3 n_band floats) to
    // node seg_node[j], e in [seg_start[j], seg_start[j + 1])
    int* ent_b = nullptr;
    float* ent_w = nullptr;
    int* seg_start = nullptr;
    unsigned* seg_node = nullptr;
    int n_seg = 0;
};

namespace vlr {

__device__ __forceinline__ int nbx(int c) { return (c < 0) ? 0 : (c > 7 ? 2 : 1); }

// phi at local coordinate (x, y, z) of leaf `slot` (may leave the leaf by one voxel).
__device__ __forceinline__ float adj_read(const float* __restrict__ phi, const int* __restrict__ nbr, int slot, int x,
                                          int y, int z, float hw) {
    int s = nbr[slot * kNbr + nbx(x) * 9 + nbx(y) * 3 + nbx(z)];
    if (s >= 0) return phi[(size_t)s * kLeafVoxels + voxel_off(x, y, z)];
    int cx = min(max(x, 0), 7), cy = min(max(y, 0), 7), cz = min(max(z, 0), 7);
    return copysignf(hw, phi[(size_t)slot * kLeafVoxels + ((cx << 6) | (cy << 3) | cz)]);
}

// Trilinear upsample of component a of the staggered field at voxel point p.
__device__ __forceinline__ float stag_sample(const float* __restrict__ V, int n, float H, int a, float px, float py,
                                             float pz) {
    float g[3] = {px / H, py / H, pz / H};
    for (int q = 0; q < 3; ++q)
        if (q != a) g[q] -= 0.5f;
    int i0[3];
    float w[3];
    for (int q = 0; q < 3; ++q) {
        float f = floorf(g[q]);
        i0[q] = (int)f;
        w[q] = g[q] - f;
    }
    auto at = [&](int i, int j, int k) {
        i = min(max(i, 0), n - 1);
        j = min(max(j, 0), n - 1);
        k = min(max(k, 0), n - 1);
        return V[(size_t)a * n * n * n + ((size_t)i * n + j) * n + k];
    };
    float c00 = at(i0[0], i0[1], i0[2]) * (1 - w[0]) + at(i0[0] + 1, i0[1], i0[2]) * w[0];
    float c01 = at(i0[0], i0[1], i0[2] + 1) * (1 - w[0]) + at(i0[0] + 1, i0[1], i0[2] + 1) * w[0];
    float c10 = at(i0[0], i0[1] + 1, i0[2]) * (1 - w[0]) + at(i0[0] + 1, i0[1] + 1, i0[2]) * w[0];
    float c11 = at(i0[0], i0[1] + 1, i0[2] + 1) * (1 - w[0]) + at(i0[0] + 1, i0[1] + 1, i0[2] + 1) * w[0];
    float c0 = c00 * (1 - w[1]) + c10 * w[1], c1 = c01 * (1 - w[1]) + c11 * w[1];
    return c0 * (1 - w[2]) + c1 * w[2];
}

__global__ void k_adj_upsample(const int* __restrict__ bvox, const int4* __restrict__ origin, int nb,
                               const float* __restrict__ V, int n, float H, float3* __restrict__ ub) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
        int sv = bvox[b], s = sv >> 9, off = sv & 511;
        int4 o = origin[s];
        float px = (float)(o.x + (off >> 6)), py = (float)(o.y + ((off >> 3) & 7)), pz = (float)(o.z + (off & 7));
        ub[b] = make_float3(stag_sample(V, n, H, 0, px, py, pz), stag_sample(V, n, H, 1, px, py, pz),
                            stag_sample(V, n, H, 2, px, py, pz));
    }
}

// Foot offset, floor and weights of band voxel b at step k.
struct Foot {
    int fx, fy, fz;     // floor of the foot, relative to the voxel
    float wx, wy, wz;   // fractions
};
__device__ __forceinline__ Foot foot_of(float3 u, float s) {
    float ox = s * u.x, oy = s * u.y, oz = s * u.z;  // s = -dt c_k
    Foot f;
    float bx = floorf(ox), by = floorf(oy), bz = floorf(oz);
    f.fx = (int)bx;
    f.fy = (int)by;
    f.fz = (int)bz;
    f.wx = ox - bx;
    f.wy = oy - by;
    f.wz = oz - bz;
    return f;
}

// One warp's chunk of the band list: up to 32 band voxels of one leaf, packed
// as (leaf << 6 | first chunk of its leaf << 5 | voxels - 1, first band
// index).  Lanes past the chunk repeat its first voxel (they take part in the
// shuffles and store nothing); row holds the leaf's neighbour slots, lane d
// the one at leaf offset d.
struct Chunk {
    int leaf, b, off, row;
    bool on;
};
__device__ __forceinline__ Chunk load_chunk(int2 h, const int* __restrict__ bvox, const int* __restrict__ nbr,
                                            int lane) {
    Chunk k;
    k.leaf = h.x >> 6;
    k.row = lane < kNbr ? __ldg(&nbr[(size_t)k.leaf * kNbr + lane]) : -1;
    k.on = lane <= (h.x & 31);
    k.b = k.on ? h.y + lane : h.y;
    k.off = __ldg(&bvox[k.b]) & 511;
    return k;
}

// The kernels of a pass form a chain in which each reads what the one before
// wrote, and at 10^4-10^5 band voxels a kernel is a few dependent trips to
// memory long, so its launch and its trips for fixed data count as much as the
// step itself.  Each is launched so that it may start while the one before
// still runs: it loads the chunk, voxels, feet and neighbour slots, which no
// kernel of the chain writes, waits for the one before (chain_wait), and only
// then reads state.  State pointers are not __restrict__: a read-only load
// could be moved above the wait or be served from a stale line.  The next
// kernel is let in after the wait, so no more than two are under way and the
// buffers of the step before are free.  64 steps there and back on 77k band
// voxels (192 kernels) went from 1018-1073 to 897-926 us.
__device__ __forceinline__ void chain_wait() {
    dep_wait();
    dep_launch();
}

// Resident CTAs of 256 threads per SM of the chunk kernels.  At 7.67M band
// voxels 5, 6, 7 and 8 take 101, 98, 102 and 103 us a forward step and 176,
// 170, 176 and 178 us a transpose (7 and 8 spill).
constexpr int kChunkCtas = 6;
constexpr int kWideCtas = 4;  // k_adj_lambda with three candidate rows in flight

// The chain header -> voxel, foot, neighbour slots -> corners is three trips
// to memory per chunk, and a band beyond L2 pays DRAM latency for each.  So
// every warp asks for the lines of the chunk one wave of warps ahead to be
// brought into L2: its list entries, per-voxel records and neighbour row and,
// once per leaf, the leaf's part of the pool arrays.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Lanes `from` on take the 128-byte lines of [p, p + bytes).
__device__ __forceinline__ void prefetch_lines(const void* p, int bytes, int lane, int from) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)127;
    const int n = (int)((reinterpret_cast<uintptr_t>(p) + bytes + 127 - a) >> 7);
    if (lane >= from && lane < from + n) prefetch_l2(reinterpret_cast<const char*>(a) + (lane - from) * 128);
}

// Leaf offset (0, 1, 2) of local coordinate c in [-8, 15].
__device__ __forceinline__ int leaf_of(int c) { return (c + 8) >> 3; }

// One forward step over the band voxels, one warp per chunk.  Non-band voxels
// never change and every state buffer holds phi_0 there from creation, so
// they are not touched.  chk: the new values in band order (a checkpoint, or
// phi_K), when not null.  GRAD: the trilinear gradient of src at the foot, in
// band order (the backward pass's recomputation); dst may then be null.
//
// Bound: instruction issue (70 % of the slots at 7.67M band voxels) and the
// latency of header -> voxel, foot, slots -> eight corners (24 bytes a voxel
// from HBM, 28 us there).  One thread per voxel
// with a neighbour-table load per corner took 121 us there, slots by shuffles
// 110 us, and 96 us with the next wave's lines prefetched into L2; 2.5 against
// 3.6 us at 77k voxels (launch-bound).
template <bool GRAD>
__global__ void __launch_bounds__(256, kChunkCtas)
    k_adj_forward(const int2* __restrict__ chunks, int n_chunks, int ahead, const int* __restrict__ bvox,
                  const int* __restrict__ nbr, const float3* __restrict__ ub, const float* src,
                  float* __restrict__ dst, float* __restrict__ chk, float3* __restrict__ grad, float s, float hw,
                  unsigned* err) {
    const int lane = threadIdx.x & 31;
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c >= n_chunks) return;
    const Chunk k = load_chunk(__ldg(&chunks[c]), bvox, nbr, lane);
    const bool more = c + ahead < n_chunks;
    const int2 ha = more ? __ldg(&chunks[c + ahead]) : make_int2(0, 0);
    const Foot f = foot_of(ub[k.b], s);
    int x = (k.off >> 6) + f.fx, y = ((k.off >> 3) & 7) + f.fy, z = (k.off & 7) + f.fz;
    const bool bad = x < -8 || y < -8 || z < -8 || x > 14 || y > 14 || z > 14;
    if (bad) x = y = z = 0;
    const int lx[2] = {leaf_of(x) * 9, leaf_of(x + 1) * 9}, ly[2] = {leaf_of(y) * 3, leaf_of(y + 1) * 3},
              lz[2] = {leaf_of(z), leaf_of(z + 1)};
    const int ox[2] = {(x & 7) << 6, ((x + 1) & 7) << 6}, oy[2] = {(y & 7) << 3, ((y + 1) & 7) << 3},
              oz[2] = {z & 7, (z + 1) & 7};
    int sl[8];
    int miss = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        sl[q] = __shfl_sync(0xffffffffu, k.row, lx[q >> 2] + ly[(q >> 1) & 1] + lz[q & 1]);
        miss |= sl[q];
    }
    chain_wait();
    float v[8];
    if (miss >= 0) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
            v[q] = src[(size_t)sl[q] * kLeafVoxels + (ox[q >> 2] | oy[(q >> 1) & 1] | oz[q & 1])];
    } else {
        // a corner in an absent leaf: copysign(hw, the leaf's own value at the clamped position)
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (sl[q] >= 0) {
                v[q] = src[(size_t)sl[q] * kLeafVoxels + (ox[q >> 2] | oy[(q >> 1) & 1] | oz[q & 1])];
            } else {
                const int cx = min(max(x + (q >> 2), 0), 7), cy = min(max(y + ((q >> 1) & 1), 0), 7),
                          cz = min(max(z + (q & 1), 0), 7);
                v[q] = copysignf(hw, src[(size_t)k.leaf * kLeafVoxels + ((cx << 6) | (cy << 3) | cz)]);
            }
        }
    }
    if (more) {
        const int na = (ha.x & 31) + 1;
        if (ha.x & 32) prefetch_lines(src + (size_t)(ha.x >> 6) * kLeafVoxels, 2048, lane, 0);
        prefetch_lines(ub + ha.y, 12 * na, lane, 17);
        prefetch_lines(bvox + ha.y, 4 * na, lane, 22);
        prefetch_lines(nbr + (size_t)(ha.x >> 6) * kNbr, 4 * kNbr, lane, 24);
        if (lane == 31) prefetch_l2(&chunks[min(c + 2 * ahead, n_chunks - 1)]);
    }
    const float c00 = v[0] * (1 - f.wx) + v[4] * f.wx, c01 = v[1] * (1 - f.wx) + v[5] * f.wx;
    const float c10 = v[2] * (1 - f.wx) + v[6] * f.wx, c11 = v[3] * (1 - f.wx) + v[7] * f.wx;
    const float c0 = c00 * (1 - f.wy) + c10 * f.wy, c1 = c01 * (1 - f.wy) + c11 * f.wy;
    float val = c0 * (1 - f.wz) + c1 * f.wz;
    const size_t t = (size_t)k.leaf * kLeafVoxels + k.off;
    if (bad) {
        if (k.on) atomicOr(err, kErrReach);
        val = src[t];
    }
    if (!k.on) return;
    if (dst) dst[t] = val;
    if (chk) chk[k.b] = val;
    if constexpr (GRAD) {
        const float wx[2] = {1 - f.wx, f.wx}, wy[2] = {1 - f.wy, f.wy}, wz[2] = {1 - f.wz, f.wz};
        grad[k.b] = make_float3(
            wy[0] * wz[0] * (v[4] - v[0]) + wy[1] * wz[0] * (v[6] - v[2]) + wy[0] * wz[1] * (v[5] - v[1]) +
                wy[1] * wz[1] * (v[7] - v[3]),
            wx[0] * wz[0] * (v[2] - v[0]) + wx[1] * wz[0] * (v[6] - v[4]) + wx[0] * wz[1] * (v[3] - v[1]) +
                wx[1] * wz[1] * (v[7] - v[5]),
            wx[0] * wy[0] * (v[1] - v[0]) + wx[1] * wy[0] * (v[5] - v[4]) + wx[0] * wy[1] * (v[3] - v[2]) +
                wx[1] * wy[1] * (v[7] - v[6]));
    }
}

__global__ void k_adj_scatter_band(const int* __restrict__ bvox, int nb, const float* in, float* __restrict__ phi) {
    chain_wait();
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) phi[bvox[b]] = in[b];
}

// A band voxel's foot as the gathers read it: floor offsets packed as three
// biased 7-bit fields (bit 31 marks a band voxel, other pool voxels hold 0)
// and the fractions, so a candidate costs one word and a hit one more load,
// not a chain of band-index, velocity and lambda lookups.
__device__ __forceinline__ unsigned pack_foot(const Foot& f) {
    return 0x80000000u | ((unsigned)(f.fx + 64) << 14) | ((unsigned)(f.fy + 64) << 7) | (unsigned)(f.fz + 64);
}

// Feet of the band voxels for step factor s; lam (band order) or null: 0.
__global__ void k_adj_pack(const int* __restrict__ bvox, int nb, const float3* __restrict__ ub,
                           const float* lam, float s, unsigned* __restrict__ foot_pk,
                           float4* __restrict__ foot_w) {
    chain_wait();
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
        const Foot f = foot_of(ub[b], s);
        const int sv = bvox[b];
        foot_pk[sv] = pack_foot(f);
        foot_w[sv] = make_float4(f.wx, f.wy, f.wz, lam ? lam[b] : 0.f);
    }
}

// Per leaf, the smallest and largest velocity (or displacement) component per
// axis over its band voxels (+inf and -inf without any), one warp per leaf; a
// NaN counts as 0, the offset its conversion to an integer gives.
__global__ void k_adj_urange(const float3* __restrict__ ub, const int* __restrict__ lstart, int n_leaves,
                             float* __restrict__ urange) {
    const int lane = threadIdx.x & 31;
    for (int leaf = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; leaf < n_leaves;
         leaf += (gridDim.x * blockDim.x) >> 5) {
        float lo[3], hi[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = INFINITY;
            hi[a] = -INFINITY;
        }
        for (int b = lstart[leaf] + lane; b < lstart[leaf + 1]; b += 32) {
            const float3 u3 = ub[b];
            const float u[3] = {u3.x, u3.y, u3.z};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float v = u[a] == u[a] ? u[a] : 0.f;
                lo[a] = fminf(lo[a], v);
                hi[a] = fmaxf(hi[a], v);
            }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
                hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
            }
        if (lane == 0) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                urange[(size_t)leaf * 6 + a] = lo[a];
                urange[(size_t)leaf * 6 + 3 + a] = hi[a];
            }
        }
    }
}

// urange folded over each leaf's 27-leaf neighbourhood.
__global__ void k_adj_nrange(const int* __restrict__ nbr, const float* __restrict__ urange, int n_leaves,
                             float* __restrict__ nrange) {
    for (int leaf = blockIdx.x * blockDim.x + threadIdx.x; leaf < n_leaves; leaf += gridDim.x * blockDim.x) {
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (int d = 0; d < kNbr; ++d) {
            const int s = nbr[(size_t)leaf * kNbr + d];
            if (s < 0) continue;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                lo[a] = fminf(lo[a], urange[(size_t)s * 6 + a]);
                hi[a] = fmaxf(hi[a], urange[(size_t)s * 6 + 3 + a]);
            }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            nrange[(size_t)leaf * 6 + a] = lo[a];
            nrange[(size_t)leaf * 6 + 3 + a] = hi[a];
        }
    }
}

// Candidate offsets [lo, hi] along an axis for the corners of a leaf whose
// neighbourhood's velocities lie in [ulo, uhi]: a band voxel x = b + dx has b
// in its foot cell only if dx = -f(x) - {0, 1}, f(x) = floor(s u(x)) its foot
// offset, and x lies in the 27-leaf neighbourhood (|f| <= R < 8).  Rounding
// and floor are monotone, so the offsets' extremes are those of s ulo and
// s uhi.  An empty neighbourhood gives an empty window.
__device__ __forceinline__ void window_of(float ulo, float uhi, float s, int R, int& lo, int& hi) {
    if (!(ulo <= uhi)) {
        lo = 1;
        hi = 0;
        return;
    }
    const int fa = (int)floorf(s * ulo), fb = (int)floorf(s * uhi);
    lo = max(-max(fa, fb) - 1, -1 - R);
    hi = min(-min(fa, fb), R);
}

// What a step of the backward pass does with lambda_k(b), beyond returning it
// in band order (out, when not null):
//   a fixed displacement writes it to the other lam_pool buffer;
//   a staggered field adds lambda_{k+1}(b) s grad phi_k(p(b)) to G(b) (stores
//   it on the first step) and packs the feet of the next step (k - 1) into
//   the other foot buffers.
struct BackOut {
    float* out;            // band order, or null
    float* lam_pool;       // fixed displacement: pool order, or null on the last step
    const float3* grad;    // staggered: gradient at the feet of this step, band order
    float3* G;
    int first;             // staggered: the first step of the backward pass
    const float3* ub;
    float s, s_next;
    unsigned* foot_pk;     // staggered: buffers of the next step, null on the last
    float4* foot_w;
};

__device__ __forceinline__ void back_store(const BackOut& o, int b, size_t sv, float lam_own, float lam) {
    if (o.out) o.out[b] = lam;
    if (o.lam_pool) o.lam_pool[sv] = lam;
    if (o.G) {
        const float3 g = o.grad[b];
        float3 t = o.first ? make_float3(0.f, 0.f, 0.f) : o.G[b];
        t.x += lam_own * o.s * g.x;
        t.y += lam_own * o.s * g.y;
        t.z += lam_own * o.s * g.z;
        o.G[b] = t;
    }
    if (o.foot_pk) {
        const Foot f = foot_of(o.ub[b], o.s_next);
        o.foot_pk[sv] = pack_foot(f);
        o.foot_w[sv] = make_float4(f.wx, f.wy, f.wz, lam);
    }
}

// i, j, k of corner b in candidate x's foot cell as bits 14, 7 and 0, or a
// word with other bits set when b is no corner of it.  key packs 64 - dx,
// 64 - dy, 64 - dz like a foot (with bit 31): the difference's fields are
// b - (x + floor offset), and since they stay within +-14 a field outside
// {0, 1} leaves some of its bits 1..6 set, borrows included.
constexpr unsigned kCorner = (1u << 14) | (1u << 7) | 1u;
__device__ __forceinline__ unsigned cell_key(int dx, int dy, int dz) {
    return 0x80000000u | ((unsigned)(64 - dx) << 14) | ((unsigned)(64 - dy) << 7) | (unsigned)(64 - dz);
}

// lambda of the candidate times its weight for the corner, added to acc.
__device__ __forceinline__ void add_corner(float& acc, unsigned t, const float4& w, float lam) {
    const float wx = (t >> 14) & 1u ? w.x : 1 - w.x, wy = (t >> 7) & 1u ? w.y : 1 - w.y, wz = t & 1u ? w.z : 1 - w.z;
    acc += lam * wx * wy * wz;
}

// The candidates (dy.., dz..) of Y rows of Z offsets at x offset dx, added to
// plane in (y, z) order; their words are loaded before the first is tested.
// Offsets past the window (y1, z1) test nothing; they lie within R + 8 < 16 of
// the voxel, and their leaf offset is held to the neighbourhood.
template <bool LAM, int Y, int Z>
__device__ __forceinline__ void add_candidates(float& plane, int row, int x, int cy, int cz, int dx, int dy, int dz,
                                               int y1, int z1, const unsigned* foot_pk, const float4* foot_w,
                                               const float* lam_in) {
    unsigned t[Y * Z], e[Y * Z];
#pragma unroll
    for (int q = 0; q < Y * Z; ++q) {
        const int ry = q / Z, rz = q % Z, y = cy + dy + ry, z = cz + dz + rz;
        const int ns = __shfl_sync(0xffffffffu, row, leaf_of(x) * 9 + min(leaf_of(y), 2) * 3 + min(leaf_of(z), 2));
        e[q] = (unsigned)ns * kLeafVoxels + (unsigned)voxel_off(x, y, z);
        t[q] = ~0u;
        if (ns >= 0 && dy + ry <= y1 && dz + rz <= z1) t[q] = cell_key(dx, dy + ry, dz + rz) - foot_pk[e[q]];
    }
#pragma unroll
    for (int q = 0; q < Y * Z; ++q)
        if (!(t[q] & ~kCorner)) {
            const float4 w = foot_w[e[q]];
            add_corner(plane, t[q], w, LAM ? lam_in[e[q]] : w.w);
        }
}

// Adjoint of step k as a gather:
//   lambda'(b) = sum over band voxels x of lambda(x) w_b(p(x))  (b as a corner)
// A step moves a voxel by at most R = reach voxels per axis, so b is a corner
// of x's foot cell only if x lies in b + [-1-R, R]^3, and only if it lies in
// the leaf's window (window_of); those candidates are visited in a fixed order
// (x, then y, then z ascending, one partial sum per x, added in x order),
// each x's foot taken from the same foot_of()
// as the forward step, so the transpose is exact and the sum order fixed:
// deterministic, with no sort and no float atomics.  Offsets outside the
// window hold no corner, so the window changes neither the contributing terms
// nor their order; smooth fields leave 2-3 offsets per axis, against 2R + 2.
//
// One warp per chunk of a leaf's band voxels: the window is uniform, a
// neighbour slot costs a shuffle, and the words of several candidates are
// loaded before the first is tested: kNarrow three along z; kThreeRows three
// rows of three, the whole depth of a window at a reach of one voxel; kDeep
// three rows of three, or one row of five or nine where the window is deeper,
// so that every instance adds in the same order.  Where the neighbourhood has
// one foot offset (floor(s u) equal at both ends of its range on every axis,
// the common case of a smooth field), candidate and corner correspond one to
// one, so no candidate word is read or tested; voxels off the band hold
// lambda 0 and weight 0 and add nothing.  LAM: lambda read from lam_in (pool
// order), else from the foot record.
//
// Bound: instruction issue and L1 throughput of the 8-27 candidate words and 8
// hits per voxel (32 bytes a voxel from HBM).  7.67M band voxels of a level
// set: 373 us one thread per voxel with its own gradient term, 313 us in
// chunks without it (770 instructions a chunk), 197 us with the untested
// path, 166 us with the prefetch.  16 steps back on 77k band voxels in a rough
// field, windows five and nine deep: 629 us and 1.95 ms cut into threes (which
// adds them out of order), 469 us and 1.92 ms by kDeep; 64 steps on a 256^3
// sphere, reach one: 849 us by kDeep, 822 us by kThreeRows.
enum Rows { kNarrow, kThreeRows, kDeep };

template <bool LAM, Rows ROWS>
__global__ void __launch_bounds__(256, ROWS == kNarrow ? kChunkCtas : kWideCtas)
    k_adj_lambda(const int2* __restrict__ chunks, int n_chunks, int ahead, const int* __restrict__ bvox,
                 const int* __restrict__ nbr, const float* __restrict__ nrange, const unsigned* foot_pk,
                 const float4* foot_w, const float* lam_in, int R, BackOut o) {
    const int lane = threadIdx.x & 31;
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c >= n_chunks) return;
    const int2 h = __ldg(&chunks[c]);
    const bool more = c + ahead < n_chunks;
    const int2 ha = more ? __ldg(&chunks[c + ahead]) : make_int2(0, 0);
    const Chunk k = load_chunk(h, bvox, nbr, lane);
    int x0, x1, y0, y1, z0, z1;
    const float* nr = nrange + (size_t)k.leaf * 6;
    window_of(__ldg(&nr[0]), __ldg(&nr[3]), o.s, R, x0, x1);
    window_of(__ldg(&nr[1]), __ldg(&nr[4]), o.s, R, y0, y1);
    window_of(__ldg(&nr[2]), __ldg(&nr[5]), o.s, R, z0, z1);
    if (more) {
        const int na = (ha.x & 31) + 1, leaf = ha.x >> 6;
        if (ha.x & 32) {
            const char* w = reinterpret_cast<const char*>(foot_w + (size_t)leaf * kLeafVoxels);
            prefetch_l2(w + lane * 128);
            prefetch_l2(w + 4096 + lane * 128);
            if (LAM) prefetch_lines(lam_in + (size_t)leaf * kLeafVoxels, 2048, lane, 0);
            prefetch_lines(nrange + (size_t)leaf * 6, 24, lane, 20);
        }
        prefetch_lines(bvox + ha.y, 4 * na, lane, 22);
        prefetch_lines(nbr + (size_t)leaf * kNbr, 4 * kNbr, lane, 24);
        if (lane == 31) prefetch_l2(&chunks[min(c + 2 * ahead, n_chunks - 1)]);
    }
    const int cx = k.off >> 6, cy = (k.off >> 3) & 7, cz = k.off & 7;
    chain_wait();
    float acc = 0.f;
    if (x1 - x0 == 1 && y1 - y0 == 1 && z1 - z0 == 1) {
        // one foot offset in the neighbourhood: the eight candidates are
        // the eight corners in order, (1, 1, 1) first
        unsigned e[8];
        bool there[8];
        float plane[2] = {0.f, 0.f};
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int x = cx + x0 + (q >> 2), y = cy + y0 + ((q >> 1) & 1), z = cz + z0 + (q & 1);
            const int ns = __shfl_sync(0xffffffffu, k.row, leaf_of(x) * 9 + leaf_of(y) * 3 + leaf_of(z));
            there[q] = ns >= 0;
            e[q] = (unsigned)ns * kLeafVoxels + (unsigned)voxel_off(x, y, z);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (!there[q]) continue;
            const float4 w = foot_w[e[q]];
            const float l = LAM ? lam_in[e[q]] : w.w;
            const float wx = q >> 2 ? 1 - w.x : w.x, wy = (q >> 1) & 1 ? 1 - w.y : w.y, wz = q & 1 ? 1 - w.z : w.z;
            plane[q >> 2] += l * wx * wy * wz;
        }
        acc = plane[0] + plane[1];
        x1 = x0 - 1;  // no candidate left for the general loop
    }
    for (int dx = x0; dx <= x1; ++dx) {
        const int x = cx + dx;
        float plane = 0.f;
        if (ROWS == kThreeRows || (ROWS == kDeep && z1 - z0 < 3)) {
            for (int dy = y0; dy <= y1; dy += 3)
                add_candidates<LAM, 3, 3>(plane, k.row, x, cy, cz, dx, dy, z0, y1, z1, foot_pk, foot_w, lam_in);
        } else if (ROWS == kDeep && z1 - z0 < 5) {
            for (int dy = y0; dy <= y1; ++dy)
                add_candidates<LAM, 1, 5>(plane, k.row, x, cy, cz, dx, dy, z0, y1, z1, foot_pk, foot_w, lam_in);
        } else {
            constexpr int Z = ROWS == kDeep ? 9 : 3;
            for (int dy = y0; dy <= y1; ++dy)
                for (int dz = z0; dz <= z1; dz += Z)
                    add_candidates<LAM, 1, Z>(plane, k.row, x, cy, cz, dx, dy, dz, y1, z1, foot_pk, foot_w, lam_in);
        }
        acc += plane;
    }
    if (!k.on) return;
    const size_t sv = (size_t)k.leaf * kLeafVoxels + k.off;
    back_store(o, k.b, sv, LAM ? 0.f : foot_w[sv].w, acc);
}

// k_adj_lambda for small bands and a reach of one voxel, four lanes per band
// voxel: lane q of the quad visits offset dx = q - 2 of the whole window
// [-2, 1]^3 (dy, dz ascending) and the quad sums its four partial sums in the
// fixed order ((q0 + q1) + q2) + q3: k_adj_lambda's sums.  Fills the GPU
// where one thread per band voxel leaves most warp slots empty; what is left
// is one chain of loads (voxel, 4 neighbour slots, 16 candidate words, up to
// 4 foot records), so all of each kind are issued together.
template <bool LAM>
__global__ void __launch_bounds__(256) k_adj_lambda_quad(const int* __restrict__ bvox, int nb,
                                                        const int* __restrict__ nbr,
                                                        const unsigned* foot_pk, const float4* foot_w,
                                                        const float* lam_in, BackOut o) {
    const int q = threadIdx.x & 3;
    bool first = true;
    for (long long gq = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 2; gq < nb;
         gq += ((long long)gridDim.x * blockDim.x) >> 2) {
        const int b = (int)gq;
        const int sv = bvox[b], slot = sv >> 9, off = sv & 511;
        const int cy = (off >> 3) & 7, cz = off & 7;
        const int dx = q - 2, x = (off >> 6) + dx;
        // offsets -2..1 along an axis meet at most two leaves, those of the first and the last
        const int* nrow = nbr + (size_t)slot * kNbr + leaf_of(x) * 9;
        const int ya = leaf_of(cy - 2), yb = leaf_of(cy + 1), za = leaf_of(cz - 2), zb = leaf_of(cz + 1);
        const int s4[4] = {__ldg(&nrow[ya * 3 + za]), __ldg(&nrow[ya * 3 + zb]), __ldg(&nrow[yb * 3 + za]),
                           __ldg(&nrow[yb * 3 + zb])};
        if (first) chain_wait();
        first = false;
        unsigned t[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            const int dy = (c >> 2) - 2, dz = (c & 3) - 2, y = cy + dy, z = cz + dz;
            const int u0 = leaf_of(z) == za ? s4[0] : s4[1], u1 = leaf_of(z) == za ? s4[2] : s4[3];
            const int ns = leaf_of(y) == ya ? u0 : u1;
            t[c] = ~0u;
            if (ns >= 0)
                t[c] = cell_key(dx, dy, dz) - foot_pk[(size_t)ns * kLeafVoxels + voxel_off(x, y, z)];
        }
        float acc = 0.f;
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            if (t[c] & ~kCorner) continue;
            const int y = cy + (c >> 2) - 2, z = cz + (c & 3) - 2;
            const int u0 = leaf_of(z) == za ? s4[0] : s4[1], u1 = leaf_of(z) == za ? s4[2] : s4[3];
            const size_t e = (size_t)(leaf_of(y) == ya ? u0 : u1) * kLeafVoxels + voxel_off(x, y, z);
            const float4 w = foot_w[e];
            add_corner(acc, t[c], w, LAM ? lam_in[e] : w.w);
        }
        // the quad's lanes are consecutive; sum in lane order
        const unsigned qmask = 0xFu << (threadIdx.x & 28);
        const float a1 = __shfl_sync(qmask, acc, (threadIdx.x & 31 & ~3) + 1);
        const float a2 = __shfl_sync(qmask, acc, (threadIdx.x & 31 & ~3) + 2);
        const float a3 = __shfl_sync(qmask, acc, (threadIdx.x & 31 & ~3) + 3);
        if (q == 0) back_store(o, b, (size_t)sv, LAM ? 0.f : foot_w[sv].w, ((acc + a1) + a2) + a3);
    }
}

// Transpose of the upsample.  Entry e = (b * 3 + a) * 8 + q is corner q of
// component a at band voxel b: its node, and its weight there.
__device__ __forceinline__ unsigned vel_entry(const int* __restrict__ bvox, const int4* __restrict__ origin, int e,
                                              int n, float H, float* wt) {
    const int b = e / 24, a = (e >> 3) % 3, q = e & 7;
    const int sv = bvox[b], off = sv & 511;
    const int4 o = origin[sv >> 9];
    float g[3] = {(float)(o.x + (off >> 6)) / H, (float)(o.y + ((off >> 3) & 7)) / H, (float)(o.z + (off & 7)) / H};
    int node[3];
    float w = 1.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (c != a) g[c] -= 0.5f;
        const float fl = floorf(g[c]);
        const float f = g[c] - fl;
        const int d = (q >> (2 - c)) & 1;
        node[c] = min(max((int)fl + d, 0), n - 1);
        w *= d ? f : 1 - f;
    }
    *wt = w;
    return (unsigned)((size_t)a * n * n * n + ((size_t)node[0] * n + node[1]) * n + node[2]);
}

__global__ void k_adj_vel_keys(const int* __restrict__ bvox, const int4* __restrict__ origin, int ne, int n, float H,
                               unsigned* __restrict__ keys, unsigned* __restrict__ ids) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += gridDim.x * blockDim.x) {
        float w;
        keys[e] = vel_entry(bvox, origin, e, n, H, &w);
        ids[e] = (unsigned)e;
    }
}

// Sorted entries -> source (b * 3 + a) and weight; head = 1 where a node starts.
__global__ void k_adj_vel_entries(const int* __restrict__ bvox, const int4* __restrict__ origin, int ne, int n,
                                  float H, const unsigned* __restrict__ keys, const unsigned* __restrict__ ids,
                                  int* __restrict__ ent_b, float* __restrict__ ent_w, int* __restrict__ head) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < ne; j += gridDim.x * blockDim.x) {
        const int e = (int)ids[j];
        float w;
        vel_entry(bvox, origin, e, n, H, &w);
        ent_b[j] = e >> 3;
        ent_w[j] = w;
        head[j] = j == 0 || keys[j] != keys[j - 1];
    }
}

__global__ void k_adj_vel_segments(const unsigned* __restrict__ keys, const int* __restrict__ head,
                                   const int* __restrict__ rank, int ne, int* __restrict__ seg_start,
                                   unsigned* __restrict__ seg_node) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < ne; j += gridDim.x * blockDim.x)
        if (head[j]) {
            seg_start[rank[j]] = j;
            seg_node[rank[j]] = keys[j];
        }
}

// dL/dV: eight lanes per node sum its entries (lane l takes entries l, l + 8,
// ...; the eight partial sums are folded by xor shuffles): a fixed order.
__global__ void k_adj_vel_sum(const int* __restrict__ seg_start, const unsigned* __restrict__ seg_node, int n_seg,
                              const int* __restrict__ ent_b, const float* __restrict__ ent_w,
                              const float* __restrict__ G, float* __restrict__ out) {
    const int l = threadIdx.x & 7;
    for (int base = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; (base & ~3) < n_seg;
         base += (gridDim.x * blockDim.x) >> 3) {
        const bool on = base < n_seg;
        const int e0 = on ? seg_start[base] : 0, e1 = on ? seg_start[base + 1] : 0;
        float s = 0.f;
        for (int e = e0 + l; e < e1; e += 8) s += G[ent_b[e]] * ent_w[e];
#pragma unroll
        for (int d = 4; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (on && l == 0) out[seg_node[base]] = s;
    }
}

// Chunks of the band list: leaf i's band voxels [lstart[i], lstart[i + 1])
// in groups of 32; cnt = groups per leaf, pos = their exclusive sum.
__global__ void k_adj_chunk_count(const int* __restrict__ lstart, int n, int* __restrict__ cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        cnt[i] = (lstart[i + 1] - lstart[i] + 31) >> 5;
}

__global__ void k_adj_chunk_fill(const int* __restrict__ lstart, const int* __restrict__ pos, int n,
                                 int2* __restrict__ chunks) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int j = pos[i];
        const int e = lstart[i + 1];
        for (int b = lstart[i]; b < e; b += 32) chunks[j++] = make_int2(i << 6 | (b == lstart[i] ? 32 : 0) | (min(e - b, 32) - 1), b);
    }
}

__global__ void k_adj_hash_insert(const int4* origin, int n, uint64_t* hkey, int* hval, int hcap, long long b0,
                                  long long b1, long long b2, unsigned* err);
__global__ void k_adj_nbr(const int4* origin, int n, const uint64_t* hkey, const int* hval, int hcap, long long b0,
                          long long b1, long long b2, int* nbr);

__global__ void k_adj_hash_insert(const int4* origin, int n, uint64_t* hkey, int* hval, int hcap, long long b0,
                                  long long b1, long long b2, unsigned* err) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    long long base[3] = {b0, b1, b2};
    int4 o = origin[i];
    uint64_t key = pack_key(o.x >> 3, o.y >> 3, o.z >> 3, base);
    uint32_t m = (uint32_t)hcap - 1u, p = (uint32_t)mix64(key) & m;
    for (int probe = 0; probe < hcap; ++probe) {
        unsigned long long prev =
            atomicCAS((unsigned long long*)&hkey[p], (unsigned long long)kEmptyKey, (unsigned long long)key);
        if (prev == kEmptyKey) {
            hval[p] = i;
            return;
        }
        p = (p + 1u) & m;
    }
    atomicOr(err, kErrHashFull);
}

__global__ void k_adj_nbr(const int4* origin, int n, const uint64_t* hkey, const int* hval, int hcap, long long b0,
                          long long b1, long long b2, int* nbr) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * kNbr) return;
    int i = t / kNbr, d = t % kNbr;
    HashView h{hkey, hval, hcap, {b0, b1, b2}};
    int4 o = origin[i];
    nbr[t] = hash_find_leaf(h, (long long)(o.x >> 3) + d / 9 - 1, (long long)(o.y >> 3) + (d / 3) % 3 - 1,
                            (long long)(o.z >> 3) + d % 3 - 1);
}

}  // namespace vlr

using namespace vlr;

namespace {

int blocks_for(vlr_ctx* ctx, long long n) { return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, ctx->sm_count * 8ll)); }

void adj_drop_graphs(vlr_adjoint* a) {
    if (a->fwd_exec) cudaGraphExecDestroy(a->fwd_exec);
    if (a->bwd_exec) cudaGraphExecDestroy(a->bwd_exec);
    a->fwd_exec = a->bwd_exec = nullptr;
}

void adj_free(vlr_adjoint* a) {
    adj_drop_graphs(a);
    if (a->block) {  // holds these
        a->checkpoints = nullptr;
        a->segment = a->G = nullptr;
        a->foot_pk[0] = a->foot_pk[1] = nullptr;
        a->foot_w[0] = a->foot_w[1] = nullptr;
        if (a->block_pooled) cudaFreeAsync(a->block, a->ctx->stream);
        else cudaFree(a->block);
    }
    void* ptrs[] = {a->origin, a->nbr, a->hkey, a->hval, a->phi[0], a->phi[1], a->phi_init, a->bidx, a->bvox,
                    a->ub, a->vel, a->checkpoints, a->segment, a->lam[0], a->lam[1], a->G, a->gvel, a->lstart,
                    a->chunks, a->urange, a->nrange, a->foot_pk[0], a->foot_pk[1], a->foot_w[0], a->foot_w[1],
                    a->lam_pool[0], a->lam_pool[1], a->ent_b, a->ent_w, a->seg_start, a->seg_node};
    for (void* p : ptrs) cudaFree(p);
}

// Steps between checkpoints for the caller's wish: results do not depend on
// them, memory does, 12 C bytes a band voxel for the gradients of a segment
// and 4 steps / C for the checkpoints.  A wish up to 40 stands (the plan then
// takes about the memory that sorting its entries takes at creation), and is
// never more than the steps; a longer segment is cut to where both together are
// least.
int checkpoint_steps(int wish, int steps) {
    return std::min({wish, steps, std::max(40, (int)std::ceil(std::sqrt(steps / 3.0)))});
}

// Per-axis displacement bound of one step in whole voxels: |s_k u| <= dt max|V|
// (the upsample is a convex combination of V and |cos| <= 1).
int reach_of(const float* vel, size_t nvel, double dt) {
    double m = 0.0;
    for (size_t i = 0; i < nvel; ++i) m = std::max(m, (double)std::fabs(vel[i]));
    return std::max(1, (int)std::ceil(dt * m * (1.0 + 1e-6)));
}

float step_factor(const vlr_adjoint* a, int k) {
    if (a->disp) return 1.0f;  // the displacement already holds -dt and the integrator
    // s_k = -dt cos(pi t_{k+1} / T)
    const double pi = 3.14159265358979323846;
    double t1 = a->t0 + (double)(k + 1) * a->dt;
    return (float)(-a->dt * std::cos(pi * t1 / a->period));
}

// CTAs of 256 threads (8 warps) for the chunk kernels, one chunk a warp (a
// persistent grid with the next chunk's loads held in registers spilled: the
// forward kernel 150 us against 110), and the chunks of one wave of warps.
int chunk_blocks(const vlr_adjoint* a) { return (a->n_chunks + 7) / 8; }
int chunk_wave(const vlr_ctx* ctx) { return ctx->sm_count * kChunkCtas * 8; }

// Step k from src into dst (and, in band order, into chk); with grad the
// gradient of src at the feet too.
int enqueue_forward_step(vlr_ctx* ctx, vlr_adjoint* a, int k, const float* src, float* dst, float* chk,
                         float3* grad) {
    cudaStream_t st = ctx->stream;
    const int B = chunk_blocks(a);
    if (grad)
        VLR_TIMED(ctx, "k_adj_forward",
                  VLR_CUDA(ctx, pdl_launch(k_adj_forward<true>, B, 256, 0, st, a->chunks, a->n_chunks, chunk_wave(ctx),
                                           a->bvox, a->nbr, a->ub, src, dst, chk, grad, step_factor(a, k), a->hw,
                                           ctx->d_errword)));
    else
        VLR_TIMED(ctx, "k_adj_forward",
                  VLR_CUDA(ctx, pdl_launch(k_adj_forward<false>, B, 256, 0, st, a->chunks, a->n_chunks, chunk_wave(ctx),
                                           a->bvox, a->nbr, a->ub, src, dst, chk, (float3*)nullptr, step_factor(a, k),
                                           a->hw, ctx->d_errword)));
    return VLR_OK;
}

// The forward step loop from the initial state, enqueued without waiting:
// phi_K on the band into lam[1], and for a staggered field phi_k at every
// multiple of C (but 0, which is phi_init) into the checkpoints.  Step 0 reads
// phi_init; both state buffers hold its non-band values from creation.
int adj_forward_enqueue(vlr_ctx* ctx, vlr_adjoint* a) {
    const size_t nb = (size_t)a->n_band;
    const float* src = a->phi_init;
    for (int k = 0; k < a->steps; ++k) {
        float* dst = a->phi[k & 1];
        float* chk = nullptr;
        if (k + 1 == a->steps) chk = a->lam[1];
        else if (!a->disp && (k + 1) % a->chk_every == 0) chk = a->checkpoints + (size_t)((k + 1) / a->chk_every) * nb;
        int rc = enqueue_forward_step(ctx, a, k, src, dst, chk, nullptr);
        if (rc) return rc;
        src = dst;
    }
    return VLR_OK;
}

// One step of the lambda recursion, from foot buffer `cur` (and lam_pool cur).
int enqueue_lambda_step(vlr_ctx* ctx, vlr_adjoint* a, int cur, const BackOut& o) {
    cudaStream_t st = ctx->stream;
    const int nb = a->n_band;
    const unsigned* pk = a->foot_pk[a->disp ? 0 : cur];
    const float4* w = a->foot_w[a->disp ? 0 : cur];
    // The quad wins while its voxels fit one wave (3 CTAs of 64 voxels per SM,
    // 28,416 here).  A pass of 64 steps, quad and windowed: 12,971 band voxels
    // 514 and 619 us, 19,525 542 and 639, 30,368 710 and 641, 51,229 813 and
    // 675.  It covers a reach of one voxel only.
    if (a->gather == 2 || (a->gather == 0 && a->reach == 1 && nb <= ctx->sm_count * 3 * 64)) {
        const int B = blocks_for(ctx, 4ll * nb);
        if (a->disp)
            VLR_TIMED(ctx, "k_adj_lambda",
                      VLR_CUDA(ctx, pdl_launch(k_adj_lambda_quad<true>, B, 256, 0, st, a->bvox, nb, a->nbr, pk, w,
                                               a->lam_pool[cur], o)));
        else
            VLR_TIMED(ctx, "k_adj_lambda",
                      VLR_CUDA(ctx, pdl_launch(k_adj_lambda_quad<false>, B, 256, 0, st, a->bvox, nb, a->nbr, pk, w,
                                               (const float*)nullptr, o)));
    } else {
        const int B = chunk_blocks(a);
        // Three candidate rows in flight shorten the chain of trips while the
        // warps fit two waves (4 CTAs of 8 per SM); past that the one-row
        // kernel's six CTAs cover it.  A pass of 64 steps, one row -> three:
        // 51,229 band voxels 839 -> 675 us, 77,406 886 -> 813, 152,937 1188 ->
        // 1054, 309,106 1818 -> 1802, 610,952 3052 -> 3180.
        const bool wide = a->n_chunks <= 2 * ctx->sm_count * kWideCtas * 8;
        auto launch = [&](auto* kernel, const float* lam) {
            return pdl_launch(kernel, B, 256, 0, st, a->chunks, a->n_chunks, chunk_wave(ctx), a->bvox, a->nbr, a->nrange,
                              pk, w, lam, a->reach, o);
        };
        // At a reach of one |s u| < 1 (reach_of), so foot offsets are -1 and 0
        // and windows at most three deep.
        const Rows rows = !wide ? kNarrow : a->reach == 1 ? kThreeRows : kDeep;
        auto pick = [&](auto* narrow, auto* three, auto* deep) {
            return rows == kNarrow ? narrow : rows == kThreeRows ? three : deep;
        };
        if (a->disp)
            VLR_TIMED(ctx, "k_adj_lambda", VLR_CUDA(ctx, launch(pick(k_adj_lambda<true, kNarrow>, k_adj_lambda<true, kThreeRows>,
                                                                     k_adj_lambda<true, kDeep>), (const float*)a->lam_pool[cur])));
        else
            VLR_TIMED(ctx, "k_adj_lambda", VLR_CUDA(ctx, launch(pick(k_adj_lambda<false, kNarrow>, k_adj_lambda<false, kThreeRows>,
                                                                     k_adj_lambda<false, kDeep>), (const float*)nullptr)));
    }
    return VLR_OK;
}

// The backward step loop from lambda_K in lam[1] to lambda_0 in lam[0] (and,
// for a staggered field, G), enqueued without waiting.
int adj_backward_enqueue(vlr_ctx* ctx, vlr_adjoint* a) {
    cudaStream_t st = ctx->stream;
    const int nb = a->n_band, K = a->steps, C = a->chk_every;
    int cur = 0;
    BackOut o = {};
    if (a->disp) {
        // fixed feet (packed at creation): the recursion is linear in lambda alone
        k_adj_scatter_band<<<blocks_for(ctx, nb), 256, 0, st>>>(a->bvox, nb, a->lam[1], a->lam_pool[0]);
        o.s = 1.0f;
        for (int k = K - 1; k >= 0; --k, cur ^= 1) {
            o.out = k == 0 ? a->lam[0] : nullptr;
            o.lam_pool = k == 0 ? nullptr : a->lam_pool[cur ^ 1];
            int rc = enqueue_lambda_step(ctx, a, cur, o);
            if (rc) return rc;
        }
        return VLR_OK;
    }
    VLR_TIMED(ctx, "k_adj_pack",
              k_adj_pack<<<blocks_for(ctx, nb), 256, 0, st>>>(a->bvox, nb, a->ub, a->lam[1], step_factor(a, K - 1),
                                                              a->foot_pk[0], a->foot_w[0]));
    o.G = a->G;
    o.ub = a->ub;
    for (int seg = (K - 1) / C; seg >= 0; --seg) {
        const int k0 = seg * C, k1 = std::min(K, k0 + C);
        // gradients of phi_k0 .. phi_{k1-1} at the feet, recomputing the states from the checkpoint
        const float* src = a->phi_init;
        if (seg) {
            VLR_CUDA(ctx, pdl_launch(k_adj_scatter_band, blocks_for(ctx, nb), 256, 0, st, a->bvox, nb,
                                     a->checkpoints + (size_t)seg * nb, a->phi[1]));
            src = a->phi[1];
        }
        for (int k = k0; k < k1; ++k) {
            float* dst = a->phi[(k - k0) & 1];
            int rc = enqueue_forward_step(ctx, a, k, src, k + 1 < k1 ? dst : nullptr, nullptr,
                                          a->segment + (size_t)(k - k0) * nb);
            if (rc) return rc;
            src = dst;
        }
        for (int k = k1 - 1; k >= k0; --k, cur ^= 1) {
            o.out = k == 0 ? a->lam[0] : nullptr;
            o.grad = a->segment + (size_t)(k - k0) * nb;
            o.first = k == K - 1;
            o.s = step_factor(a, k);
            o.s_next = k ? step_factor(a, k - 1) : 0.f;
            o.foot_pk = k ? a->foot_pk[cur ^ 1] : nullptr;
            o.foot_w = k ? a->foot_w[cur ^ 1] : nullptr;
            int rc = enqueue_lambda_step(ctx, a, cur, o);
            if (rc) return rc;
        }
    }
    return VLR_OK;
}

// Velocity ranges of the leaves and of their neighbourhoods, from ub.
int enqueue_ranges(vlr_ctx* ctx, vlr_adjoint* a) {
    const int n = a->n_leaves;
    k_adj_urange<<<blocks_for(ctx, 32ll * n), 256, 0, ctx->stream>>>(a->ub, a->lstart, n, a->urange);
    k_adj_nrange<<<blocks_for(ctx, n), 256, 0, ctx->stream>>>(a->nbr, a->urange, n, a->nrange);
    VLR_CUDA(ctx, cudaGetLastError());
    return VLR_OK;
}

// The chunk list from lstart (synchronises; allocates a->chunks).
int make_chunks(vlr_ctx* ctx, vlr_adjoint* a) {
    const int n = a->n_leaves;
    int* cnt = nullptr;
    VLR_CUDA(ctx, cudaMallocFromPoolAsync(&cnt, sizeof(int) * (2 * (size_t)n + 1), ctx->pool, ctx->stream));
    int* pos = cnt + n;
    k_adj_chunk_count<<<blocks_for(ctx, n), 256, 0, ctx->stream>>>(a->lstart, n, cnt);
    int rc = scan_exclusive(ctx, cnt, pos, n, pos + n);
    if (!rc) rc = read_int(ctx, pos + n, &a->n_chunks);
    cudaError_t e = rc ? cudaSuccess : cudaMalloc(&a->chunks, sizeof(int2) * std::max(a->n_chunks, 1));
    if (!rc && e == cudaSuccess) {
        k_adj_chunk_fill<<<blocks_for(ctx, n), 256, 0, ctx->stream>>>(a->lstart, pos, n, a->chunks);
        e = cudaGetLastError();
    }
    cudaFreeAsync(cnt, ctx->stream);
    return rc || e == cudaSuccess ? rc : check_cuda(ctx, e, "adjoint chunk list");
}

// Blocks up to this size come from the context's pool, which keeps them for the
// next plan; larger ones go back to the device.
constexpr size_t kPoolBlock = 32u << 20;

// Bytes of the temporaries of make_vel_entries for n_band voxels (576 each).
size_t vel_temp_bytes(int n_band) {
    const int ne = 24 * n_band;
    return ((radix_scratch_bytes(ne, 4) + 255) & ~(size_t)255) + sizeof(int) * (4 * (size_t)ne + 1);
}

// The sorted entries of upsample^T (synchronises; allocates them), by way of
// vel_temp_bytes at blk.
int make_vel_entries(vlr_ctx* ctx, vlr_adjoint* a, char* blk) {
    cudaStream_t st = ctx->stream;
    const int ne = a->n_band * 24, n = a->n_stag, B = blocks_for(ctx, ne);
    const float H = (float)a->H;
    unsigned* keys = (unsigned*)(blk + ((radix_scratch_bytes(ne, 4) + 255) & ~(size_t)255));
    unsigned* ids = keys + ne;
    int* head = (int*)(ids + ne);
    int* rank = head + ne;
    unsigned *ks = nullptr, *is = nullptr;
    VLR_CUDA(ctx, cudaMalloc(&a->ent_b, sizeof(int) * ne));
    VLR_CUDA(ctx, cudaMalloc(&a->ent_w, sizeof(float) * ne));
    k_adj_vel_keys<<<B, 256, 0, st>>>(a->bvox, a->origin, ne, n, H, keys, ids);
    int rc = radix_sort(ctx, keys, ids, ne, bits_for(3ll * n * n * n - 1), blk, &ks, &is);
    if (rc) return rc;
    k_adj_vel_entries<<<B, 256, 0, st>>>(a->bvox, a->origin, ne, n, H, ks, is, a->ent_b, a->ent_w, head);
    rc = scan_exclusive(ctx, head, rank, ne, rank + ne);
    if (!rc) rc = read_int(ctx, rank + ne, &a->n_seg);
    if (rc) return rc;
    VLR_CUDA(ctx, cudaMalloc(&a->seg_start, sizeof(int) * ((size_t)a->n_seg + 1)));
    VLR_CUDA(ctx, cudaMalloc(&a->seg_node, sizeof(unsigned) * a->n_seg));
    k_adj_vel_segments<<<B, 256, 0, st>>>(ks, head, rank, ne, a->seg_start, a->seg_node);
    VLR_CUDA(ctx, cudaMemcpyAsync(a->seg_start + a->n_seg, &ne, sizeof(int), cudaMemcpyHostToDevice, st));
    VLR_CUDA(ctx, cudaGetLastError());
    return VLR_OK;
}

// Run `enqueue` through a CUDA graph captured on first use (or directly while
// per-kernel timing is on, which brackets launches with events).
template <class F>
int run_captured(vlr_ctx* ctx, cudaGraphExec_t* exec, F&& enqueue) {
    if (ctx->timer.enabled) return enqueue();
    if (!*exec) {
        VLR_CUDA(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        const int rc = enqueue();
        cudaGraph_t g = nullptr;
        const cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
        if (rc) {
            if (g) cudaGraphDestroy(g);
            return rc;
        }
        if (e != cudaSuccess) return check_cuda(ctx, e, "cudaStreamEndCapture");
        const cudaError_t e2 = cudaGraphInstantiate(exec, g, 0);
        cudaGraphDestroy(g);
        if (e2 != cudaSuccess) return check_cuda(ctx, e2, "cudaGraphInstantiate");
    }
    VLR_CUDA(ctx, cudaGraphLaunch(*exec, ctx->stream));
    return VLR_OK;
}

// Level-set adjoint setup, leaves in list order: origins, phi_0 in f32 voxel
// units and the band (active voxel) count of each leaf.
template <typename T>
__global__ void k_adjls_gather(const int* __restrict__ list, int n, const int4* __restrict__ ls_origin,
                               const uint64_t* __restrict__ mask, const T* __restrict__ vals, int4* __restrict__ origin,
                               float* __restrict__ phi, int* __restrict__ cnt) {
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const int s = list[i];
        if (threadIdx.x == 0) origin[i] = ls_origin[s];
        for (int t = threadIdx.x; t < kLeafVoxels; t += blockDim.x)
            phi[(size_t)i * kLeafVoxels + t] = to_f(vals[(size_t)s * kLeafVoxels + t]);
        if (threadIdx.x < 32) {
            int c = threadIdx.x < 8 ? __popcll(mask[(size_t)s * 8 + threadIdx.x]) : 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
            if (threadIdx.x == 0) cnt[i] = c;
        }
    }
}

// out[b] = phi_0 at band voxel b's coordinate minus (sx, sy, sz), |s| <= 8,
// read with the adjoint's rule for missing leaves.
__global__ void k_adj_shifted(const int* __restrict__ bvox, int nb, const int* __restrict__ nbr,
                              const float* __restrict__ phi, int sx, int sy, int sz, float hw, float* __restrict__ out) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
        const int sv = bvox[b], slot = sv >> 9, off = sv & 511;
        out[b] = adj_read(phi, nbr, slot, (off >> 6) - sx, ((off >> 3) & 7) - sy, (off & 7) - sz, hw);
    }
}

// Band indices: leaf i's active voxels take pos[i], pos[i] + 1, ... in ZYX order.
__global__ void __launch_bounds__(512) k_adjls_band(const int* __restrict__ list, int n,
                                                   const uint64_t* __restrict__ mask, const int* __restrict__ pos,
                                                   int* __restrict__ bidx, int* __restrict__ bvox) {
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const int s = list[i];
        const int t = threadIdx.x, w = t >> 6;
        const uint64_t word = mask[(size_t)s * 8 + w];
        int before = __popcll(word & ((1ull << (t & 63)) - 1ull));
        for (int q = 0; q < w; ++q) before += __popcll(mask[(size_t)s * 8 + q]);
        const size_t v = (size_t)i * kLeafVoxels + t;
        if ((word >> (t & 63)) & 1ull) {
            const int b = pos[i] + before;
            bidx[v] = b;
            bvox[b] = (int)v;
        } else {
            bidx[v] = -1;
        }
    }
}

}  // namespace

extern "C" {

int vlr_adj_create_level_set(vlr_ctx* ctx, vlr_level_set* ls, int steps, int checkpoint_every, vlr_adjoint** out) {
    if (!ctx || !ls || !out) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    if (steps < 1 || checkpoint_every < 1) return set_error(ctx, VLR_ERR_INVALID, "bad adjoint parameters");
    if (ls->n_grids != 1) return set_error(ctx, VLR_ERR_UNSUPPORTED, "level-set adjoint of a single grid only");
    if (ls->vel_kind != MVEL_CONSTANT && ls->vel_kind != MVEL_CURL)
        return set_error(ctx, VLR_ERR_UNSUPPORTED,
                         "level-set adjoint needs a time-independent velocity (constant or curl noise)");
    if (ls->key_bits > kKeyBits) return set_error(ctx, VLR_ERR_EXTENT, "grid too wide for the adjoint's hash");
    *out = nullptr;
    cudaStream_t st = ctx->stream;
    int n = 0;
    int rc = read_int(ctx, ls->scalars, &n);
    if (rc) return rc;
    if (n <= 0) return set_error(ctx, VLR_ERR_INVALID, "empty level set");
    if ((long long)n * kLeafVoxels >= (1ll << 31)) return set_error(ctx, VLR_ERR_CAPACITY, "too many leaves");
    const vlr::MGridParams& P = ls->h_params[0];
    vlr_adjoint* a = new vlr_adjoint();
    a->ctx = ctx;
    a->n_leaves = n;
    a->hw = P.hw;
    a->dt = ls->sp.dt;
    a->t0 = ls->sp.t0;
    a->period = 1.0;
    a->steps = steps;
    a->chk_every = checkpoint_every;
    a->disp = 1;
    for (int k = 0; k < 3; ++k) a->base[k] = P.base[k];
    auto fail = [&](int code) {
        adj_free(a);
        delete a;
        return code;
    };
    const size_t pool = (size_t)n * kLeafVoxels;
    int* cnt = nullptr;  // n + 1 counts, then n + 1 positions
#define ADJ_MALLOC(p, bytes) \
    do { cudaError_t e_ = cudaMalloc(&(p), (bytes)); if (e_ != cudaSuccess) return fail(check_cuda(ctx, e_, "cudaMalloc")); } while (0)
    ADJ_MALLOC(a->origin, sizeof(int4) * n);
    ADJ_MALLOC(a->phi_init, sizeof(float) * pool);
    ADJ_MALLOC(a->bidx, sizeof(int) * pool);
    ADJ_MALLOC(cnt, sizeof(int) * (2 * (size_t)n + 4));
    int* pos = cnt + n + 2;
    const int gb = (int)std::min<long long>(n, (long long)ctx->sm_count * 8);
    if (ls->precision == VLR_PREC_F16)
        k_adjls_gather<__half><<<gb, 256, 0, st>>>(ls->list, n, ls->origin, ls->mask, (const __half*)ls->vals[0],
                                                  a->origin, a->phi_init, cnt);
    else
        k_adjls_gather<float><<<gb, 256, 0, st>>>(ls->list, n, ls->origin, ls->mask, (const float*)ls->vals[0],
                                                 a->origin, a->phi_init, cnt);
    rc = scan_exclusive(ctx, cnt, pos, n, pos + n);
    if (rc) {
        cudaFree(cnt);
        return fail(rc);
    }
    int nb = 0;
    rc = read_int(ctx, pos + n, &nb);
    if (rc || nb <= 0) {
        cudaFree(cnt);
        return fail(rc ? rc : set_error(ctx, VLR_ERR_INVALID, "empty band"));
    }
    a->n_band = nb;
    a->hcap = 64;
    while ((size_t)a->hcap < 2 * (size_t)n) a->hcap <<= 1;
    ADJ_MALLOC(a->bvox, sizeof(int) * nb);
    ADJ_MALLOC(a->nbr, sizeof(int) * kNbr * (size_t)n);
    ADJ_MALLOC(a->hkey, sizeof(uint64_t) * a->hcap);
    ADJ_MALLOC(a->hval, sizeof(int) * a->hcap);
    ADJ_MALLOC(a->phi[0], sizeof(float) * pool);
    ADJ_MALLOC(a->phi[1], sizeof(float) * pool);
    ADJ_MALLOC(a->ub, sizeof(float3) * nb);
    ADJ_MALLOC(a->lam[0], sizeof(float) * nb);
    ADJ_MALLOC(a->lam[1], sizeof(float) * nb);
    ADJ_MALLOC(a->lstart, sizeof(int) * ((size_t)n + 1));
    ADJ_MALLOC(a->foot_pk[0], sizeof(unsigned) * pool);
    ADJ_MALLOC(a->foot_w[0], sizeof(float4) * pool);
    ADJ_MALLOC(a->lam_pool[0], sizeof(float) * pool);
    ADJ_MALLOC(a->lam_pool[1], sizeof(float) * pool);
    ADJ_MALLOC(a->urange, sizeof(float) * 6 * (size_t)n);
    ADJ_MALLOC(a->nrange, sizeof(float) * 6 * (size_t)n);
#undef ADJ_MALLOC
    for (float* p : a->phi)
        VLR_CUDA(ctx, cudaMemcpyAsync(p, a->phi_init, sizeof(float) * pool, cudaMemcpyDeviceToDevice, st));
    VLR_CUDA(ctx, cudaMemcpyAsync(a->lstart, pos, sizeof(int) * ((size_t)n + 1), cudaMemcpyDeviceToDevice, st));
    VLR_CUDA(ctx, cudaMemsetAsync(a->foot_pk[0], 0, sizeof(unsigned) * pool, st));
    // off the band: weight 0, lambda 0
    VLR_CUDA(ctx, cudaMemsetAsync(a->foot_w[0], 0, sizeof(float4) * pool, st));
    for (float* p : a->lam_pool) VLR_CUDA(ctx, cudaMemsetAsync(p, 0, sizeof(float) * pool, st));
    VLR_CUDA(ctx, cudaMemsetAsync(a->hkey, 0xFF, sizeof(uint64_t) * a->hcap, st));  // kEmptyKey
    k_adjls_band<<<gb, 512, 0, st>>>(ls->list, n, ls->mask, pos, a->bidx, a->bvox);
    k_adj_hash_insert<<<(n + 255) / 256, 256, 0, st>>>(a->origin, n, a->hkey, a->hval, a->hcap, a->base[0], a->base[1],
                                                       a->base[2], ctx->d_errword);
    k_adj_nbr<<<(int)(((size_t)n * kNbr + 255) / 256), 256, 0, st>>>(a->origin, n, a->hkey, a->hval, a->hcap,
                                                                      a->base[0], a->base[1], a->base[2], a->nbr);
    unsigned* d_max = reinterpret_cast<unsigned*>(cnt);  // the counts are consumed
    VLR_CUDA(ctx, cudaMemsetAsync(d_max, 0, sizeof(unsigned), st));
    if (ls->vel_kind == MVEL_CURL)
        k_m_feet<MVEL_CURL><<<gb, 128, 0, st>>>(a->origin, n, a->bidx, ls->d_params, ls->d_tab, (float)ls->sp.dt,
                                                ls->sp.integrator, a->ub, d_max, ctx->d_errword);
    else
        k_m_feet<MVEL_CONSTANT><<<gb, 128, 0, st>>>(a->origin, n, a->bidx, ls->d_params, ls->d_tab,
                                                    (float)ls->sp.dt, ls->sp.integrator, a->ub, d_max,
                                                    ctx->d_errword);
    VLR_CUDA(ctx, cudaGetLastError());
    // the displacement is fixed: its feet, ranges and chunks stand for every pass
    k_adj_pack<<<blocks_for(ctx, nb), 256, 0, st>>>(a->bvox, nb, a->ub, nullptr, 1.0f, a->foot_pk[0], a->foot_w[0]);
    rc = enqueue_ranges(ctx, a);
    if (!rc) rc = make_chunks(ctx, a);
    if (rc) {
        cudaFree(cnt);
        return fail(rc);
    }
    unsigned mbits = 0;
    VLR_CUDA(ctx, cudaMemcpyAsync(&mbits, d_max, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    cudaError_t e = cudaStreamSynchronize(st);
    cudaFree(cnt);
    if (e != cudaSuccess) return fail(check_cuda(ctx, e, "level-set adjoint setup"));
    rc = consume_device_errors(ctx, "vlr_adj_create_level_set");
    if (rc) return fail(rc);
    float mx;
    std::memcpy(&mx, &mbits, sizeof(mx));
    a->reach = std::max(1, (int)std::ceil((double)mx * (1.0 + 1e-6)));
    if (a->reach > 6) return fail(set_error(ctx, VLR_ERR_REACH, "backtrace displacement exceeds 6 voxels per step"));
    *out = a;
    return VLR_OK;
}

int vlr_adj_set_gather(vlr_ctx* ctx, vlr_adjoint* a, int mode) {
    if (!ctx || !a) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    if (mode < 0 || mode > 2) return set_error(ctx, VLR_ERR_INVALID, "gather mode must be 0, 1 or 2");
    if (mode == 2 && a->reach != 1)
        return set_error(ctx, VLR_ERR_INVALID, "the quad gather covers a reach of one voxel per step only");
    if (mode != a->gather) adj_drop_graphs(a);
    a->gather = mode;
    return VLR_OK;
}

int vlr_adj_shifted_phi0(vlr_ctx* ctx, const vlr_adjoint* a, int sx, int sy, int sz, float* d_out) {
    if (!ctx || !a || !d_out) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    if (sx < -8 || sx > 8 || sy < -8 || sy > 8 || sz < -8 || sz > 8)
        return set_error(ctx, VLR_ERR_INVALID, "shift beyond 8 voxels");
    k_adj_shifted<<<blocks_for(ctx, a->n_band), 256, 0, ctx->stream>>>(a->bvox, a->n_band, a->nbr, a->phi_init, sx,
                                                                        sy, sz, a->hw, d_out);
    VLR_CUDA(ctx, cudaGetLastError());
    return VLR_OK;
}

int vlr_adj_displacement(vlr_ctx* ctx, const vlr_adjoint* a, float* out) {
    if (!ctx || !a || !out) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    if (!a->disp) return set_error(ctx, VLR_ERR_UNSUPPORTED, "not a level-set adjoint");
    VLR_CUDA(ctx, cudaMemcpyAsync(out, a->ub, sizeof(float3) * a->n_band, cudaMemcpyDeviceToHost, ctx->stream));
    VLR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return VLR_OK;
}

int vlr_adj_create(vlr_ctx* ctx, const int32_t* origins, const uint64_t* masks, const float* phi, size_t n_leaves,
                   float half_width, const float* vel, int n_stag, double stag_cell, double dt, double period,
                   double t0, int steps, int checkpoint_every, vlr_adjoint** out) {
    if (!ctx || !origins || !masks || !phi || !vel || !out || n_leaves == 0)
        return set_error(ctx, VLR_ERR_INVALID, "null argument");
    if (n_stag < 2 || steps < 1 || checkpoint_every < 1 || !(stag_cell > 0.0) || !(dt > 0.0))
        return set_error(ctx, VLR_ERR_INVALID, "bad adjoint parameters");
    *out = nullptr;
    vlr_adjoint* a = new vlr_adjoint();
    a->ctx = ctx;
    a->n_leaves = (int)n_leaves;
    a->hw = half_width;
    a->n_stag = n_stag;
    a->H = stag_cell;
    a->dt = dt;
    a->period = period;
    a->t0 = t0;
    a->steps = steps;
    a->chk_every = checkpoint_steps(checkpoint_every, steps);
    auto fail = [&](int rc) {
        adj_free(a);
        delete a;
        return rc;
    };
    int rc = choose_base(ctx, origins, n_leaves, a->base);
    if (rc) return fail(rc);
    // band: active voxels, in leaf order then ZYX
    std::vector<int> bidx(n_leaves * 512, -1), bvox, lstart;
    for (size_t i = 0; i < n_leaves; ++i) {
        lstart.push_back((int)bvox.size());
        for (int off = 0; off < 512; ++off)
            if ((masks[8 * i + (off >> 6)] >> (off & 63)) & 1ull) {
                bidx[i * 512 + off] = (int)bvox.size();
                bvox.push_back((int)(i * 512 + off));
            }
    }
    lstart.push_back((int)bvox.size());
    a->n_band = (int)bvox.size();
    if (a->n_band == 0) return fail(set_error(ctx, VLR_ERR_INVALID, "empty band"));
    const size_t nb = (size_t)a->n_band;
    a->hcap = 64;
    while ((size_t)a->hcap < 2 * n_leaves) a->hcap <<= 1;
    std::vector<int4> o4(n_leaves);
    for (size_t i = 0; i < n_leaves; ++i) o4[i] = make_int4(origins[3 * i], origins[3 * i + 1], origins[3 * i + 2], 0);
    size_t nvel = 3ull * n_stag * n_stag * n_stag;
    if (nb > (size_t)INT32_MAX / 24) return fail(set_error(ctx, VLR_ERR_CAPACITY, "band too large for a staggered adjoint"));
#define ADJ_MALLOC(p, bytes) \
    do { cudaError_t e_ = cudaMalloc(&(p), (bytes)); if (e_ != cudaSuccess) return fail(check_cuda(ctx, e_, "cudaMalloc")); } while (0)
    ADJ_MALLOC(a->origin, sizeof(int4) * n_leaves);
    ADJ_MALLOC(a->nbr, sizeof(int) * kNbr * n_leaves);
    ADJ_MALLOC(a->hkey, sizeof(uint64_t) * a->hcap);
    ADJ_MALLOC(a->hval, sizeof(int) * a->hcap);
    ADJ_MALLOC(a->phi[0], sizeof(float) * 512 * n_leaves);
    ADJ_MALLOC(a->phi[1], sizeof(float) * 512 * n_leaves);
    ADJ_MALLOC(a->phi_init, sizeof(float) * 512 * n_leaves);
    ADJ_MALLOC(a->bidx, sizeof(int) * 512 * n_leaves);
    ADJ_MALLOC(a->bvox, sizeof(int) * nb);
    ADJ_MALLOC(a->ub, sizeof(float3) * nb);
    ADJ_MALLOC(a->vel, sizeof(float) * nvel);
    ADJ_MALLOC(a->lam[0], sizeof(float) * nb);
    ADJ_MALLOC(a->lam[1], sizeof(float) * nb);
    ADJ_MALLOC(a->gvel, sizeof(float) * nvel);
    ADJ_MALLOC(a->lstart, sizeof(int) * (n_leaves + 1));
    ADJ_MALLOC(a->urange, sizeof(float) * 6 * n_leaves);
    ADJ_MALLOC(a->nrange, sizeof(float) * 6 * n_leaves);
    cudaStream_t st = ctx->stream;
    VLR_CUDA(ctx, cudaMemcpyAsync(a->lstart, lstart.data(), sizeof(int) * (n_leaves + 1), cudaMemcpyHostToDevice, st));
    VLR_CUDA(ctx, cudaMemcpyAsync(a->origin, o4.data(), sizeof(int4) * n_leaves, cudaMemcpyHostToDevice, st));
    VLR_CUDA(ctx, cudaMemcpyAsync(a->phi_init, phi, sizeof(float) * 512 * n_leaves, cudaMemcpyHostToDevice, st));
    for (float* p : a->phi)
        VLR_CUDA(ctx, cudaMemcpyAsync(p, a->phi_init, sizeof(float) * 512 * n_leaves, cudaMemcpyDeviceToDevice, st));
    VLR_CUDA(ctx, cudaMemcpyAsync(a->bidx, bidx.data(), sizeof(int) * 512 * n_leaves, cudaMemcpyHostToDevice, st));
    VLR_CUDA(ctx, cudaMemcpyAsync(a->bvox, bvox.data(), sizeof(int) * nb, cudaMemcpyHostToDevice, st));
    a->reach = reach_of(vel, nvel, dt);
    if (a->reach > 6) return fail(set_error(ctx, VLR_ERR_REACH, "dt * max|V| exceeds 6 voxels per step"));
    VLR_CUDA(ctx, cudaMemcpyAsync(a->vel, vel, sizeof(float) * nvel, cudaMemcpyHostToDevice, st));
    std::vector<uint64_t> hk(a->hcap, kEmptyKey);
    VLR_CUDA(ctx, cudaMemcpyAsync(a->hkey, hk.data(), sizeof(uint64_t) * a->hcap, cudaMemcpyHostToDevice, st));
    k_adj_hash_insert<<<(int)((n_leaves + 255) / 256), 256, 0, st>>>(a->origin, (int)n_leaves, a->hkey, a->hval,
                                                                     a->hcap, a->base[0], a->base[1], a->base[2],
                                                                     ctx->d_errword);
    k_adj_nbr<<<(int)((n_leaves * kNbr + 255) / 256), 256, 0, st>>>(a->origin, (int)n_leaves, a->hkey, a->hval, a->hcap,
                                                                    a->base[0], a->base[1], a->base[2], a->nbr);
    k_adj_upsample<<<blocks_for(ctx, nb), 256, 0, st>>>(a->bvox, a->origin, (int)nb, a->vel, n_stag, (float)stag_cell,
                                                        a->ub);
    rc = enqueue_ranges(ctx, a);
    if (!rc) rc = make_chunks(ctx, a);
    if (rc) return fail(rc);
    // one block, first for the temporaries of the entries, then for the buffers of the passes
    const size_t n_chk = (size_t)(steps / a->chk_every) + 1, pool = 512 * n_leaves;
    const struct {
        void** p;
        size_t bytes;
    } own[] = {{(void**)&a->checkpoints, sizeof(float) * nb * n_chk},
               {(void**)&a->segment, sizeof(float3) * nb * a->chk_every},
               {(void**)&a->G, sizeof(float3) * nb},
               {(void**)&a->foot_pk[0], sizeof(unsigned) * pool},
               {(void**)&a->foot_pk[1], sizeof(unsigned) * pool},
               {(void**)&a->foot_w[0], sizeof(float4) * pool},
               {(void**)&a->foot_w[1], sizeof(float4) * pool}};
    size_t bytes = 0;
    for (const auto& o : own) bytes += (o.bytes + 255) & ~(size_t)255;
    bytes = std::max(bytes, vel_temp_bytes(a->n_band));
    a->block_pooled = bytes <= kPoolBlock;
    const cudaError_t eb = a->block_pooled ? cudaMallocFromPoolAsync((void**)&a->block, bytes, ctx->pool, st)
                                           : cudaMalloc((void**)&a->block, bytes);
    if (eb != cudaSuccess) return fail(check_cuda(ctx, eb, "adjoint buffers"));
#undef ADJ_MALLOC
    rc = make_vel_entries(ctx, a, a->block);
    if (rc) return fail(rc);
    bytes = 0;
    for (const auto& o : own) {
        *o.p = a->block + bytes;
        bytes += (o.bytes + 255) & ~(size_t)255;
    }
    for (int q = 0; q < 2; ++q) {  // off the band: no foot, weight 0, lambda 0
        VLR_CUDA(ctx, cudaMemsetAsync(a->foot_pk[q], 0, sizeof(unsigned) * pool, st));
        VLR_CUDA(ctx, cudaMemsetAsync(a->foot_w[q], 0, sizeof(float4) * pool, st));
    }
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(check_cuda(ctx, e, "adjoint setup"));
    rc = consume_device_errors(ctx, "vlr_adj_create");
    if (rc) return fail(rc);
    *out = a;
    return VLR_OK;
}

int vlr_adj_band(vlr_ctx* ctx, const vlr_adjoint* a, int32_t* coords, size_t cap, size_t* n) {
    if (!ctx || !a || !n) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    *n = (size_t)a->n_band;
    if (!coords) return VLR_OK;
    if (cap < *n) return set_error(ctx, VLR_ERR_CAPACITY, "coordinate buffer too small");
    std::vector<int> bvox(a->n_band);
    std::vector<int4> o4(a->n_leaves);
    VLR_CUDA(ctx, cudaMemcpy(bvox.data(), a->bvox, sizeof(int) * a->n_band, cudaMemcpyDeviceToHost));
    VLR_CUDA(ctx, cudaMemcpy(o4.data(), a->origin, sizeof(int4) * a->n_leaves, cudaMemcpyDeviceToHost));
    for (int b = 0; b < a->n_band; ++b) {
        int s = bvox[b] >> 9, off = bvox[b] & 511;
        coords[3 * b] = o4[s].x + (off >> 6);
        coords[3 * b + 1] = o4[s].y + ((off >> 3) & 7);
        coords[3 * b + 2] = o4[s].z + (off & 7);
    }
    return VLR_OK;
}

int vlr_adj_set_inputs(vlr_ctx* ctx, vlr_adjoint* a, const float* phi0_band, const float* vel) {
    if (!ctx || !a) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    if (vel && a->disp) return set_error(ctx, VLR_ERR_UNSUPPORTED, "a level-set adjoint has no velocity field input");
    cudaStream_t st = ctx->stream;
    if (phi0_band) {
        VLR_CUDA(ctx, cudaMemcpyAsync(a->lam[1], phi0_band, sizeof(float) * a->n_band, cudaMemcpyHostToDevice, st));
        k_adj_scatter_band<<<blocks_for(ctx, a->n_band), 256, 0, st>>>(a->bvox, a->n_band, a->lam[1], a->phi_init);
    }
    if (vel) {
        size_t nvel = 3ull * a->n_stag * a->n_stag * a->n_stag;
        const int reach = reach_of(vel, nvel, a->dt);
        if (reach > 6) return set_error(ctx, VLR_ERR_REACH, "dt * max|V| exceeds 6 voxels per step");
        if (reach != a->reach) adj_drop_graphs(a);
        a->reach = reach;
        VLR_CUDA(ctx, cudaMemcpyAsync(a->vel, vel, sizeof(float) * nvel, cudaMemcpyHostToDevice, st));
        k_adj_upsample<<<blocks_for(ctx, a->n_band), 256, 0, st>>>(a->bvox, a->origin, a->n_band, a->vel, a->n_stag,
                                                                   (float)a->H, a->ub);
        const int rc = enqueue_ranges(ctx, a);
        if (rc) return rc;
    }
    VLR_CUDA(ctx, cudaGetLastError());
    VLR_CUDA(ctx, cudaStreamSynchronize(st));
    return VLR_OK;
}

// Forward K steps from the initial state; checkpoints every C steps; writes
// phi_K on the band (host, n_band floats) when phi_k_band is not null.
int vlr_adj_forward_device(vlr_ctx* ctx, vlr_adjoint* a, float* d_phi_k_band) {
    if (!ctx || !a) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    int rc = run_captured(ctx, &a->fwd_exec, [&]() { return adj_forward_enqueue(ctx, a); });
    if (rc) return rc;
    if (d_phi_k_band)
        VLR_CUDA(ctx, cudaMemcpyAsync(d_phi_k_band, a->lam[1], sizeof(float) * a->n_band, cudaMemcpyDeviceToDevice,
                                      ctx->stream));
    return VLR_OK;
}

int vlr_adj_forward(vlr_ctx* ctx, vlr_adjoint* a, float* phi_k_band) {
    int rc = vlr_adj_forward_device(ctx, a, nullptr);
    if (rc) return rc;
    if (phi_k_band)
        VLR_CUDA(ctx, cudaMemcpyAsync(phi_k_band, a->lam[1], sizeof(float) * a->n_band, cudaMemcpyDeviceToHost,
                                      ctx->stream));
    return consume_device_errors(ctx, "vlr_adj_forward");  // waits for the stream
}

// Backward pass (vlr_adj_forward must have run): grad_phik_band = dL/dphi_K
// on the band; writes dL/dphi_0 (n_band) and dL/dV (3 n^3), host buffers.
int vlr_adj_backward_device(vlr_ctx* ctx, vlr_adjoint* a, const float* d_grad_phik_band, float* d_grad_phi0_band,
                            float* d_grad_vel) {
    if (!ctx || !a || !d_grad_phik_band) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    if (d_grad_vel && a->disp) return set_error(ctx, VLR_ERR_UNSUPPORTED, "a level-set adjoint has no velocity gradient");
    cudaStream_t st = ctx->stream;
    const size_t nb = (size_t)a->n_band;
    if (d_grad_phik_band != a->lam[1])
        VLR_CUDA(ctx, cudaMemcpyAsync(a->lam[1], d_grad_phik_band, sizeof(float) * nb, cudaMemcpyDeviceToDevice, st));
    int rc = run_captured(ctx, &a->bwd_exec, [&]() { return adj_backward_enqueue(ctx, a); });
    if (rc) return rc;
    float* lam = a->lam[0];
    a->lam_final = lam;
    if (d_grad_phi0_band)
        VLR_CUDA(ctx, cudaMemcpyAsync(d_grad_phi0_band, lam, sizeof(float) * nb, cudaMemcpyDeviceToDevice, st));
    if (d_grad_vel) {
        size_t nvel = 3ull * a->n_stag * a->n_stag * a->n_stag;
        VLR_CUDA(ctx, cudaMemsetAsync(d_grad_vel, 0, sizeof(float) * nvel, st));
        VLR_TIMED(ctx, "k_adj_emit_vel",
                  k_adj_vel_sum<<<blocks_for(ctx, 8ll * a->n_seg), 256, 0, st>>>(
                      a->seg_start, a->seg_node, a->n_seg, a->ent_b, a->ent_w, reinterpret_cast<const float*>(a->G),
                      d_grad_vel));
        VLR_CUDA(ctx, cudaGetLastError());
    }
    return VLR_OK;
}

int vlr_adj_backward(vlr_ctx* ctx, vlr_adjoint* a, const float* grad_phik_band, float* grad_phi0_band,
                     float* grad_vel) {
    if (!ctx || !a || !grad_phik_band) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    if (grad_vel && a->disp) return set_error(ctx, VLR_ERR_UNSUPPORTED, "a level-set adjoint has no velocity gradient");
    cudaStream_t st = ctx->stream;
    const size_t nb = (size_t)a->n_band;
    VLR_CUDA(ctx, cudaMemcpyAsync(a->lam[1], grad_phik_band, sizeof(float) * nb, cudaMemcpyHostToDevice, st));
    int rc = vlr_adj_backward_device(ctx, a, a->lam[1], nullptr, grad_vel ? a->gvel : nullptr);
    if (rc) return rc;
    if (grad_phi0_band)
        VLR_CUDA(ctx, cudaMemcpyAsync(grad_phi0_band, a->lam_final, sizeof(float) * nb, cudaMemcpyDeviceToHost, st));
    if (grad_vel)
        VLR_CUDA(ctx, cudaMemcpyAsync(grad_vel, a->gvel, sizeof(float) * 3ull * a->n_stag * a->n_stag * a->n_stag,
                                      cudaMemcpyDeviceToHost, st));
    return consume_device_errors(ctx, "vlr_adj_backward");  // waits for the stream
}

void vlr_adj_destroy(vlr_adjoint* a) {
    if (!a) return;
    if (a->ctx) cudaStreamSynchronize(a->ctx->stream);
    adj_free(a);
    delete a;
}

}  // extern "C"
