// Reference-semantics kernels: the Sharc.Volrus advection step on flat device
// leaves, bit-exact with the crate's CPU code.
//   k_advect_ref      advect_level_set            src/tools/advection.rs:32-56
//   k_sample_points   sample_trilinear            src/tools/interpolation.rs:11-48
//   k_cross_sign, k_cross_bits, k_emit_crossings
//                     find_zero_crossings         src/tools/level_set_track.rs:14-47
//   k_rebuild_window  rebuild_narrow_band         src/tools/level_set_track.rs:80-114
//   k_rebuild_brute   (same, any half-width)
//   k_trim            trim_narrow_band            src/tools/level_set_track.rs:53-68
//   k_sphere          make_level_set_sphere       src/tools/sphere.rs:17-59
// One CTA works on one 8^3 leaf; activity masks are produced with warp ballots.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "ref_ops.hpp"

namespace vlr {

// ------------------------------------------------------------- advection

// Velocity comes from three grids (VelocityField::sample,
// src/tools/advection.rs:18-24).  The output keeps the input's activity mask;
// inactive voxels read background (the leaf is freshly allocated in the
// reference, src/tree/internal.rs:127-143).
//
// One warp per leaf.  It lists the leaf's active voxels (about 30 % of them)
// so that its lanes work on 32 of them at a time, and finds the velocity
// grids' leaves at the first one by hash; every other lookup goes from those
// leaves through their neighbour rows, the hash serving only samples that
// leave the 27-leaf neighbourhood.  SAME: the velocity grids share their
// transform (as a VelocityField's usually do), so the f64 position and the
// fractions are computed once for the three.  Results gather in a shared tile
// and leave as whole lines.
//
// Bound: instruction issue and load latency of 32 slot lookups and 32 corner
// reads per voxel (10.5 KB a leaf from HBM with three velocity grids).  17.5k
// leaves, 2.9M active voxels (L2-resident): 396 us with a hash search per
// sample and four voxels a thread, 359 us listed and hinted, 196 us with the
// branch-free slots of read_cell, 161 us in CTAs of two leaves at 64 registers
// (eight leaves a CTA wait for the fullest one; four: 163 us).
constexpr int kAdvWarps = 2;

template <bool SAME>
__global__ void __launch_bounds__(32 * kAdvWarps, 16) k_advect_ref(GridView g, GridView vx, GridView vy, GridView vz,
                                                              double dt, float* __restrict__ out_values,
                                                              uint64_t* __restrict__ out_mask,
                                                              int* __restrict__ nonempty) {
    __shared__ unsigned short s_list[kAdvWarps][kLeafVoxels];
    __shared__ __align__(16) float s_out[kAdvWarps][kLeafVoxels];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int slot = blockIdx.x * kAdvWarps + w;
    if (slot >= g.n) return;
    const int4 o = g.origin[slot];
    // lane l lists bits [16 (l & 3), + 16) of mask word l >> 2
    const uint64_t word = g.mask[(size_t)slot * 8 + (lane >> 2)];
    unsigned bits = (unsigned)(word >> (16 * (lane & 3))) & 0xffffu;
    const int c = __popc(bits);
    int incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
    }
    const int count = __shfl_sync(0xffffffffu, incl, 31);
    if ((lane & 3) == 0) out_mask[(size_t)slot * 8 + (lane >> 2)] = word;
    if (lane == 0) nonempty[slot] = count > 0;
    if (count == 0) return;  // dropped from the output
    for (int p = incl - c; bits; bits &= bits - 1u)
        s_list[w][p++] = (unsigned short)((lane >> 2) * 64 + 16 * (lane & 3) + __ffs(bits) - 1);
    float4* tile = reinterpret_cast<float4*>(s_out[w]);
    const float bg = g.background;
#pragma unroll
    for (int q = 0; q < 4; ++q) tile[q * 32 + lane] = make_float4(bg, bg, bg, bg);
    __syncwarp();
    auto world = [&](int off, double* p) {
        index_to_world_ref(g.mat, o.x + (off >> 6), o.y + ((off >> 3) & 7), o.z + (off & 7), p);
    };
    Hint hv[3];
    {
        double p[3];
        world(s_list[w][0], p);
        const GridView* v = lane == 1 ? &vy : (lane == 2 ? &vz : &vx);
        Hint h;
        if (lane < 3) {
            const Cell q = cell_of(*v, p[0], p[1], p[2]);
            h = hint_at(*v, q.i, q.j, q.k);
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            hv[a].slot = __shfl_sync(0xffffffffu, h.slot, a);
            hv[a].x = __shfl_sync(0xffffffffu, h.x, a);
            hv[a].y = __shfl_sync(0xffffffffu, h.y, a);
            hv[a].z = __shfl_sync(0xffffffffu, h.z, a);
        }
    }
    Hint hg;
    hg.slot = slot;
    hg.x = o.x >> 3;
    hg.y = o.y >> 3;
    hg.z = o.z >> 3;
    for (int i = lane; i < count; i += 32) {
        const int off = s_list[w][i];
        double p[3];
        world(off, p);
        double v0, v1, v2;
        if (SAME) {
            const Cell q = cell_of(vx, p[0], p[1], p[2]);
            v0 = (double)read_cell(vx, q, hv[0]);
            v1 = (double)read_cell(vy, q, hv[1]);
            v2 = (double)read_cell(vz, q, hv[2]);
        } else {
            v0 = (double)sample_trilinear_ref(vx, p[0], p[1], p[2], hv[0]);
            v1 = (double)sample_trilinear_ref(vy, p[0], p[1], p[2], hv[1]);
            v2 = (double)sample_trilinear_ref(vz, p[0], p[1], p[2], hv[2]);
        }
        s_out[w][off] = sample_trilinear_ref(g, __dsub_rn(p[0], __dmul_rn(dt, v0)), __dsub_rn(p[1], __dmul_rn(dt, v1)),
                                             __dsub_rn(p[2], __dmul_rn(dt, v2)), hg);
    }
    __syncwarp();
    float4* out = reinterpret_cast<float4*>(out_values + (size_t)slot * kLeafVoxels);
#pragma unroll
    for (int q = 0; q < 4; ++q) out[q * 32 + lane] = tile[q * 32 + lane];
}

__global__ void k_sample_points(GridView g, const double* __restrict__ pts, int n, float* __restrict__ out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = sample_trilinear_ref(g, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
}

// ------------------------------------------------------- zero crossings

// Value and activity of voxel (x, y, z) given in the local frame of leaf
// `slot` (coordinates may leave the leaf by one voxel).
__device__ inline void local_get(const GridView& g, int slot, int x, int y, int z, float& v, bool& on) {
    int dx = (x < 0) ? -1 : (x > 7 ? 1 : 0);
    int dy = (y < 0) ? -1 : (y > 7 ? 1 : 0);
    int dz = (z < 0) ? -1 : (z > 7 ? 1 : 0);
    int s = slot;
    if (dx | dy | dz) s = g.nbr[slot * kNbr + (dx + 1) * 9 + (dy + 1) * 3 + (dz + 1)];
    if (s < 0) {
        v = g.background;
        on = false;
        return;
    }
    int off = voxel_off(x, y, z);
    v = g.values[(size_t)s * kLeafVoxels + off];
    on = mask_bit(g.mask + (size_t)s * 8, off);
}

// find_zero_crossings on bit masks.  A voxel is a crossing if it is active and
// exactly zero, or if its product with an active 6-neighbour is negative: for
// products that do not underflow, if their signs differ.  k_cross_sign streams
// the values once into per-leaf masks of the positive, negative and zero
// active voxels (NaN is none of them, and its product is not negative);
// k_cross_bits then compares 64 voxels at a time against the six shifted
// masks.  A leaf holding a non-zero |v| < 2^-62, whose products may round to
// zero, is flagged, and its candidates and its neighbours' are decided by the
// products themselves.
//
// Bound: the ballots of the pass over the values (half the issue slots; 30 % of
// HBM from a cold cache, 2.2 KB a leaf), then the latency of the neighbours'
// words.  17.5k leaves (L2-resident) take 12 us for the signs and 8 us for the
// bits; one thread per voxel with a table lookup per neighbour took 83 us.
constexpr float kTinyValue = 2.16840434497100887e-19f;  // 2^-62

// One warp per leaf: 16 coalesced rows of 32 values, a ballot each, lane w
// keeping word w.
__global__ void __launch_bounds__(256) k_cross_sign(const uint64_t* __restrict__ mask, const float* __restrict__ values,
                                                   int n, unsigned* __restrict__ pos, unsigned* __restrict__ neg,
                                                   unsigned* __restrict__ zero, unsigned char* __restrict__ tiny) {
    const int lane = threadIdx.x & 31;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
        const float* v = values + (size_t)i * kLeafVoxels;
        const unsigned act = lane < 16 ? reinterpret_cast<const unsigned*>(mask)[(size_t)i * 16 + lane] : 0u;
        float x[16];
#pragma unroll
        for (int w = 0; w < 16; ++w) x[w] = v[w * 32 + lane];
        unsigned p = 0, m = 0, z = 0;
        bool t = false;
#pragma unroll
        for (int w = 0; w < 16; ++w) {
            const unsigned bp = __ballot_sync(0xffffffffu, x[w] > 0.0f), bm = __ballot_sync(0xffffffffu, x[w] < 0.0f),
                           bz = __ballot_sync(0xffffffffu, x[w] == 0.0f);
            const float a = fabsf(x[w]);
            const bool on = (__shfl_sync(0xffffffffu, act, w) >> lane) & 1u;
            t |= on && a > 0.0f && a < kTinyValue;
            if (lane == w) {
                p = bp & act;
                m = bm & act;
                z = bz & act;
            }
        }
        const bool any = __any_sync(0xffffffffu, t);
        if (lane < 16) {
            pos[(size_t)i * 16 + lane] = p;
            neg[(size_t)i * 16 + lane] = m;
            zero[(size_t)i * 16 + lane] = z;
        }
        if (lane == 0) tiny[i] = any;
    }
}

// The voxels of plane word (leaf, x) that have a 6-neighbour in mask m (bit
// y * 8 + z); nb: the leaf's face neighbours -x, +x, -y, +y, -z, +z.
__device__ __forceinline__ uint64_t near6(const uint64_t* __restrict__ m, int leaf, int x, const int* nb) {
    constexpr uint64_t Z0 = 0x0101010101010101ull, Z7 = 0x8080808080808080ull;
    const uint64_t c = m[(size_t)leaf * 8 + x];
    auto word = [&](int s, int w) { return s >= 0 ? m[(size_t)s * 8 + w] : 0ull; };
    const uint64_t xm = x > 0 ? m[(size_t)leaf * 8 + x - 1] : word(nb[0], 7);
    const uint64_t xp = x < 7 ? m[(size_t)leaf * 8 + x + 1] : word(nb[1], 0);
    return xm | xp | (c << 8) | (c >> 8) | (word(nb[2], x) >> 56) | (word(nb[3], x) << 56) | ((c << 1) & ~Z0) |
           ((c >> 1) & ~Z7) | ((word(nb[4], x) & Z7) >> 7) | ((word(nb[5], x) & Z0) << 7);
}

// Where a leaf's rows lie in the list's order.  The pool is sorted by (x, y,
// z) of origin, so the leaves of one origin x are a run [g0, g0 + gn) and
// those of one (x, y) a run [c0, c0 + cn) in it; in global (x, y, z) order the
// run's 8 planes follow one another, in a plane the (x, y) runs, in a run its
// 8 rows y, in a row the leaves: no sort is needed.
struct RowPlace {
    int g0, gn, c0, cn;
};
__device__ __forceinline__ size_t row_of(const RowPlace& r, int leaf, int x, int y) {
    return (size_t)r.g0 * 64 + (size_t)x * 8 * r.gn + (size_t)(r.c0 - r.g0) * 8 + (size_t)y * r.cn + (leaf - r.c0);
}

// Eight lanes per leaf, one plane word each.  xmask: the zero masks on entry,
// the crossing masks on return; *any is set when there is one.  rows (when
// not null): the crossings of each row at its place in the list's order,
// place[leaf] for the pass that writes them.
__global__ void __launch_bounds__(256) k_cross_bits(GridView g, const uint64_t* __restrict__ pos,
                                                   const uint64_t* __restrict__ neg,
                                                   const unsigned char* __restrict__ tiny, uint64_t* __restrict__ xmask,
                                                   int* __restrict__ any, int* __restrict__ rows,
                                                   RowPlace* __restrict__ place) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int leaf = t >> 3, x = t & 7;
    const bool on = leaf < g.n;
    uint64_t cross = 0;
    if (on) {
        const int* row = g.nbr + (size_t)leaf * kNbr;
        const int nb[6] = {row[4], row[22], row[10], row[16], row[12], row[14]};
        const uint64_t p = pos[t], m = neg[t], z = xmask[t];
        cross = z | (p & near6(neg, leaf, x, nb)) | (m & near6(pos, leaf, x, nb));
        bool exact = tiny[leaf];
#pragma unroll
        for (int q = 0; q < 6; ++q) exact |= nb[q] >= 0 && tiny[nb[q]];
        if (exact) {
            for (uint64_t w = cross & ~z; w; w &= w - 1) {
                const int b = __ffsll((long long)w) - 1, y = b >> 3, zz = b & 7;
                const float val = g.values[(size_t)leaf * kLeafVoxels + x * 64 + b];
                bool yes = false;
                for (int q = 0; q < 6; ++q) {
                    const int s = (q & 1) ? 1 : -1;
                    float nv;
                    bool non;
                    local_get(g, leaf, x + (q >> 1 == 0 ? s : 0), y + (q >> 1 == 1 ? s : 0), zz + (q >> 1 == 2 ? s : 0),
                              nv, non);
                    yes |= non && __fmul_rn(val, nv) < 0.0f;
                }
                if (!yes) cross &= ~(1ull << b);
            }
        }
        xmask[t] = cross;
    }
    if (__any_sync(0xffffffffu, cross != 0ull) && (threadIdx.x & 31) == 0) *any = 1;
    if (!rows) return;
    // lane x of a leaf's eight searches one end of its runs: first leaf with
    // the same x, first with a larger x, and the same for (x, y)
    int lo = 0;
    if (on && x < 4) {
        const int4 o = g.origin[leaf];
        int hi = g.n;
        while (lo < hi) {
            const int mid = lo + ((hi - lo) >> 1);
            const int4 c = g.origin[mid];
            const bool less = c.x < o.x || (x >= 2 && c.x == o.x && c.y < o.y);
            const bool same = c.x == o.x && (x < 2 || c.y == o.y);
            if (less || ((x & 1) && same)) lo = mid + 1;
            else hi = mid;
        }
    }
    const int base = threadIdx.x & 24;
    RowPlace r;
    r.g0 = __shfl_sync(0xffffffffu, lo, base);
    r.gn = __shfl_sync(0xffffffffu, lo, base + 1) - r.g0;
    r.c0 = __shfl_sync(0xffffffffu, lo, base + 2);
    r.cn = __shfl_sync(0xffffffffu, lo, base + 3) - r.c0;
    if (!on) return;
    if (x == 0) place[leaf] = r;
#pragma unroll
    for (int y = 0; y < 8; ++y) rows[row_of(r, leaf, x, y)] = __popc((unsigned)(cross >> (8 * y)) & 0xffu);
}

// The crossings of each row (64 threads per leaf, one row each) at its scanned position.
__global__ void __launch_bounds__(256) k_emit_crossings(GridView g, const uint64_t* __restrict__ xmask,
                                                       const int* __restrict__ rows,
                                                       const RowPlace* __restrict__ place, int* __restrict__ coords) {
    const int leaf = (blockIdx.x * blockDim.x + threadIdx.x) >> 6, r = threadIdx.x & 63;
    if (leaf >= g.n) return;
    unsigned b = reinterpret_cast<const unsigned char*>(xmask)[(size_t)leaf * 64 + r];
    if (!b) return;
    const int x = r >> 3, y = r & 7;
    const int4 o = g.origin[leaf];
    size_t j = 3 * (size_t)rows[row_of(place[leaf], leaf, x, y)];
    for (; b; b &= b - 1, j += 3) {
        coords[j] = o.x + x;
        coords[j + 1] = o.y + y;
        coords[j + 2] = o.z + __ffs(b) - 1;
    }
}

// --------------------------------------------------------------- rebuild

// Nearest crossing by squared index distance inside a cube window of half
// size R <= 8, using the crossing masks of the 27 neighbouring leaves staged
// in shared memory.  A z-row of 8 voxels is one byte of a mask, so each
// (dx, dy) pair of the window is one 24-bit row test.
__global__ void __launch_bounds__(256) k_rebuild_window(GridView g, float* __restrict__ values,
                                                       uint64_t* __restrict__ mask, const uint64_t* __restrict__ xmask,
                                                       int R, float vs, float band, int* __restrict__ nonempty) {
    __shared__ uint64_t s_x[kNbr * 8];
    int slot = blockIdx.x;
    if (slot >= g.n) return;
    for (int t = threadIdx.x; t < kNbr * 8; t += blockDim.x) {
        int d = t >> 3;
        int s = g.nbr[slot * kNbr + d];
        s_x[t] = (s < 0) ? 0ull : xmask[(size_t)s * 8 + (t & 7)];
    }
    __syncthreads();
    const unsigned char* sb = (const unsigned char*)s_x;  // leaf d occupies bytes [64d, 64d+64)
    uint64_t* m = mask + (size_t)slot * 8;
    bool keep_any = false;
    for (int r = 0; r < 2; ++r) {
        int off = threadIdx.x + 256 * r;
        bool on = mask_bit(m, off);
        bool keep = false;
        if (on) {
            int x = off >> 6, y = (off >> 3) & 7, z = off & 7;
            int best = INT_MAX;
            for (int dx = -R; dx <= R; ++dx) {
                int xx = x + dx;
                int lxo = (xx < 0) ? 0 : (xx > 7 ? 2 : 1);
                int xl = xx & 7;
                for (int dy = -R; dy <= R; ++dy) {
                    int dxy = dx * dx + dy * dy;
                    if (dxy >= best) continue;
                    int yy = y + dy;
                    int lyo = (yy < 0) ? 0 : (yy > 7 ? 2 : 1);
                    int yl = yy & 7;
                    int dbase = lxo * 9 + lyo * 3;
                    int byte_idx = xl * 8 + yl;
                    unsigned row = (unsigned)sb[(dbase + 0) * 64 + byte_idx] |
                                   ((unsigned)sb[(dbase + 1) * 64 + byte_idx] << 8) |
                                   ((unsigned)sb[(dbase + 2) * 64 + byte_idx] << 16);
                    int c = z + 8;
                    unsigned lo_mask = (2u << c) - 1u;                      // bits <= c
                    unsigned win = ((c + R + 1 >= 32) ? 0xffffffffu : ((1u << (c + R + 1)) - 1u)) &
                                   ~((c - R <= 0) ? 0u : ((1u << (c - R)) - 1u));
                    unsigned wr = row & win;
                    if (!wr) continue;
                    int dz = 32;
                    unsigned lo = wr & lo_mask;
                    if (lo) dz = c - (31 - __clz(lo));
                    unsigned hi = wr >> c;
                    if (hi) dz = min(dz, __ffs(hi) - 1);
                    int d2 = dxy + dz * dz;
                    if (d2 < best) best = d2;
                }
            }
            if (best != INT_MAX) {
                float old = values[(size_t)slot * kLeafVoxels + off];
                float sign = (old >= 0.0f) ? 1.0f : -1.0f;
                float md = __fsqrt_rn((float)best);
                float nv = __fmul_rn(__fmul_rn(sign, md), vs);
                if (fabsf(nv) < band) {
                    keep = true;
                    values[(size_t)slot * kLeafVoxels + off] = nv;
                }
            }
            if (!keep) values[(size_t)slot * kLeafVoxels + off] = g.background;
        }
        unsigned b = __ballot_sync(0xffffffffu, keep);
        if ((threadIdx.x & 31) == 0) ((unsigned*)m)[off >> 5] = b;
        keep_any |= keep;
    }
    int a = __syncthreads_or(keep_any);
    if (threadIdx.x == 0) nonempty[slot] = a;
}

// The same for windows of half size R <= 2 (half widths to 3), whole z-rows at
// a time: 64 threads per leaf, one row of 8 voxels each.  The 24-bit crossing
// row of every (dx, dy) in the window, shifted by |dz| = 0, 1, 2 both ways,
// joins the set of voxels with a crossing at squared distance dx^2 + dy^2 +
// dz^2 (at most 10 different), so 8 voxels cost one pass over (2R + 1)^2 words
// and a voxel's minimum is the smallest set that holds it.
//
// Bound: instruction issue (60 % of the slots) and the staging's barrier.  17.5k
// leaves, R = 2 (L2-resident, 4.2 KB a leaf): 34 us, against 179 us one voxel
// and 25 row tests at a time.
template <int R>
__global__ void __launch_bounds__(256) k_rebuild_rows(GridView g, float* __restrict__ values,
                                                     unsigned char* __restrict__ mask,
                                                     const unsigned char* __restrict__ xmask, float vs, float band,
                                                     int* __restrict__ nonempty) {
    constexpr int E = 8 + 2 * R, D = 3 * R * R;
    __shared__ unsigned s_row[4][E * E];
    __shared__ int s_any[4];
    const int q = threadIdx.x >> 6, r = threadIdx.x & 63;
    const int slot = blockIdx.x * 4 + q;
    const bool leaf = slot < g.n;
    if (r == 0) s_any[q] = 0;
    if (leaf) {
        for (int i = r; i < E * E; i += 64) {
            const int X = i / E - R, Y = i % E - R;
            const int* nb = g.nbr + (size_t)slot * kNbr + ((X + 8) >> 3) * 9 + ((Y + 8) >> 3) * 3;
            const int at = (X & 7) * 8 + (Y & 7);
            unsigned w = 0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int s = nb[d];
                if (s >= 0) w |= (unsigned)xmask[(size_t)s * 64 + at] << (8 * d);
            }
            s_row[q][i] = w;
        }
    }
    __syncthreads();
    if (leaf) {
        const unsigned on = mask[(size_t)slot * 64 + r];
        unsigned keep = 0;
        if (on) {
            unsigned at[D + 1] = {};  // at[d2]: voxels with a crossing at squared distance d2
            const unsigned* row = s_row[q] + (r >> 3) * E + (r & 7);
#pragma unroll
            for (int dx = 0; dx <= 2 * R; ++dx)
#pragma unroll
                for (int dy = 0; dy <= 2 * R; ++dy) {
                    const unsigned w = row[dx * E + dy];
                    const int s = (dx - R) * (dx - R) + (dy - R) * (dy - R);
#pragma unroll
                    for (int dz = 0; dz <= R; ++dz) at[s + dz * dz] |= (w >> (8 - dz)) | (w >> (8 + dz));
                }
            float* v = values + (size_t)slot * kLeafVoxels + r * 8;
            float4 v4[2] = {reinterpret_cast<float4*>(v)[0], reinterpret_cast<float4*>(v)[1]};
            float* x = reinterpret_cast<float*>(v4);
#pragma unroll
            for (int z = 0; z < 8; ++z) {
                int best = -1;
#pragma unroll
                for (int d = D; d >= 0; --d)
                    if ((at[d] >> z) & 1u) best = d;
                if (!((on >> z) & 1u)) continue;
                const float sign = (x[z] >= 0.0f) ? 1.0f : -1.0f;
                const float nv = __fmul_rn(__fmul_rn(sign, __fsqrt_rn((float)best)), vs);
                const bool k = best >= 0 && fabsf(nv) < band;
                x[z] = k ? nv : g.background;
                keep |= (k ? 1u : 0u) << z;
            }
            reinterpret_cast<float4*>(v)[0] = v4[0];
            reinterpret_cast<float4*>(v)[1] = v4[1];
        }
        mask[(size_t)slot * 64 + r] = (unsigned char)keep;
        if (keep) s_any[q] = 1;
    }
    __syncthreads();
    if (leaf && r == 0) nonempty[slot] = s_any[q];
}

// Literal form of the reference loop for any half-width: f32 distances to
// every crossing, folded with min.
__global__ void __launch_bounds__(256) k_rebuild_brute(GridView g, float* __restrict__ values,
                                                      uint64_t* __restrict__ mask, const int* __restrict__ cross,
                                                      int n_cross, float vs, float band, int* __restrict__ nonempty) {
    int slot = blockIdx.x;
    if (slot >= g.n) return;
    int4 o = g.origin[slot];
    uint64_t* m = mask + (size_t)slot * 8;
    bool keep_any = false;
    for (int r = 0; r < 2; ++r) {
        int off = threadIdx.x + 256 * r;
        bool keep = false;
        if (mask_bit(m, off)) {
            int x = o.x + (off >> 6), y = o.y + ((off >> 3) & 7), z = o.z + (off & 7);
            float md = 3.402823466e+38f;
            for (int c = 0; c < n_cross; ++c) {
                float dx = __int2float_rn((int)((unsigned)x - (unsigned)cross[3 * c]));
                float dy = __int2float_rn((int)((unsigned)y - (unsigned)cross[3 * c + 1]));
                float dz = __int2float_rn((int)((unsigned)z - (unsigned)cross[3 * c + 2]));
                float d = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
                md = fminf(md, d);
            }
            float old = values[(size_t)slot * kLeafVoxels + off];
            float sign = (old >= 0.0f) ? 1.0f : -1.0f;
            float nv = __fmul_rn(__fmul_rn(sign, md), vs);
            if (fabsf(nv) < band) {
                keep = true;
                values[(size_t)slot * kLeafVoxels + off] = nv;
            } else {
                values[(size_t)slot * kLeafVoxels + off] = g.background;
            }
        }
        unsigned b = __ballot_sync(0xffffffffu, keep);
        if ((threadIdx.x & 31) == 0) ((unsigned*)m)[off >> 5] = b;
        keep_any |= keep;
    }
    int a = __syncthreads_or(keep_any);
    if (threadIdx.x == 0) nonempty[slot] = a;
}

// ------------------------------------------------------------------ trim

__global__ void __launch_bounds__(256) k_trim(GridView g, float* __restrict__ values, uint64_t* __restrict__ mask,
                                             float thr, int* __restrict__ nonempty) {
    int slot = blockIdx.x;
    if (slot >= g.n) return;
    uint64_t* m = mask + (size_t)slot * 8;
    bool keep_any = false;
    for (int r = 0; r < 2; ++r) {
        int off = threadIdx.x + 256 * r;
        bool keep = false;
        if (mask_bit(m, off)) {
            float v = values[(size_t)slot * kLeafVoxels + off];
            if (fabsf(v) >= thr) values[(size_t)slot * kLeafVoxels + off] = g.background;
            else keep = true;
        }
        unsigned b = __ballot_sync(0xffffffffu, keep);
        if ((threadIdx.x & 31) == 0) ((unsigned*)m)[off >> 5] = b;
        keep_any |= keep;
    }
    int a = __syncthreads_or(keep_any);
    if (threadIdx.x == 0) nonempty[slot] = a;
}

// ---------------------------------------------------------------- sphere

// One CTA per candidate leaf of the sphere's index bounding box, leaves
// enumerated x-major (lexicographic origin order).
__global__ void __launch_bounds__(512) k_sphere(int lx0, int ly0, int lz0, int nly, int nlz, int n_cand, int imin,
                                               int jmin, int kmin, int imax, int jmax, int kmax, double radius,
                                               double c0, double c1, double c2, double vs, float bg,
                                               int4* __restrict__ origin, uint64_t* __restrict__ mask,
                                               float* __restrict__ values, int* __restrict__ nonempty) {
    int cand = blockIdx.x;
    if (cand >= n_cand) return;
    int lx = lx0 + cand / (nly * nlz);
    int ly = ly0 + (cand / nlz) % nly;
    int lz = lz0 + cand % nlz;
    int off = threadIdx.x;
    int i = lx * 8 + (off >> 6), j = ly * 8 + ((off >> 3) & 7), k = lz * 8 + (off & 7);
    bool on = false;
    float val = bg;
    if (i >= imin && i <= imax && j >= jmin && j <= jmax && k >= kmin && k <= kmax) {
        double wx = __dsub_rn(__dmul_rn((double)i, vs), c0);
        double wy = __dsub_rn(__dmul_rn((double)j, vs), c1);
        double wz = __dsub_rn(__dmul_rn((double)k, vs), c2);
        double dist = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(wx, wx), __dmul_rn(wy, wy)), __dmul_rn(wz, wz)));
        float sdf = __double2float_rn(__dsub_rn(dist, radius));
        if (fabsf(sdf) < bg) {
            on = true;
            val = sdf;
        }
    }
    values[(size_t)cand * kLeafVoxels + off] = val;
    unsigned b = __ballot_sync(0xffffffffu, on);
    if ((off & 31) == 0) ((unsigned*)(mask + (size_t)cand * 8))[off >> 5] = b;
    int a = __syncthreads_or(on);
    if (off == 0) {
        origin[cand] = make_int4(lx * 8, ly * 8, lz * 8, 0);
        nonempty[cand] = a;
    }
}

// ================================================================ host side

GridView make_view(const vlr_grid* g) {
    GridView v;
    v.origin = g->origin;
    v.mask = g->mask;
    v.values = (const float*)g->values;
    v.nbr = g->nbr;
    v.hash.key = g->hkey;
    v.hash.val = g->hval;
    v.hash.cap = g->hcap;
    for (int a = 0; a < 3; ++a) v.hash.base[a] = g->base[a];
    v.n = g->n;
    v.background = g->background;
    v.inv_vs = 1.0 / g->xf.voxel_size;
    for (int a = 0; a < 3; ++a) v.t_origin[a] = g->xf.origin[a];
    for (int q = 0; q < 12; ++q) v.mat[q] = g->xf.affine[q];
    return v;
}

int advect_ref(vlr_ctx* ctx, const vlr_grid* g, const vlr_grid* vx, const vlr_grid* vy, const vlr_grid* vz, double dt,
               vlr_grid* out) {
    out->ctx = ctx;
    out->kind = VLR_KIND_F32_WORLD;
    out->background = g->background;
    // Grid::with_affine keeps the affine and resets the legacy transform to
    // uniform(affine.voxel_size) (src/grid.rs:378-388).
    out->xf = g->xf;
    out->xf.voxel_size = g->xf.affine_voxel_size;
    out->xf.origin[0] = out->xf.origin[1] = out->xf.origin[2] = 0.0;
    for (int a = 0; a < 3; ++a) out->base[a] = g->base[a];
    std::memcpy(out->box, g->box, sizeof(g->box));
    int rc = grid_alloc(ctx, out, std::max(g->n, 1));
    if (rc) return rc;
    out->n = g->n;
    if (g->n == 0) return grid_index(ctx, out);
    int* nonempty = nullptr;
    VLR_CUDA(ctx, cudaMallocFromPoolAsync(&nonempty, sizeof(int) * g->n, ctx->pool, ctx->stream));
    VLR_CUDA(ctx, cudaMemcpyAsync(out->origin, g->origin, sizeof(int4) * g->n, cudaMemcpyDeviceToDevice, ctx->stream));
    const GridView v[3] = {make_view(vx), make_view(vy), make_view(vz)};
    bool same = true;
    for (int q = 1; q < 3; ++q) {
        same = same && v[q].inv_vs == v[0].inv_vs;
        for (int a = 0; a < 3; ++a) same = same && v[q].t_origin[a] == v[0].t_origin[a];
    }
    auto* kernel = same ? k_advect_ref<true> : k_advect_ref<false>;
    VLR_TIMED(ctx, "k_advect_ref",
              kernel<<<(g->n + kAdvWarps - 1) / kAdvWarps, 32 * kAdvWarps, 0, ctx->stream>>>(
                  make_view(g), v[0], v[1], v[2], dt, (float*)out->values, out->mask, nonempty));
    VLR_CUDA(ctx, cudaGetLastError());
    // the output has the input's leaves (less those without active voxels), so
    // an output that keeps them all takes the input's index as it is
    rc = grid_compact(ctx, out, nonempty, "advect_level_set", g);
    cudaFreeAsync(nonempty, ctx->stream);
    return rc;
}

int sample_points(vlr_ctx* ctx, const vlr_grid* g, const double* h_pts, size_t n, float* h_out) {
    if (n == 0) return VLR_OK;
    double* d_pts = nullptr;
    VLR_CUDA(ctx, cudaMallocFromPoolAsync(&d_pts, (sizeof(double) * 3 + sizeof(float)) * n, ctx->pool, ctx->stream));
    float* d_out = reinterpret_cast<float*>(d_pts + 3 * n);
    int rc = h2d_copy(ctx, d_pts, h_pts, sizeof(double) * 3 * n);
    if (!rc) {
        k_sample_points<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(make_view(g), d_pts, (int)n, d_out);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = check_cuda(ctx, e, "k_sample_points");
    }
    if (!rc) rc = d2h_copy(ctx, h_out, d_out, sizeof(float) * n);
    cudaFreeAsync(d_pts, ctx->stream);
    return rc;
}

// Device buffers of a crossing search over n leaves, in one block.
struct CrossBufs {
    char* block = nullptr;
    uint64_t* xmask = nullptr;  // crossing masks
    uint64_t* pos = nullptr;
    uint64_t* neg = nullptr;
    unsigned char* tiny = nullptr;
    int* any = nullptr;         // 1 when there is a crossing
    int* total = nullptr;       // their number (with rows)
    int* flags = nullptr;       // one int per leaf, for the caller
    int* rows = nullptr;        // 64 n ints
    RowPlace* place = nullptr;
};

static int alloc_cross(vlr_ctx* ctx, int n, bool rows, CrossBufs& b) {
    const size_t m = (size_t)n;
    auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
    const size_t need = up(192 * m) + up(m) + 256 + up(4 * m) + (rows ? up(sizeof(RowPlace) * m) + up(256 * m) : 0);
    VLR_CUDA(ctx, cudaMallocFromPoolAsync((void**)&b.block, need, ctx->pool, ctx->stream));
    char* p = b.block;
    auto take = [&](size_t v) {
        char* r = p;
        p += up(v);
        return r;
    };
    b.xmask = (uint64_t*)take(192 * m);
    b.pos = b.xmask + 8 * m;
    b.neg = b.pos + 8 * m;
    b.tiny = (unsigned char*)take(m);
    b.any = (int*)take(8);
    b.total = b.any + 1;
    b.flags = (int*)take(4 * m);
    if (rows) {
        b.place = (RowPlace*)take(sizeof(RowPlace) * m);
        b.rows = (int*)take(256 * m);
    }
    return VLR_OK;
}

// Crossing masks (and row counts, scanned into positions) on the device, enqueued.
static int crossings(vlr_ctx* ctx, const vlr_grid* g, CrossBufs& b) {
    cudaStream_t st = ctx->stream;
    VLR_CUDA(ctx, cudaMemsetAsync(b.any, 0, 2 * sizeof(int), st));
    const int n = g->n;
    VLR_TIMED(ctx, "k_cross_sign",
              k_cross_sign<<<std::min((n + 7) / 8, ctx->sm_count * 8), 256, 0, st>>>(
                  g->mask, (const float*)g->values, n, (unsigned*)b.pos, (unsigned*)b.neg, (unsigned*)b.xmask, b.tiny));
    VLR_TIMED(ctx, "k_crossings", k_cross_bits<<<(n + 31) / 32, 256, 0, st>>>(make_view(g), b.pos, b.neg, b.tiny,
                                                                             b.xmask, b.any, b.rows, b.place));
    VLR_CUDA(ctx, cudaGetLastError());
    return b.rows ? scan_exclusive(ctx, b.rows, b.rows, 64ll * n, b.total) : VLR_OK;
}

static void emit_crossings(vlr_ctx* ctx, const vlr_grid* g, const CrossBufs& b, int* d_coords) {
    k_emit_crossings<<<(g->n + 3) / 4, 256, 0, ctx->stream>>>(make_view(g), b.xmask, b.rows, b.place, d_coords);
}

int find_zero_crossings(vlr_ctx* ctx, const vlr_grid* g, int32_t* h_coords, size_t cap, size_t* count) {
    *count = 0;
    if (g->n == 0) return VLR_OK;
    CrossBufs b;
    int* d_coords = nullptr;
    auto run = [&]() -> int {
        int rc = alloc_cross(ctx, g->n, true, b);
        if (!rc) rc = crossings(ctx, g, b);
        int total = 0;
        if (!rc) rc = read_int(ctx, b.total, &total);
        if (rc) return rc;
        *count = (size_t)total;
        if (total == 0 || !h_coords || cap == 0) return VLR_OK;
        VLR_CUDA(ctx, cudaMallocFromPoolAsync(&d_coords, sizeof(int) * 3 * (size_t)total, ctx->pool, ctx->stream));
        emit_crossings(ctx, g, b, d_coords);
        VLR_CUDA(ctx, cudaGetLastError());
        return d2h_copy(ctx, h_coords, d_coords, sizeof(int) * 3 * std::min<size_t>(cap, (size_t)total));
    };
    const int rc = run();
    if (d_coords) cudaFreeAsync(d_coords, ctx->stream);
    if (b.block) cudaFreeAsync(b.block, ctx->stream);
    return rc;
}

int trim_narrow_band(vlr_ctx* ctx, vlr_grid* g, float half_width) {
    if (g->n == 0) return VLR_OK;
    float vs = (float)g->xf.voxel_size;
    float thr = half_width * vs;
    int* flags = nullptr;
    VLR_CUDA(ctx, cudaMallocFromPoolAsync(&flags, sizeof(int) * g->n, ctx->pool, ctx->stream));
    GridView v = make_view(g);
    VLR_TIMED(ctx, "k_trim", k_trim<<<g->n, 256, 0, ctx->stream>>>(v, (float*)g->values, g->mask, thr, flags));
    VLR_CUDA(ctx, cudaGetLastError());
    const int rc = grid_compact(ctx, g, flags, "trim_narrow_band");
    cudaFreeAsync(flags, ctx->stream);
    return rc;
}

int rebuild_narrow_band(vlr_ctx* ctx, vlr_grid* g, float half_width) {
    if (g->n == 0) return VLR_OK;
    float vs = (float)g->xf.voxel_size;
    float band = half_width * vs;
    const bool window = std::isfinite(half_width) && vs > 0.0f && half_width <= 9.0f;
    CrossBufs b;
    int* d_coords = nullptr;
    auto run = [&]() -> int {
        int rc = alloc_cross(ctx, g->n, !window, b);
        if (!rc) rc = crossings(ctx, g, b);
        int total = 0;
        if (!rc) rc = read_int(ctx, window ? b.any : b.total, &total);
        if (rc) return rc;
        if (total == 0) return VLR_OK;  // no crossings: the grid is returned unchanged (level_set_track.rs:85-87)
        GridView v = make_view(g);
        if (window) {
            int R = std::max(0, (int)std::ceil(half_width) - 1);
            // whole rows while the sets of distances fit in registers (R <= 2)
            if (R <= 2) {
                auto* rows = R == 2 ? k_rebuild_rows<2> : (R == 1 ? k_rebuild_rows<1> : k_rebuild_rows<0>);
                VLR_TIMED(ctx, "k_rebuild_window",
                          rows<<<(g->n + 3) / 4, 256, 0, ctx->stream>>>(v, (float*)g->values, (unsigned char*)g->mask,
                                                                       (const unsigned char*)b.xmask, vs, band,
                                                                       b.flags));
            } else {
                VLR_TIMED(ctx, "k_rebuild_window",
                          k_rebuild_window<<<g->n, 256, 0, ctx->stream>>>(v, (float*)g->values, g->mask, b.xmask, R,
                                                                         vs, band, b.flags));
            }
        } else {
            VLR_CUDA(ctx, cudaMallocFromPoolAsync(&d_coords, sizeof(int) * 3 * (size_t)total, ctx->pool, ctx->stream));
            emit_crossings(ctx, g, b, d_coords);
            k_rebuild_brute<<<g->n, 256, 0, ctx->stream>>>(v, (float*)g->values, g->mask, d_coords, total, vs, band,
                                                          b.flags);
        }
        VLR_CUDA(ctx, cudaGetLastError());
        return grid_compact(ctx, g, b.flags, "rebuild_narrow_band");
    };
    const int rc = run();
    if (d_coords) cudaFreeAsync(d_coords, ctx->stream);
    if (b.block) cudaFreeAsync(b.block, ctx->stream);
    return rc;
}

static int32_t sat_i32(double v) {
    if (std::isnan(v)) return 0;
    if (v <= -2147483648.0) return INT32_MIN;
    if (v >= 2147483647.0) return INT32_MAX;
    return (int32_t)v;
}

int make_sphere(vlr_ctx* ctx, double radius, const double c[3], double vs, double hw, vlr_grid* out) {
    double band = hw * vs;
    float bg = (float)band;
    double extent = radius + band;
    double inv = 1.0 / vs;
    int32_t imin = sat_i32(std::floor((c[0] - extent) * inv));
    int32_t jmin = sat_i32(std::floor((c[1] - extent) * inv));
    int32_t kmin = sat_i32(std::floor((c[2] - extent) * inv));
    int32_t imax = sat_i32(std::ceil((c[0] + extent) * inv));
    int32_t jmax = sat_i32(std::ceil((c[1] + extent) * inv));
    int32_t kmax = sat_i32(std::ceil((c[2] + extent) * inv));
    out->ctx = ctx;
    out->kind = VLR_KIND_F32_WORLD;
    out->background = bg;
    // set_transform(VoxelTransform::uniform(vs)) (src/tools/sphere.rs:36-38)
    std::memset(&out->xf, 0, sizeof(out->xf));
    out->xf.voxel_size = vs;
    out->xf.affine[0] = out->xf.affine[5] = out->xf.affine[10] = vs;
    out->xf.affine_voxel_size = vs;
    if (imin > imax || jmin > jmax || kmin > kmax) {
        out->base[0] = out->base[1] = out->base[2] = -kKeyHalf;
        int rc = grid_alloc(ctx, out, 1);
        if (rc) return rc;
        out->n = 0;
        return grid_index(ctx, out);
    }
    long long lx0 = imin >> 3, ly0 = jmin >> 3, lz0 = kmin >> 3;
    long long nlx = (imax >> 3) - lx0 + 1, nly = (jmax >> 3) - ly0 + 1, nlz = (kmax >> 3) - lz0 + 1;
    long long n_cand = nlx * nly * nlz;
    if (n_cand > (1ll << 26)) return set_error(ctx, VLR_ERR_CAPACITY, "sphere bounding box too large");
    int32_t corner[6] = {imin, jmin, kmin, imax, jmax, kmax};
    int32_t bb[6] = {corner[0], corner[1], corner[2], corner[3], corner[4], corner[5]};
    int rc = choose_base(ctx, bb, 2, out->base, out->box);
    if (rc) return rc;
    rc = grid_alloc(ctx, out, (int)n_cand);
    if (rc) return rc;
    out->n = (int)n_cand;
    int* flags = nullptr;
    VLR_CUDA(ctx, cudaMallocFromPoolAsync(&flags, sizeof(int) * n_cand, ctx->pool, ctx->stream));
    k_sphere<<<(unsigned)n_cand, 512, 0, ctx->stream>>>((int)lx0, (int)ly0, (int)lz0, (int)nly, (int)nlz, (int)n_cand,
                                                        imin, jmin, kmin, imax, jmax, kmax, radius, c[0], c[1], c[2],
                                                        vs, bg, out->origin, out->mask, (float*)out->values, flags);
    VLR_CUDA(ctx, cudaGetLastError());
    // indexed after the compaction: most candidates of the box are dropped
    rc = grid_compact(ctx, out, flags, "make_level_set_sphere");
    cudaFreeAsync(flags, ctx->stream);
    if (!rc && out->n == (int)n_cand) rc = grid_index(ctx, out);
    return rc;
}

}  // namespace vlr
