// volume_to_mesh (src/tools/volume_to_mesh.rs:46-201): marching-cubes
// isosurface of a world-unit f32 grid, with the reference's cell order, vertex
// numbering and vertex positions.
//
// The reference visits the 8^3 cell tiles of every leaf and of its 6 face
// neighbours, tiles in ascending (x, y, z) of origin and cells x-major within a
// tile (volume_to_mesh.rs:58-97); a cell reads its 8 corners with Grid::get,
// flags the edges whose corners classify differently against the isovalue,
// and creates an edge's vertex the first time a processed cell flags it (a
// HashMap edge cache, volume_to_mesh.rs:144-186), so vertex i is the i-th
// first-touched edge in that order, interpolated from the creating cell's
// first endpoint toward its second.  Triangles follow per cell in visit order.
//
// On the GPU:
//   tile list      the tiles as one bit each of the leaves' bounding box (the
//                  box grown by a tile), x-major, so that bit order is visit
//                  order and a tile's rank is a prefix count: k_mc_mark sets
//                  the bits of every leaf and its face neighbours,
//                  k_mc_count + scan rank them, k_mc_list writes the list.
//                  A box much emptier than that (tile_list) sorts the seven
//                  candidates per leaf as 63-bit keys instead (k_mc_cand,
//                  radix sort, k_mc_unique) and ranks through a hash.
//   k_mc_classify  one CTA per tile: the signs of its 9^3 corners as 81 rows of
//                  9 bits, the cells whose corners differ by row operations
//                  on them, and for those (compacted, about one in five of a
//                  tile on the surface) the case and which of its flagged
//                  edges the cell creates: an edge belongs to up to 4 cells,
//                  and the cell creates it iff none of the other processed
//                  cells precedes it in visit order (decided from the 27
//                  neighbour tiles' ranks); per-cell word = case | creator
//                  mask | in-tile rank of its first created vertex; per-tile
//                  counts and mask of such cells
//   (scans)        tile bases of vertices and triangles
//   k_mc_emit      one CTA per tile with triangles, its listed cells: creators
//                  write their vertex (f64, the reference's rounding: f32 t,
//                  then pa + t * (pb - pa)); the other flagged edges look up
//                  their creator's index; each cell writes its triangles at
//                  its scanned offset
// Sphere of radius 96 (6,822 tiles, 337k vertices, 673k triangles): classify
// 43 us and emit 46 us (one thread per cell of a 512-thread CTA, every tile
// staged: 133 and 139), the tile list 28 us in 5 launches (the sort: 106 us in
// 22).  Bound: instruction issue (61 % of the slots), the barriers of a tile
// (classify) and the loads of its slots and creators' words (emit); the mesh's
// copy to the host is ten times either.
// So the output order needs no sort and no atomics: every index is a prefix
// count in visit order.
//
// Triangle table.  Vertices depend only on the edge table, which is the
// classification rule.  Triangles come from the crate's own 256-case table
// (src/tools/volume_to_mesh.rs:246-503, the classic Lorensen & Cline / Bourke
// table), carried in mc_tri_table.inc with the same corner and edge
// numbering, so each cell emits the same triangles in the same order as the
// crate; a cell's triangles are the table row's triples up to its -1.
#include <algorithm>
#include <cstring>
#include <mutex>

#include "box_reduce.cuh"
#include "ref_ops.hpp"
#include "sort_reduce.hpp"

namespace vlr {
namespace {

constexpr int kCornerOff[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0}, {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
constexpr int kEdgeEnds[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                  {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};
// the crate's triangle table (src/tools/volume_to_mesh.rs:246-503), 16 entries per case, -1 terminated
constexpr int8_t kTriTable[256][16] = {
#include "mc_tri_table.inc"
};

struct McTable {
    int8_t tri[256][16];
    uint8_t ntri[256];
    // the 3 other cells holding edge e: (dx+1) | (dy+1) << 2 | (dz+1) << 4 | e' << 8,
    // e' the edge's index in that cell
    int nb[12][3];
};

McTable build_mc_table() {
    McTable t;
    for (int cs = 0; cs < 256; ++cs) {
        int n = 0;
        while (n < 15 && kTriTable[cs][n] >= 0) n += 3;
        std::memcpy(t.tri[cs], kTriTable[cs], 16);
        t.ntri[cs] = (uint8_t)(n / 3);
    }
    // an edge along axis a with lower corner L lies in the 4 cells at
    // delta = (L_u - du) e_u + (L_w - dw) e_w, du, dw in {0, 1}; in the cell
    // at delta its lower corner is L - delta
    for (int e = 0; e < 12; ++e) {
        const int a = kEdgeEnds[e][0], b = kEdgeEnds[e][1];
        int L[3], axis = 0;
        for (int k = 0; k < 3; ++k) {
            L[k] = std::min(kCornerOff[a][k], kCornerOff[b][k]);
            if (kCornerOff[a][k] != kCornerOff[b][k]) axis = k;
        }
        const int u = (axis + 1) % 3, w = (axis + 2) % 3;
        int q = 0;
        for (int du = 0; du < 2; ++du)
            for (int dw = 0; dw < 2; ++dw) {
                int d[3] = {0, 0, 0};
                d[u] = L[u] - du;
                d[w] = L[w] - dw;
                if (d[u] == 0 && d[w] == 0) continue;
                int M[3];
                for (int k = 0; k < 3; ++k) M[k] = L[k] - d[k];
                int e2 = -1;
                for (int f = 0; f < 12 && e2 < 0; ++f) {
                    int N[3], ax2 = 0;
                    for (int k = 0; k < 3; ++k) {
                        N[k] = std::min(kCornerOff[kEdgeEnds[f][0]][k], kCornerOff[kEdgeEnds[f][1]][k]);
                        if (kCornerOff[kEdgeEnds[f][0]][k] != kCornerOff[kEdgeEnds[f][1]][k]) ax2 = k;
                    }
                    if (ax2 == axis && N[0] == M[0] && N[1] == M[1] && N[2] == M[2]) e2 = f;
                }
                t.nb[e][q++] = (d[0] + 1) | ((d[1] + 1) << 2) | ((d[2] + 1) << 4) | (e2 << 8);
            }
    }
    return t;
}

const McTable& mc_table() {
    static const McTable t = build_mc_table();
    return t;
}

// read by case, which differs from lane to lane: global memory, not constant
__device__ __align__(16) int8_t d_mc_tri[256][16];
__device__ uint8_t d_mc_ntri[256];
__constant__ int c_mc_nb[12][3];
// corner offsets and edge endpoints for device code (same as kCornerOff, kEdgeEnds)
__constant__ int c_corner[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0},
                                   {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
__constant__ int c_edge[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                  {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};

std::mutex g_mc_mu;
bool g_mc_ready[128] = {};

// Copies the triangle table into this device's constant memory (once per
// device, with that device current).
int ensure_tables(vlr_ctx* ctx) {
    const int dev = ctx->device;
    if (dev < 0 || dev >= 128) return set_error(ctx, VLR_ERR_INVALID, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_mc_mu);
    if (!g_mc_ready[dev]) {
        const McTable& t = mc_table();
        DeviceGuard guard(dev);
        VLR_CUDA(ctx, guard.status);
        VLR_CUDA(ctx, cudaMemcpyToSymbol(d_mc_tri, t.tri, sizeof(t.tri)));
        VLR_CUDA(ctx, cudaMemcpyToSymbol(d_mc_ntri, t.ntri, sizeof(t.ntri)));
        VLR_CUDA(ctx, cudaMemcpyToSymbol(c_mc_nb, t.nb, sizeof(t.nb)));
        g_mc_ready[dev] = true;
    }
    return VLR_OK;
}

constexpr long long kAxisLim = 1ll << kKeyBits;
constexpr uint64_t kBadKey = ~0ull;

// x-major key of a tile (leaf coordinates relative to the grid's hash base):
// ascending keys are ascending (x, y, z), the reference's Coord order.
__host__ __device__ inline uint64_t tile_key(long long lx, long long ly, long long lz, const long long* base) {
    const long long rx = lx - base[0], ry = ly - base[1], rz = lz - base[2];
    if (rx < 0 || ry < 0 || rz < 0 || rx >= kAxisLim || ry >= kAxisLim || rz >= kAxisLim) return kBadKey;
    return ((uint64_t)rx << 42) | ((uint64_t)ry << 21) | (uint64_t)rz;
}

struct TileBase {
    long long b[3];
};

__global__ void k_mc_cand(const int4* __restrict__ origin, int n, TileBase tb, uint64_t* __restrict__ keys,
                          unsigned* __restrict__ idx, unsigned* __restrict__ err) {
    const int d[7][3] = {{0, 0, 0}, {-1, 0, 0}, {1, 0, 0}, {0, -1, 0}, {0, 1, 0}, {0, 0, -1}, {0, 0, 1}};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < 7ll * n;
         i += (long long)gridDim.x * blockDim.x) {
        const int s = (int)(i / 7), j = (int)(i % 7);
        const int4 o = origin[s];
        uint64_t k = tile_key((long long)(o.x >> 3) + d[j][0], (long long)(o.y >> 3) + d[j][1],
                              (long long)(o.z >> 3) + d[j][2], tb.b);
        if (k == kBadKey) atomicOr(err, kErrExtent);
        keys[i] = k;
        idx[i] = (unsigned)i;
    }
}

__global__ void k_mc_unique(const uint64_t* __restrict__ sorted, int n, int* __restrict__ flag) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint64_t k = sorted[i];
        flag[i] = (k != kBadKey && (i == 0 || k != sorted[i - 1])) ? 1 : 0;
    }
}

__global__ void k_mc_compact(const uint64_t* __restrict__ sorted, const int* __restrict__ flag,
                             const int* __restrict__ pos, int n, uint64_t* __restrict__ tiles) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (flag[i]) tiles[pos[i]] = sorted[i];
}

__global__ void k_mc_hash_clear(uint64_t* key, int* val, int cap) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += gridDim.x * blockDim.x) {
        key[i] = kEmptyKey;
        val[i] = -1;
    }
}

__global__ void k_mc_hash_insert(const uint64_t* __restrict__ tiles, int m, uint64_t* hkey, int* hval, int cap,
                                 unsigned* err) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        const uint64_t k = tiles[i];
        const uint32_t msk = (uint32_t)cap - 1u;
        uint32_t p = (uint32_t)mix64(k) & msk;
        bool done = false;
        for (int probe = 0; probe < cap && !done; ++probe) {
            const unsigned long long prev = atomicCAS((unsigned long long*)&hkey[p], kEmptyKey, k);
            if (prev == kEmptyKey || prev == k) {
                hval[p] = i;
                done = true;
            }
            p = (p + 1u) & msk;
        }
        if (!done) atomicOr(err, kErrHashFull);
    }
}

// Ranks of the processed tiles: a bit per tile of a box (with the set bits
// before each word), or a hash of their keys.
struct TileIndex {
    const unsigned* bits;  // null: the hash
    const int* before;
    int lo[3], dim[3];     // the box: lower corner and extents (leaf coordinates)
    HashView th;
    TileBase tb;
};

__host__ __device__ inline long long tile_bit(const int* lo, const int* dim, long long x, long long y, long long z) {
    return ((x - lo[0]) * dim[1] + (y - lo[1])) * dim[2] + (z - lo[2]);
}

__device__ inline int tile_rank(const TileIndex& t, long long x, long long y, long long z) {
    if (t.bits) {
        if (x < t.lo[0] || y < t.lo[1] || z < t.lo[2] || x >= t.lo[0] + t.dim[0] || y >= t.lo[1] + t.dim[1] ||
            z >= t.lo[2] + t.dim[2])
            return -1;
        const long long b = tile_bit(t.lo, t.dim, x, y, z);
        const unsigned w = t.bits[b >> 5], m = 1u << (b & 31);
        return (w & m) ? t.before[b >> 5] + __popc(w & (m - 1u)) : -1;
    }
    const uint64_t k = tile_key(x, y, z, t.tb.b);
    return k == kBadKey ? -1 : hash_find(t.th, k);
}

__constant__ int c_face[7][3] = {{0, 0, 0}, {-1, 0, 0}, {1, 0, 0}, {0, -1, 0}, {0, 1, 0}, {0, 0, -1}, {0, 0, 1}};

__global__ void k_mc_mark(const int4* __restrict__ origin, int n, TileIndex t, unsigned* __restrict__ bits) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < 7ll * n;
         i += (long long)gridDim.x * blockDim.x) {
        const int4 o = origin[i / 7];
        const int* d = c_face[i % 7];
        const long long b = tile_bit(t.lo, t.dim, (o.x >> 3) + d[0], (o.y >> 3) + d[1], (o.z >> 3) + d[2]);
        atomicOr(&bits[b >> 5], 1u << (b & 31));
    }
}

__global__ void k_mc_count(const unsigned* __restrict__ bits, long long words, int* __restrict__ cnt) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < words;
         i += (long long)gridDim.x * blockDim.x)
        cnt[i] = __popc(bits[i]);
}

__global__ void k_mc_list(TileIndex t, long long words, uint64_t* __restrict__ tiles) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < words;
         i += (long long)gridDim.x * blockDim.x) {
        int r = t.before[i];
        for (unsigned w = t.bits[i]; w; w &= w - 1u) {
            const long long b = 32 * i + __ffs(w) - 1;
            const long long z = b % t.dim[2], y = b / t.dim[2] % t.dim[1], x = b / t.dim[2] / t.dim[1];
            tiles[r++] = tile_key(x + t.lo[0], y + t.lo[1], z + t.lo[2], t.tb.b);
        }
    }
}

// ---------------------------------------------------------------- cells

constexpr int kMcThreads = 128;

struct TileCtx {
    long long t[3];  // leaf coordinates of the tile
};

__device__ inline TileCtx tile_of(uint64_t key, const TileBase& tb) {
    return TileCtx{{(long long)(key >> 42) + tb.b[0], (long long)((key >> 21) & (kAxisLim - 1)) + tb.b[1],
                    (long long)(key & (kAxisLim - 1)) + tb.b[2]}};
}

// Slots of the 8 leaves that hold the tile's corners, and the ranks of its 27
// neighbour tiles (-1: not processed), by separate warps.
__device__ inline void stage_slots(const GridView& g, const TileIndex& ti, const TileCtx& tc, int* s_leaf, int* s_tr) {
    const int t = threadIdx.x;
    if (t < 8) s_leaf[t] = hash_find_leaf(g.hash, tc.t[0] + (t >> 2), tc.t[1] + ((t >> 1) & 1), tc.t[2] + (t & 1));
    if (t >= 32 && t < 32 + 27) {
        const int q = t - 32;
        s_tr[q] = tile_rank(ti, tc.t[0] + q / 9 - 1, tc.t[1] + (q / 3) % 3 - 1, tc.t[2] + q % 3 - 1);
    }
}

// Corner (x, y, z) in [0, 8] of the tile.
__device__ inline float corner_value(const GridView& g, const int* s_leaf, int x, int y, int z) {
    const int slot = s_leaf[((x >> 3) << 2) | ((y >> 3) << 1) | (z >> 3)];
    return slot >= 0 ? g.values[(size_t)slot * kLeafVoxels + voxel_off(x, y, z)] : g.background;
}

// The listed cells (bit z of byte x * 8 + y of the tile's mask), ascending, by
// the first 64 threads; every thread gets their count.
__device__ inline int list_cells(unsigned bits, unsigned short* s_list, int* s_w) {
    const int t = threadIdx.x, lane = t & 31;
    int x = t < 64 ? __popc(bits) : 0;
    const int c = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31 && t < 64) s_w[t >> 5] = x;
    __syncthreads();
    if (t < 64)
        for (int p = (t >= 32 ? s_w[0] : 0) + x - c; bits; bits &= bits - 1u)
            s_list[p++] = (unsigned short)(t * 8 + __ffs(bits) - 1);
    const int n = s_w[0] + s_w[1];
    __syncthreads();
    return n;
}

// Exclusive block scan of one int per thread; *total = the sum.
__device__ inline int block_scan(int v, int* s_w, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_w[w] = x;
    __syncthreads();
    int before = x - v, all = 0;
#pragma unroll
    for (int q = 0; q < kMcThreads / 32; ++q) {
        if (q < w) before += s_w[q];
        all += s_w[q];
    }
    *total = all;
    __syncthreads();
    return before;
}

// Another cell holding the edge: its tile offset (-1..1 per axis) and local
// cell coordinates; `order` compares it with the current cell in visit order
// (negative: visited earlier).
struct CellRef {
    int toff[3];
    int loc[3];
};

__device__ inline CellRef cell_at(const int* loc, const int* delta) {
    CellRef r;
    for (int k = 0; k < 3; ++k) {
        const int v = loc[k] + delta[k];
        r.toff[k] = v < 0 ? -1 : (v > 7 ? 1 : 0);
        r.loc[k] = v & 7;
    }
    return r;
}

__device__ inline CellRef loc_self(const int* loc) {
    const int zero[3] = {0, 0, 0};
    return cell_at(loc, zero);
}

__device__ inline int tr_index(const int* toff) { return (toff[0] + 1) * 9 + (toff[1] + 1) * 3 + (toff[2] + 1); }

// lexicographic comparison of (tile offset, local cell) pairs
__device__ inline bool visited_before(const CellRef& a, const CellRef& b) {
    for (int k = 0; k < 3; ++k)
        if (a.toff[k] != b.toff[k]) return a.toff[k] < b.toff[k];
    for (int k = 0; k < 3; ++k)
        if (a.loc[k] != b.loc[k]) return a.loc[k] < b.loc[k];
    return false;
}

// The other cell holding edge e of the cell at `loc` listed q-th in c_mc_nb,
// and the edge's index there.
__device__ inline CellRef edge_nb(int e, int q, const int* loc, int& e2) {
    const int code = c_mc_nb[e][q];
    const int delta[3] = {(code & 3) - 1, ((code >> 2) & 3) - 1, ((code >> 4) & 3) - 1};
    e2 = code >> 8;
    return cell_at(loc, delta);
}

__device__ inline unsigned edge_flags(int ci) {
    unsigned m = 0;
#pragma unroll
    for (int e = 0; e < 12; ++e) m |= (unsigned)(((ci >> c_edge[e][0]) ^ (ci >> c_edge[e][1])) & 1) << e;
    return m;
}

__global__ void __launch_bounds__(kMcThreads) k_mc_classify(GridView g, TileIndex ti,
                                                           const uint64_t* __restrict__ tiles, float iso,
                                                           uint32_t* __restrict__ words,
                                                           unsigned char* __restrict__ cells, int* __restrict__ vcount,
                                                           int* __restrict__ tcount) {
    __shared__ unsigned short s_row[81];  // bit z: corner (x, y, z) lies below the isovalue
    __shared__ unsigned short s_list[512];
    __shared__ int s_leaf[8], s_tr[27], s_w[kMcThreads / 32];
    const TileCtx tc = tile_of(tiles[blockIdx.x], ti.tb);
    const int t = threadIdx.x;
    stage_slots(g, ti, tc, s_leaf, s_tr);
    __syncthreads();
    if (t < 81) {
        const int x = t / 9, y = t % 9;
        const int s0 = s_leaf[((x >> 3) << 2) | ((y >> 3) << 1)];
        const float bg = g.background;
        float4 a = make_float4(bg, bg, bg, bg), b = a;
        if (s0 >= 0) {
            const float4* v = reinterpret_cast<const float4*>(g.values + (size_t)s0 * kLeafVoxels + voxel_off(x, y, 0));
            a = v[0];
            b = v[1];
        }
        const float e = corner_value(g, s_leaf, x, y, 8);
        unsigned r = 0;
        r |= (unsigned)(a.x < iso) | (unsigned)(a.y < iso) << 1 | (unsigned)(a.z < iso) << 2 | (unsigned)(a.w < iso) << 3;
        r |= (unsigned)(b.x < iso) << 4 | (unsigned)(b.y < iso) << 5 | (unsigned)(b.z < iso) << 6 |
             (unsigned)(b.w < iso) << 7 | (unsigned)(e < iso) << 8;
        s_row[t] = (unsigned short)r;
    }
    __syncthreads();
    unsigned on = 0;
    if (t < 64) {
        const unsigned short* r = s_row + (t >> 3) * 9 + (t & 7);
        const unsigned all = r[0] & r[1] & r[9] & r[10], any = r[0] | r[1] | r[9] | r[10];
        on = ((any | (any >> 1)) & ~(all & (all >> 1))) & 0xffu;
        cells[(size_t)blockIdx.x * 64 + t] = (unsigned char)on;
    }
    const int n = list_cells(on, s_list, s_w);
    int vrun = 0, trun = 0;
    for (int base = 0; base < n; base += kMcThreads) {
        const bool valid = base + t < n;
        const int c = valid ? s_list[base + t] : 0;
        const int loc[3] = {c >> 6, (c >> 3) & 7, c & 7};
        unsigned cm = 0;
        int ci = 0, nt = 0;
        if (valid) {
            const unsigned short* r = s_row + loc[0] * 9 + loc[1];
            // corners 0..3: (0,0) (1,0) (1,1) (0,1) in (x, y) at z, 4..7 at z + 1
            const unsigned q[4] = {(unsigned)r[0] >> loc[2], (unsigned)r[9] >> loc[2], (unsigned)r[10] >> loc[2],
                                   (unsigned)r[1] >> loc[2]};
#pragma unroll
            for (int k = 0; k < 4; ++k) ci |= (int)((q[k] & 1u) << k | ((q[k] >> 1) & 1u) << (4 + k));
            const unsigned fl = edge_flags(ci);
            nt = d_mc_ntri[ci];
            // this cell creates a flagged edge iff no other processed cell
            // holding it is visited earlier
            const CellRef self = loc_self(loc);
            for (int e = 0; e < 12; ++e) {
                if (!((fl >> e) & 1u)) continue;
                bool first = true;
                for (int k = 0; k < 3 && first; ++k) {
                    int e2;
                    const CellRef o = edge_nb(e, k, loc, e2);
                    if (s_tr[tr_index(o.toff)] >= 0 && visited_before(o, self)) first = false;
                }
                if (first) cm |= 1u << e;
            }
        }
        int tot;
        const int pre = block_scan(__popc(cm) | (nt << 16), s_w, &tot);  // both sums stay below 2^15
        if (valid)
            words[(size_t)blockIdx.x * 512 + c] = (uint32_t)ci | (cm << 8) | ((uint32_t)(vrun + (pre & 0xffff)) << 20);
        vrun += tot & 0xffff;
        trun += tot >> 16;
    }
    if (t == 0) {
        vcount[blockIdx.x] = vrun;
        tcount[blockIdx.x] = trun;
    }
}

__global__ void __launch_bounds__(kMcThreads) k_mc_emit(GridView g, TileIndex ti, const uint64_t* __restrict__ tiles,
                                                       float iso, double vs, const uint32_t* __restrict__ words,
                                                       const unsigned char* __restrict__ cells,
                                                       const int* __restrict__ tcount, const int* __restrict__ vbase,
                                                       const int* __restrict__ tbase, double* __restrict__ verts,
                                                       uint32_t* __restrict__ tris) {
    __shared__ unsigned short s_list[512];
    __shared__ int s_leaf[8], s_tr[27], s_w[kMcThreads / 32];
    __shared__ uint32_t s_ev[kMcThreads][13];  // vertex of each edge of a thread's cell (odd pitch)
    if (tcount[blockIdx.x] == 0) return;
    const TileCtx tc = tile_of(tiles[blockIdx.x], ti.tb);
    const int t = threadIdx.x;
    stage_slots(g, ti, tc, s_leaf, s_tr);
    const int n = list_cells(t < 64 ? cells[(size_t)blockIdx.x * 64 + t] : 0u, s_list, s_w);
    const int vb = vbase[blockIdx.x];
    size_t t0 = (size_t)tbase[blockIdx.x];
    uint32_t* ev = s_ev[t];
    for (int base = 0; base < n; base += kMcThreads) {
        const bool valid = base + t < n;
        const int c = valid ? s_list[base + t] : 0;
        const uint32_t wd = valid ? words[(size_t)blockIdx.x * 512 + c] : 0u;
        const int ci = (int)(wd & 255u);
        const int nt = valid ? d_mc_ntri[ci] : 0;
        int tot;
        const int tpre = block_scan(nt, s_w, &tot);
        if (valid) {
            const int loc[3] = {c >> 6, (c >> 3) & 7, c & 7};
            const unsigned cm = (wd >> 8) & 0xfffu;
            const int vpre = (int)(wd >> 20);
            const unsigned fl = edge_flags(ci);
            for (int e = 0; e < 12; ++e) {
                if (!((fl >> e) & 1u)) continue;
                if ((cm >> e) & 1u) {
                    const uint32_t vi = (uint32_t)(vb + vpre + __popc(cm & ((1u << e) - 1u)));
                    ev[e] = vi;
                    const int* a = c_corner[c_edge[e][0]];
                    const int* b = c_corner[c_edge[e][1]];
                    const float va = corner_value(g, s_leaf, loc[0] + a[0], loc[1] + a[1], loc[2] + a[2]);
                    const float vbv = corner_value(g, s_leaf, loc[0] + b[0], loc[1] + b[1], loc[2] + b[2]);
                    const float d = __fsub_rn(vbv, va);
                    const double f = (fabsf(d) > 1e-10f) ? (double)__fdiv_rn(__fsub_rn(iso, va), d) : 0.5;
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const long long o = 8 * tc.t[k] + loc[k];
                        const double pa = __dmul_rn((double)(o + a[k]), vs);
                        const double pb = __dmul_rn((double)(o + b[k]), vs);
                        verts[(size_t)vi * 3 + k] = __dadd_rn(pa, __dmul_rn(f, __dsub_rn(pb, pa)));
                    }
                } else {
                    // the creator: the earliest processed other cell holding the edge
                    int e2 = -1;
                    CellRef cr = loc_self(loc);
                    bool have = false;
                    for (int q = 0; q < 3; ++q) {
                        int f;
                        const CellRef o = edge_nb(e, q, loc, f);
                        if (s_tr[tr_index(o.toff)] < 0) continue;
                        if (!have || visited_before(o, cr)) {
                            cr = o;
                            e2 = f;
                            have = true;
                        }
                    }
                    const int rank = s_tr[tr_index(cr.toff)];
                    const uint32_t w2 = words[(size_t)rank * 512 + (cr.loc[0] << 6) + (cr.loc[1] << 3) + cr.loc[2]];
                    const unsigned cm2 = (w2 >> 8) & 0xfffu;
                    ev[e] = (uint32_t)(vbase[rank] + (int)(w2 >> 20) + __popc(cm2 & ((1u << e2) - 1u)));
                }
            }
            const int4 row = *reinterpret_cast<const int4*>(d_mc_tri[ci]);
            const int8_t* tri = reinterpret_cast<const int8_t*>(&row);
            uint32_t* out = tris + (t0 + tpre) * 3;
#pragma unroll
            for (int k = 0; k < 15; ++k)
                if (k < 3 * nt) out[k] = ev[tri[k]];
        }
        t0 += tot;
    }
}

// The processed tiles of a grid in visit order, and their index.
struct TileList {
    char* block = nullptr;
    uint64_t* tiles = nullptr;
    int m = 0;
    TileIndex index{};
};

int tile_list(vlr_ctx* ctx, const vlr_grid* g, TileList& L) {
    cudaStream_t st = ctx->stream;
    TileIndex& ti = L.index;
    for (int a = 0; a < 3; ++a) ti.tb.b[a] = g->base[a];
    const int thr = 256;
    auto blocks = [&](long long n) { return (int)std::max(1ll, std::min((n + thr - 1) / thr, ctx->sm_count * 8ll)); };
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    // One bit per tile of the leaves' box while its words number at most 16
    // per leaf (or 2^16: such a list costs a few launches whatever is in it):
    // 8 bytes a word against the sort's 420 bytes a leaf, and one pass over
    // them against 16 launches.  Narrow bands hold about 13 words a leaf at
    // 2.5M leaves in 8192^3 voxels, 0.2 on a single sphere; a few leaves far
    // apart take the sort.
    double bits = 1.0;
    for (int a = 0; a < 3; ++a) {
        ti.lo[a] = g->box[a] - 1;
        const long long d = (long long)g->box[3 + a] - g->box[a] + 3;
        ti.dim[a] = (int)d;
        bits *= (double)d;
    }
    if (bits <= 32.0 * std::max(65536.0, 16.0 * g->n)) {
        const long long words = ((long long)bits + 31) / 32;
        unsigned* d_bits = nullptr;
        VLR_CUDA(ctx, cudaMallocFromPoolAsync((void**)&L.block, up(4 * words) + 4 * words + 256, ctx->pool, st));
        d_bits = (unsigned*)L.block;
        int* before = (int*)(L.block + up(4 * words));
        int* total = before + words;
        ti.bits = d_bits;
        ti.before = before;
        VLR_CUDA(ctx, cudaMemsetAsync(d_bits, 0, 4 * words, st));
        k_mc_mark<<<blocks(7ll * g->n), thr, 0, st>>>(g->origin, g->n, ti, d_bits);
        k_mc_count<<<blocks(words), thr, 0, st>>>(d_bits, words, before);
        int rc = scan_exclusive(ctx, before, before, words, total);
        if (!rc) rc = read_int_checked(ctx, total, &L.m, "volume_to_mesh");
        if (rc) return rc;
        VLR_CUDA(ctx, cudaMallocFromPoolAsync((void**)&L.tiles, sizeof(uint64_t) * L.m, ctx->pool, st));
        k_mc_list<<<blocks(words), thr, 0, st>>>(ti, words, L.tiles);
        VLR_CUDA(ctx, cudaGetLastError());
        return VLR_OK;
    }
    const int n7 = 7 * g->n;
    const size_t sort_bytes = radix_scratch_bytes(n7, 8);
    char* buf = nullptr;
    VLR_CUDA(ctx, cudaMallocFromPoolAsync((void**)&buf, (size_t)n7 * (8 + 4 + 4 + 4) + sort_bytes + 1024, ctx->pool, st));
    char* p = buf;
    auto take = [&](size_t b) {
        char* r = p;
        p += b;
        return r;
    };
    uint64_t* keys = (uint64_t*)take((size_t)n7 * 8);
    unsigned* idx = (unsigned*)take((size_t)n7 * 4);
    int* flag = (int*)take((size_t)n7 * 4);
    int* pos = (int*)take((size_t)n7 * 4 + 16);
    void* scratch = (void*)(((uintptr_t)p + 255) & ~(uintptr_t)255);
    auto run = [&]() -> int {
        // 63-bit keys (a bad key, all ones, sorts last)
        k_mc_cand<<<blocks(n7), thr, 0, st>>>(g->origin, g->n, ti.tb, keys, idx, ctx->d_errword);
        uint64_t* sorted;
        unsigned* order;
        int rc = radix_sort(ctx, keys, idx, n7, 64, scratch, &sorted, &order);
        if (rc) return rc;
        k_mc_unique<<<blocks(n7), thr, 0, st>>>(sorted, n7, flag);
        rc = scan_exclusive(ctx, flag, pos, n7, pos + n7);
        if (!rc) rc = read_int_checked(ctx, pos + n7, &L.m, "volume_to_mesh");
        if (rc || L.m <= 0) return rc;
        int hcap = 64;
        while (hcap < 2ll * L.m && hcap < (1 << 30)) hcap <<= 1;
        VLR_CUDA(ctx, cudaMallocFromPoolAsync((void**)&L.tiles, sizeof(uint64_t) * L.m, ctx->pool, st));
        VLR_CUDA(ctx, cudaMallocFromPoolAsync((void**)&L.block, 12 * (size_t)hcap, ctx->pool, st));
        uint64_t* hkey = (uint64_t*)L.block;
        int* hval = (int*)(hkey + hcap);
        k_mc_compact<<<blocks(n7), thr, 0, st>>>(sorted, flag, pos, n7, L.tiles);
        k_mc_hash_clear<<<blocks(hcap), thr, 0, st>>>(hkey, hval, hcap);
        k_mc_hash_insert<<<blocks(L.m), thr, 0, st>>>(L.tiles, L.m, hkey, hval, hcap, ctx->d_errword);
        VLR_CUDA(ctx, cudaGetLastError());
        ti.bits = nullptr;
        ti.th.key = hkey;
        ti.th.val = hval;
        ti.th.cap = hcap;
        return VLR_OK;
    };
    const int rc = run();
    cudaFreeAsync(buf, st);
    return rc;
}

}  // namespace

// Marching cubes on the device: the counts, and (emit) the mesh in two
// allocations of the context's pool.
static int mesh_device(vlr_ctx* ctx, const vlr_grid* g, float iso, bool emit, double** d_verts, uint32_t** d_tris,
                       size_t* n_verts, size_t* n_tris) {
    *n_verts = 0;
    *n_tris = 0;
    if (g->n == 0) return VLR_OK;
    int rc = ensure_tables(ctx);
    if (rc) return rc;
    cudaStream_t st = ctx->stream;
    if (g->n > (1 << 27)) return set_error(ctx, VLR_ERR_CAPACITY, "volume_to_mesh: too many leaves");
    TileList L;
    char* buf = nullptr;
    auto run = [&]() -> int {
        rc = tile_list(ctx, g, L);
        const int m = L.m;
        if (rc || m <= 0) return rc;
        VLR_CUDA(ctx, cudaMallocFromPoolAsync((void**)&buf, (size_t)m * (512 * 4 + 64 + 16) + 64, ctx->pool, st));
        uint32_t* words = (uint32_t*)buf;
        unsigned char* cells = (unsigned char*)(words + (size_t)m * 512);
        int* vcount = (int*)(cells + (size_t)m * 64);
        int* tcount = vcount + m;
        int* vbase = tcount + m;        // m and the total
        int* tbase = vbase + m + 1;     // m and the total
        const GridView gv = make_view(g);
        VLR_TIMED(ctx, "k_mc_classify", k_mc_classify<<<m, kMcThreads, 0, st>>>(gv, L.index, L.tiles, iso, words, cells,
                                                                               vcount, tcount));
        VLR_CUDA(ctx, cudaGetLastError());
        rc = scan_exclusive(ctx, vcount, vbase, m, vbase + m);
        if (!rc) rc = scan_exclusive(ctx, tcount, tbase, m, tbase + m);
        if (rc) return rc;
        int* h = static_cast<int*>(ctx->pinned) + 40;
        VLR_CUDA(ctx, cudaMemcpyAsync(h, tbase + m, sizeof(int), cudaMemcpyDeviceToHost, st));
        int nv = 0;
        rc = read_int_checked(ctx, vbase + m, &nv, "volume_to_mesh");
        if (rc) return rc;
        if (nv < 0 || *h < 0)
            return set_error(ctx, VLR_ERR_CAPACITY, "volume_to_mesh: more than 2^31 vertices or triangles");
        *n_verts = (size_t)nv;
        *n_tris = (size_t)*h;
        if (!emit) return VLR_OK;
        VLR_CUDA(ctx, cudaMallocFromPoolAsync((void**)d_verts, std::max<size_t>(*n_verts, 1) * 24, ctx->pool, st));
        VLR_CUDA(ctx, cudaMallocFromPoolAsync((void**)d_tris, std::max<size_t>(*n_tris, 1) * 12, ctx->pool, st));
        VLR_TIMED(ctx, "k_mc_emit",
                  k_mc_emit<<<m, kMcThreads, 0, st>>>(gv, L.index, L.tiles, iso, g->xf.voxel_size, words, cells, tcount,
                                                     vbase, tbase, *d_verts, *d_tris));
        VLR_CUDA(ctx, cudaGetLastError());
        return VLR_OK;
    };
    rc = run();
    for (void* p : {(void*)buf, (void*)L.block, (void*)L.tiles})
        if (p) cudaFreeAsync(p, st);
    return rc;
}

int mc_triangle_table(int8_t* out) {
    std::memcpy(out, mc_table().tri, sizeof(mc_table().tri));
    return VLR_OK;
}

}  // namespace vlr

// A mesh on the device (stream-ordered allocations of the context's pool).
struct vlr_mesh {
    vlr_ctx* ctx = nullptr;
    double* verts = nullptr;
    uint32_t* tris = nullptr;
    size_t n_verts = 0, n_tris = 0;
};

using namespace vlr;

extern "C" {

void vlr_mesh_destroy(vlr_mesh* m) {
    if (!m) return;
    if (m->verts) cudaFreeAsync(m->verts, m->ctx->stream);
    if (m->tris) cudaFreeAsync(m->tris, m->ctx->stream);
    delete m;
}

int vlr_mesh_create(vlr_ctx* ctx, const vlr_grid* g, float isovalue, vlr_mesh** out, size_t* n_vertices,
                    size_t* n_triangles) {
    if (!ctx || !g || !out || !n_vertices || !n_triangles) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    *out = nullptr;
    if (g->kind != VLR_KIND_F32_WORLD) return set_error(ctx, VLR_ERR_INVALID, "grid is not a world-unit f32 grid");
    vlr_mesh* m = new vlr_mesh();
    m->ctx = ctx;
    const int rc = mesh_device(ctx, g, isovalue, true, &m->verts, &m->tris, &m->n_verts, &m->n_tris);
    *n_vertices = m->n_verts;
    *n_triangles = m->n_tris;
    if (rc) {
        vlr_mesh_destroy(m);
        return rc;
    }
    *out = m;
    return VLR_OK;
}

int vlr_mesh_read(vlr_ctx* ctx, const vlr_mesh* m, double* vertices, size_t cap_vertices, uint32_t* triangles,
                  size_t cap_triangles) {
    if (!ctx || !m) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    const size_t cv = std::min(cap_vertices, m->n_verts), ct = std::min(cap_triangles, m->n_tris);
    int rc = VLR_OK;
    if (vertices && cv) rc = d2h_copy(ctx, vertices, m->verts, cv * 24);
    if (!rc && triangles && ct) rc = d2h_copy(ctx, triangles, m->tris, ct * 12);
    return rc;
}

int vlr_volume_to_mesh(vlr_ctx* ctx, const vlr_grid* g, float isovalue, double* vertices, size_t cap_vertices,
                       uint32_t* triangles, size_t cap_triangles, size_t* n_vertices, size_t* n_triangles) {
    if (!ctx || !g || !n_vertices || !n_triangles) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    if (g->kind != VLR_KIND_F32_WORLD) return set_error(ctx, VLR_ERR_INVALID, "grid is not a world-unit f32 grid");
    vlr_mesh m;
    m.ctx = ctx;
    const bool emit = (vertices && cap_vertices) || (triangles && cap_triangles);
    int rc = mesh_device(ctx, g, isovalue, emit, &m.verts, &m.tris, n_vertices, n_triangles);
    m.n_verts = *n_vertices;
    m.n_tris = *n_triangles;
    if (!rc && emit) rc = vlr_mesh_read(ctx, &m, vertices, cap_vertices, triangles, cap_triangles);
    if (m.verts) cudaFreeAsync(m.verts, ctx->stream);
    if (m.tris) cudaFreeAsync(m.tris, ctx->stream);
    return rc;
}

int vlr_mc_triangle_table(int8_t* out) {
    if (!out) return VLR_ERR_INVALID;
    return vlr::mc_triangle_table(out);
}

}  // extern "C"
