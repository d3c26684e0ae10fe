// advect_particles / advect_particles_euler (src/tools/advection.rs:58-110)
// on particle positions: RK4 (or forward Euler) through a VelocityField of
// three grids.  VelocityField::sample is three sample_trilinear calls widened
// to f64 (src/tools/advection.rs:16-24); the position arithmetic is f64 in the
// reference's order, with explicitly rounded operations so nothing is
// contracted into an FMA.
//
// vlr_advect_points is the whole crate call: the position update followed by
// PointDataGrid::rebin (src/points/point_grid.rs:258-266), which drains every
// leaf and re-inserts each particle into the leaf of
// AffineMap::world_to_index(position) aligned to 8.  The crate drains its
// leaves in HashMap order; here leaves are drained in ascending (x, y, z)
// origin order, so with particles handed in that binned order the re-binned
// grid is a stable sort of the particles by their new leaf.  On the GPU:
//   k_points_move    position update, then the new leaf per particle as three
//                    order-preserving 29-bit keys (one per axis) and their
//                    bounding box
//   k_points_keys    one key per particle with just the bits of that box
//   (sort)           stable radix sort of (key, particle index)
//   k_points_emit    particles gathered into sorted order; a flag where the
//                    leaf changes
//   (scan)           leaf ranks; k_points_leaves writes each leaf's origin and
//                    first particle
// A box of more than 64 bits takes three stable sorts instead: z, then y, then
// x, the keys of each pass gathered in the order the previous pass left.
#include <algorithm>

#include "box_reduce.cuh"
#include "ref_ops.hpp"
#include "sort_reduce.hpp"

namespace vlr {
namespace {

struct V3 {
    double x, y, z;
};

// The velocity grids and, with HINT, the leaf of each that the particle starts
// in: its samples (a step moves it little) come from that leaf's neighbour row,
// without it every sample searches the hash.  SAME: the grids share their
// transform, so position and fractions are computed once for the three.
template <bool SAME, bool HINT>
struct Field {
    const GridView& vx;
    const GridView& vy;
    const GridView& vz;
    Hint hx, hy, hz;

    // h: the leaf of vx that holds p, a its cell there (HINT)
    __device__ __forceinline__ Field(const GridView& x, const GridView& y, const GridView& z, const V3& p, const Cell& a,
                                     const Hint& h)
        : vx(x), vy(y), vz(z) {
        if (HINT) {
            hx = h;
            const Cell b = SAME ? a : cell_of(vy, p.x, p.y, p.z);
            hy = hint_at(vy, b.i, b.j, b.k);
            const Cell c = SAME ? a : cell_of(vz, p.x, p.y, p.z);
            hz = hint_at(vz, c.i, c.j, c.k);
        }
    }

    __device__ __forceinline__ V3 operator()(const V3& p) const {
        const Cell a = cell_of(vx, p.x, p.y, p.z);
        return V3{(double)read_cell(vx, a, HINT ? hx : Hint()),
                  (double)read_cell(vy, SAME ? a : cell_of(vy, p.x, p.y, p.z), HINT ? hy : Hint()),
                  (double)read_cell(vz, SAME ? a : cell_of(vz, p.x, p.y, p.z), HINT ? hz : Hint())};
    }
};

__device__ __forceinline__ V3 scale(double s, const V3& v) {
    return V3{__dmul_rn(s, v.x), __dmul_rn(s, v.y), __dmul_rn(s, v.z)};
}

// pos + k * f (k * f rounded first, as `pos[a] + k[a] * 0.5` evaluates)
__device__ __forceinline__ V3 axpy(const V3& pos, const V3& k, double f) {
    return V3{__dadd_rn(pos.x, __dmul_rn(k.x, f)), __dadd_rn(pos.y, __dmul_rn(k.y, f)),
              __dadd_rn(pos.z, __dmul_rn(k.z, f))};
}

// pos + (k1 + 2 k2 + 2 k3 + k4) / 6, summed left to right
__device__ __forceinline__ double rk4_comb(double p, double k1, double k2, double k3, double k4) {
    const double s = __dadd_rn(__dadd_rn(__dadd_rn(k1, __dmul_rn(2.0, k2)), __dmul_rn(2.0, k3)), k4);
    return __dadd_rn(p, __ddiv_rn(s, 6.0));
}

template <class F>
__device__ __forceinline__ V3 move_in(const F& v, const V3& p, double dt, int rk4) {
    const V3 v1 = v(p);
    if (!rk4)
        return V3{__dadd_rn(p.x, __dmul_rn(dt, v1.x)), __dadd_rn(p.y, __dmul_rn(dt, v1.y)),
                  __dadd_rn(p.z, __dmul_rn(dt, v1.z))};
    const V3 k1 = scale(dt, v1);
    const V3 k2 = scale(dt, v(axpy(p, k1, 0.5)));
    const V3 k3 = scale(dt, v(axpy(p, k2, 0.5)));
    const V3 k4 = scale(dt, v(axpy(p, k3, 1.0)));
    return V3{rk4_comb(p.x, k1.x, k2.x, k3.x, k4.x), rk4_comb(p.y, k1.y, k2.y, k3.y, k4.y),
              rk4_comb(p.z, k1.z, k2.z, k3.z, k4.z)};
}

// One RK4 or forward Euler step of a position.  A warp goes by its particles'
// leaves when all of them start in one: particles without a leaf search the
// hash for every sample, and a warp that does both takes the time of both (RK4
// of 100k particles, the kernel, both and this way: most outside 125 leaves 122
// and 78 us, all outside 124 and 86, 9 % outside 20k leaves 114 and 98, all
// inside 48 and 48; 1,000 particles there 9 % outside 35 and 58).
template <bool SAME>
__device__ __forceinline__ V3 move_point(const GridView& vx, const GridView& vy, const GridView& vz, const V3& p,
                                         double dt, int rk4) {
    const Cell a = cell_of(vx, p.x, p.y, p.z);
    const Hint h = hint_at(vx, a.i, a.j, a.k);
    if (__all_sync(__activemask(), h.slot >= 0)) return move_in(Field<SAME, true>(vx, vy, vz, p, a, h), p, dt, rk4);
    return move_in(Field<SAME, false>(vx, vy, vz, p, a, h), p, dt, rk4);
}

template <bool SAME>
__global__ void k_advect_particles(GridView vx, GridView vy, GridView vz, double* __restrict__ pos, int n, double dt,
                                   int rk4) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const V3 out = move_point<SAME>(vx, vy, vz, V3{pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]}, dt, rk4);
        pos[3 * i] = out.x;
        pos[3 * i + 1] = out.y;
        pos[3 * i + 2] = out.z;
    }
}

// Whether the three grids sample at the same index position.
bool same_transform(const GridView& a, const GridView& b) {
    return a.inv_vs == b.inv_vs && a.t_origin[0] == b.t_origin[0] && a.t_origin[1] == b.t_origin[1] &&
           a.t_origin[2] == b.t_origin[2];
}

// f64::round (half away from zero) then Rust's saturating `as i32`.
__device__ __forceinline__ int32_t round_to_i32(double f) {
    const double r = round(f);
    if (r != r) return 0;
    if (r >= 2147483647.0) return 2147483647;
    if (r <= -2147483648.0) return INT32_MIN;
    return (int32_t)r;
}

struct InvRows {
    double r[12];  // rows 0..2 of the world -> index 4x4 map
};

// Leaf origin coordinate (a multiple of 8) -> order-preserving key below 2^29.
__device__ __forceinline__ unsigned leaf_key(int32_t v) { return ((unsigned)v >> 3) ^ (1u << 28); }
__device__ __forceinline__ int32_t key_leaf(unsigned k) { return (int32_t)((k ^ (1u << 28)) << 3); }

// Bound: load latency, the instruction cache (45 % of the issue slots) and the f64
// and conversion instructions of 12 samples a particle (RK4).  300k particles in
// a 64^3 field: 124 us with up to 8 hash searches a sample, 49 us from the
// particle's leaf.
template <bool SAME>
__global__ void __launch_bounds__(256) k_points_move(GridView vx, GridView vy, GridView vz,
                                                    vlr_particle* __restrict__ pts, int n, double dt, int rk4,
                                                    InvRows inv, unsigned* __restrict__ kx,
                                                    unsigned* __restrict__ ky, unsigned* __restrict__ kz,
                                                    unsigned* __restrict__ idx, int* __restrict__ box) {
    int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double* pp = pts[i].position;
        const V3 out = move_point<SAME>(vx, vy, vz, V3{pp[0], pp[1], pp[2]}, dt, rk4);
        pp[0] = out.x;
        pp[1] = out.y;
        pp[2] = out.z;
        // AffineMap::world_to_index: a*x + b*y + c*z + d, left to right, then aligned(3)
        unsigned* keys[3] = {kx, ky, kz};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double* r = inv.r + 4 * a;
            const double f = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(r[0], out.x), __dmul_rn(r[1], out.y)),
                                                 __dmul_rn(r[2], out.z)),
                                       r[3]);
            const unsigned k = leaf_key(round_to_i32(f) & ~7);
            keys[a][i] = k;
            lo[a] = min(lo[a], (int)k);
            hi[a] = max(hi[a], (int)k);
        }
        idx[i] = (unsigned)i;
    }
    block_box(lo, hi, box);
}

// Lower corner of the box and the bits of y and z in a packed key.
struct KeyBox {
    unsigned lo[3];
    int by, bz;
};

__global__ void k_points_keys(const unsigned* __restrict__ kx, const unsigned* __restrict__ ky,
                              const unsigned* __restrict__ kz, int n, KeyBox b, uint64_t* __restrict__ keys) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        keys[i] = ((uint64_t)(kx[i] - b.lo[0]) << (b.by + b.bz)) | ((uint64_t)(ky[i] - b.lo[1]) << b.bz) |
                  (uint64_t)(kz[i] - b.lo[2]);
}

__global__ void k_gather_keys(const unsigned* __restrict__ keys, const unsigned* __restrict__ perm, int n,
                              unsigned* __restrict__ out) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) out[j] = keys[perm[j]];
}

__global__ void k_points_emit(const vlr_particle* __restrict__ in, const unsigned* __restrict__ perm,
                              const unsigned* __restrict__ kx, const unsigned* __restrict__ ky,
                              const unsigned* __restrict__ kz, int n, vlr_particle* __restrict__ out,
                              int* __restrict__ head) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const unsigned i = perm[j];
        out[j] = in[i];
        int h = 1;
        if (j > 0) {
            const unsigned q = perm[j - 1];
            h = (kx[i] != kx[q]) | (ky[i] != ky[q]) | (kz[i] != kz[q]);
        }
        head[j] = h;
    }
}

__global__ void k_points_leaves(const unsigned* __restrict__ perm, const unsigned* __restrict__ kx,
                                const unsigned* __restrict__ ky, const unsigned* __restrict__ kz,
                                const int* __restrict__ head, const int* __restrict__ rank, int n,
                                int32_t* __restrict__ origins, uint32_t* __restrict__ start) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        if (!head[j]) continue;
        const int l = rank[j];
        const unsigned i = perm[j];
        origins[3 * l] = key_leaf(kx[i]);
        origins[3 * l + 1] = key_leaf(ky[i]);
        origins[3 * l + 2] = key_leaf(kz[i]);
        start[l] = (uint32_t)j;
    }
}

}  // namespace
}  // namespace vlr

using namespace vlr;

extern "C" {

int vlr_advect_particles(vlr_ctx* ctx, const vlr_grid* vx, const vlr_grid* vy, const vlr_grid* vz, double* positions,
                         size_t n, double dt, int rk4) {
    if (!ctx || !vx || !vy || !vz || (n && !positions)) return set_error(ctx, VLR_ERR_INVALID, "null argument");
    if (vx->kind != VLR_KIND_F32_WORLD || vy->kind != VLR_KIND_F32_WORLD || vz->kind != VLR_KIND_F32_WORLD)
        return set_error(ctx, VLR_ERR_INVALID, "velocity grids must be world-unit f32 grids");
    if (n == 0) return VLR_OK;
    if (n > (size_t)INT32_MAX / 3) return set_error(ctx, VLR_ERR_CAPACITY, "too many particles");
    double* d = nullptr;
    VLR_CUDA(ctx, cudaMallocFromPoolAsync(&d, sizeof(double) * 3 * n, ctx->pool, ctx->stream));
    int rc = h2d_copy(ctx, d, positions, sizeof(double) * 3 * n);
    const int blocks = (int)std::min<size_t>((n + 255) / 256, (size_t)ctx->sm_count * 16);
    const GridView gx = make_view(vx), gy = make_view(vy), gz = make_view(vz);
    auto* kernel = same_transform(gx, gy) && same_transform(gx, gz) ? k_advect_particles<true>
                                                                   : k_advect_particles<false>;
    if (!rc) {
        kernel<<<blocks, 256, 0, ctx->stream>>>(gx, gy, gz, d, (int)n, dt, rk4 ? 1 : 0);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = check_cuda(ctx, e, "k_advect_particles");
    }
    if (!rc) rc = d2h_copy(ctx, positions, d, sizeof(double) * 3 * n);
    cudaFreeAsync(d, ctx->stream);
    return rc ? rc : consume_device_errors(ctx, "vlr_advect_particles");
}

int vlr_advect_points(vlr_ctx* ctx, const vlr_grid* vx, const vlr_grid* vy, const vlr_grid* vz,
                      const double world_to_index[12], vlr_particle* particles, size_t n, double dt, int rk4,
                      int32_t* leaf_origins, uint32_t* leaf_start, size_t cap_leaves, size_t* n_leaves) {
    return vlr_advect_points_to(ctx, vx, vy, vz, world_to_index, particles, particles, n, dt, rk4, leaf_origins,
                                leaf_start, cap_leaves, n_leaves);
}

int vlr_advect_points_to(vlr_ctx* ctx, const vlr_grid* vx, const vlr_grid* vy, const vlr_grid* vz,
                         const double world_to_index[12], const vlr_particle* particles, vlr_particle* out, size_t n,
                         double dt, int rk4, int32_t* leaf_origins, uint32_t* leaf_start, size_t cap_leaves,
                         size_t* n_leaves) {
    if (!ctx || !vx || !vy || !vz || !world_to_index || !n_leaves || (n && (!particles || !out)) || !leaf_start ||
        (cap_leaves && !leaf_origins))
        return set_error(ctx, VLR_ERR_INVALID, "null argument");
    if (vx->kind != VLR_KIND_F32_WORLD || vy->kind != VLR_KIND_F32_WORLD || vz->kind != VLR_KIND_F32_WORLD)
        return set_error(ctx, VLR_ERR_INVALID, "velocity grids must be world-unit f32 grids");
    *n_leaves = 0;
    if (n == 0) {
        leaf_start[0] = 0;
        return VLR_OK;
    }
    if (n > ((size_t)1 << 28)) return set_error(ctx, VLR_ERR_CAPACITY, "more than 2^28 particles in one call");
    const int nn = (int)n;
    cudaStream_t st = ctx->stream;
    InvRows inv;
    for (int i = 0; i < 12; ++i) inv.r[i] = world_to_index[i];
    // one stream-ordered block: particles in and out, keys, permutation, flags, ranks, sort scratch
    const size_t pb = sizeof(vlr_particle) * n, wb = sizeof(unsigned) * n;
    const size_t sb = radix_scratch_bytes(nn, 8);
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t total = 2 * al(pb) + 10 * al(wb) + al(sizeof(int) * 8) + al(sb) + al(sizeof(int32_t) * 3 * n) +
                         al(sizeof(uint32_t) * (n + 1));
    char* blk = nullptr;
    if (cudaMallocFromPoolAsync((void**)&blk, total, ctx->pool, st) != cudaSuccess) {
        cudaGetLastError();
        return set_error(ctx, VLR_ERR_NOMEM, "vlr_advect_points: device allocation failed");
    }
    char* q = blk;
    auto take = [&](size_t b) {
        char* r = q;
        q += al(b);
        return r;
    };
    vlr_particle* d_in = (vlr_particle*)take(pb);
    vlr_particle* d_out = (vlr_particle*)take(pb);
    unsigned* kx = (unsigned*)take(wb);
    unsigned* ky = (unsigned*)take(wb);
    unsigned* kz = (unsigned*)take(wb);
    unsigned* idx = (unsigned*)take(wb);
    unsigned* kbuf = (unsigned*)take(wb);
    unsigned* pbuf = (unsigned*)take(wb);
    int* head = (int*)take(wb);
    int* rank = (int*)take(wb);
    uint64_t* keys = (uint64_t*)take(2 * wb);
    int* d_total = (int*)take(sizeof(int) * 8);
    int* d_box = d_total + 2;
    void* scratch = take(sb);
    int32_t* d_org = (int32_t*)take(sizeof(int32_t) * 3 * n);
    uint32_t* d_start = (uint32_t*)take(sizeof(uint32_t) * (n + 1));
    int rc = VLR_OK;
    auto fail = [&](int code) {
        cudaFreeAsync(blk, st);
        return code;
    };
    const int blocks = (int)std::min<size_t>((n + 255) / 256, (size_t)ctx->sm_count * 16);
    if ((rc = h2d_copy(ctx, d_in, particles, pb))) return fail(rc);
    const GridView gx = make_view(vx), gy = make_view(vy), gz = make_view(vz);
    auto* move = same_transform(gx, gy) && same_transform(gx, gz) ? k_points_move<true> : k_points_move<false>;
    if (cudaMemsetAsync(d_box, kBoxClear, 6 * sizeof(int), st) != cudaSuccess)
        return fail(check_cuda(ctx, cudaGetLastError(), "box"));
    VLR_TIMED(ctx, "k_points_move",
              move<<<blocks, 256, 0, st>>>(gx, gy, gz, d_in, nn, dt, rk4 ? 1 : 0, inv, kx, ky, kz, idx, d_box));
    int* hb = static_cast<int*>(ctx->pinned) + 32;
    if (cudaMemcpyAsync(hb, d_box, 6 * sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return fail(check_cuda(ctx, cudaGetLastError(), "particle update"));
    KeyBox kb;
    int kbits[3];
    for (int a = 0; a < 3; ++a) {
        kb.lo[a] = (unsigned)~hb[a];
        kbits[a] = bits_for((long long)hb[3 + a] - (long long)~hb[a]);
    }
    kb.by = kbits[1];
    kb.bz = kbits[2];
    const int bits = kbits[0] + kbits[1] + kbits[2];
    unsigned* perm = nullptr;
    if (bits <= 64) {
        k_points_keys<<<blocks, 256, 0, st>>>(kx, ky, kz, nn, kb, keys);
        uint64_t* ko = nullptr;
        rc = radix_sort(ctx, keys, idx, nn, bits, scratch, &ko, &perm);
        if (rc) return fail(rc);
    } else {
        // stable sorts by z, then y, then x: lexicographic (x, y, z), ties in
        // input order.  A sort may leave its result in its scratch, which the
        // next sort reuses, so each pass's permutation is first moved to pbuf.
        unsigned* ko = nullptr;
        if (cudaMemcpyAsync(kbuf, kz, wb, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            return fail(check_cuda(ctx, cudaGetLastError(), "key copy"));
        rc = radix_sort(ctx, kbuf, idx, nn, 29, scratch, &ko, &perm);
        if (rc) return fail(rc);
        const unsigned* axis_keys[2] = {ky, kx};
        for (int pass = 0; pass < 2; ++pass) {
            if (perm != pbuf && cudaMemcpyAsync(pbuf, perm, wb, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
                return fail(check_cuda(ctx, cudaGetLastError(), "permutation copy"));
            k_gather_keys<<<blocks, 256, 0, st>>>(axis_keys[pass], pbuf, nn, kbuf);
            rc = radix_sort(ctx, kbuf, pbuf, nn, 29, scratch, &ko, &perm);
            if (rc) return fail(rc);
        }
    }
    VLR_TIMED(ctx, "k_points_emit",
              k_points_emit<<<blocks, 256, 0, st>>>(d_in, perm, kx, ky, kz, nn, d_out, head));
    rc = scan_exclusive(ctx, head, rank, nn, d_total);
    if (rc) return fail(rc);
    k_points_leaves<<<blocks, 256, 0, st>>>(perm, kx, ky, kz, head, rank, nn, d_org, d_start);
    if (cudaGetLastError() != cudaSuccess) return fail(check_cuda(ctx, cudaGetLastError(), "k_points_leaves"));
    int leaves = 0;
    rc = read_int(ctx, d_total, &leaves);
    if (rc) return fail(rc);
    *n_leaves = (size_t)leaves;
    if ((size_t)leaves > cap_leaves) {
        fail(VLR_OK);
        return set_error(ctx, VLR_ERR_CAPACITY,
                         "vlr_advect_points: " + std::to_string(leaves) + " leaves exceed cap_leaves");
    }
    if ((rc = d2h_copy(ctx, out, d_out, pb)) ||
        (rc = d2h_copy(ctx, leaf_origins, d_org, sizeof(int32_t) * 3 * leaves)) ||
        (rc = d2h_copy(ctx, leaf_start, d_start, sizeof(uint32_t) * leaves)))
        return fail(rc);
    leaf_start[leaves] = (uint32_t)n;
    cudaFreeAsync(blk, st);
    return consume_device_errors(ctx, "vlr_advect_points");
}

}  // extern "C"
