// Stable LSD radix sort of (key, 32-bit payload) pairs, keys of 32 or 64 bits.
//
// A pass sorts by a digit of up to 8 bits, the key's bits shared evenly over
// the passes, in tiles of 2048 pairs (8 warps, 256 consecutive pairs a warp):
//   k_rs_hist     per-tile digit counts, [tile][digit]
//   k_rs_offsets  (more than kRsDirect tiles) exclusive sums of every digit's
//                 counts over the tiles, and the digits' totals
//   k_rs_scatter  rank of each pair within its tile: a warp ranks its pairs
//                 32 at a time by __match_any_sync on the digit, counting in
//                 its own row of shared memory, so the block meets twice a
//                 tile and not per round; with few tiles every block sums the
//                 counts of the tiles before it itself.
//
// Bound: launch latency at the sizes the library sorts (10^4 to 10^6 pairs).
// A pass was a histogram, a five-launch scan and a scatter that met per round
// of 256 pairs, over 32-bit keys (two sorts for a longer key): 17 us and 7
// launches a pass at 40k pairs, now 8.5 us and 2, and as many passes as the
// key has bytes (3 instead of 8 for a list of 128^3 voxels).
#include <algorithm>

#include "sort_reduce.hpp"

namespace vlr {
namespace {

constexpr int kRsThreads = 256;
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRsItems = 8;                        // pairs per thread
constexpr int kRsTile = kRsThreads * kRsItems;
constexpr int kRsWarpPairs = 32 * kRsItems;        // consecutive pairs of a warp
// Tiles up to which a scatter block sums the earlier tiles' counts itself:
// each thread reads one count per tile, so the sum grows with the tiles (the
// scatter takes 5.1 us at 20 tiles, 8.9 us at 147) while the separate kernel
// costs a launch of its own.
constexpr int kRsDirect = 160;
constexpr int kRsCols = 8;                         // digits per block of k_rs_offsets
constexpr int kRsRows = 128;                       // tile ranges per digit there

template <typename K>
__global__ void __launch_bounds__(kRsThreads) k_rs_hist(const K* __restrict__ keys, int n, int shift, unsigned dmask,
                                                       int* __restrict__ hist) {
    __shared__ int s_h[256];
    const int tile = blockIdx.x;
    s_h[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kRsItems; ++i) {
        const int p = tile * kRsTile + i * kRsThreads + threadIdx.x;
        if (p < n) atomicAdd(&s_h[(unsigned)(keys[p] >> shift) & dmask], 1);
    }
    __syncthreads();
    hist[tile * 256 + threadIdx.x] = s_h[threadIdx.x];
}

// hist[t][d] -> sum over tiles before t; tot[d] = sum over all tiles.  A block
// takes kRsCols digits, kRsRows threads a digit, each a range of tiles.
__global__ void __launch_bounds__(kRsCols* kRsRows) k_rs_offsets(int* __restrict__ hist, int n_tiles,
                                                                int* __restrict__ tot) {
    __shared__ int s_sum[kRsRows][kRsCols];
    const int c = threadIdx.x % kRsCols, r = threadIdx.x / kRsCols;
    const int d = blockIdx.x * kRsCols + c;
    const int per = (n_tiles + kRsRows - 1) / kRsRows;
    const int t0 = min(r * per, n_tiles), t1 = min(t0 + per, n_tiles);
    int s = 0;
    for (int t = t0; t < t1; ++t) s += hist[t * 256 + d];
    s_sum[r][c] = s;
    __syncthreads();
    if (r == 0) {
        int run = 0;
        for (int q = 0; q < kRsRows; ++q) {
            const int v = s_sum[q][c];
            s_sum[q][c] = run;
            run += v;
        }
        tot[d] = run;
    }
    __syncthreads();
    int run = s_sum[r][c];
    for (int t = t0; t < t1; ++t) {
        const int v = hist[t * 256 + d];
        hist[t * 256 + d] = run;
        run += v;
    }
}

template <typename K>
__global__ void __launch_bounds__(kRsThreads) k_rs_scatter(const K* __restrict__ keys_in,
                                                          const unsigned* __restrict__ vals_in, int n, int shift,
                                                          unsigned dmask, int n_tiles, const int* __restrict__ hist,
                                                          const int* __restrict__ tot, K* __restrict__ keys_out,
                                                          unsigned* __restrict__ vals_out) {
    __shared__ int s_c[kRsWarps][256];  // a warp's digit counts, then its first positions
    __shared__ int s_w[kRsWarps];
    const int tile = blockIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < kRsWarps; ++q) s_c[q][threadIdx.x] = 0;
    // this thread's digit: pairs of the digit in the tiles before, and in all
    int before = 0, all = 0;
    if (tot) {
        before = hist[tile * 256 + threadIdx.x];
        all = tot[threadIdx.x];
    } else {
#pragma unroll 8
        for (int t = 0; t < n_tiles; ++t) {
            const int v = hist[t * 256 + threadIdx.x];
            all += v;
            before += t < tile ? v : 0;
        }
    }
    __syncthreads();
    const int p0 = tile * kRsTile + w * kRsWarpPairs + lane;
    K key[kRsItems];
    unsigned val[kRsItems];
    int rank[kRsItems];
#pragma unroll
    for (int i = 0; i < kRsItems; ++i) {
        const int p = p0 + 32 * i;
        key[i] = p < n ? keys_in[p] : (K)0;
        val[i] = p < n ? vals_in[p] : 0u;
    }
#pragma unroll
    for (int i = 0; i < kRsItems; ++i) {
        const bool valid = p0 + 32 * i < n;
        const unsigned digit = (unsigned)(key[i] >> shift) & dmask;
        const unsigned peers = __match_any_sync(0xffffffffu, valid ? digit : 256u);
        const unsigned lower = peers & ((1u << lane) - 1u);
        rank[i] = valid ? s_c[w][digit] + __popc(lower) : 0;
        __syncwarp();
        if (valid && !lower) s_c[w][digit] += __popc(peers);
        __syncwarp();
    }
    // first position of the digits: exclusive sum of their totals over the block
    int x = all;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_w[w] = x;
    __syncthreads();
    int base = x - all + before;
    for (int q = 0; q < w; ++q) base += s_w[q];
#pragma unroll
    for (int q = 0; q < kRsWarps; ++q) {
        const int c = s_c[q][threadIdx.x];
        s_c[q][threadIdx.x] = base;
        base += c;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kRsItems; ++i)
        if (p0 + 32 * i < n) {
            const int dst = s_c[w][(unsigned)(key[i] >> shift) & dmask] + rank[i];
            keys_out[dst] = key[i];
            vals_out[dst] = val[i];
        }
}

int tiles_of(int n) { return (int)(((long long)n + kRsTile - 1) / kRsTile); }

template <typename K>
int sort_impl(vlr_ctx* ctx, K* keys, unsigned* vals, int n, int bits, void* scratch, K** keys_out,
              unsigned** vals_out) {
    cudaStream_t st = ctx->stream;
    *keys_out = keys;
    *vals_out = vals;
    if (n <= 0 || bits <= 0) return VLR_OK;
    const int tiles = tiles_of(n);
    K* kb = static_cast<K*>(scratch);
    unsigned* vb = reinterpret_cast<unsigned*>(kb + n);
    int* hist = reinterpret_cast<int*>(vb + n);
    int* tot = tiles > kRsDirect ? hist + (size_t)256 * tiles : nullptr;
    K* ka = keys;
    unsigned* va = vals;
    const int passes = (bits + 7) / 8, width = (bits + passes - 1) / passes;
    const unsigned dmask = (1u << width) - 1u;
    for (int p = 0; p < passes; ++p) {
        VLR_TIMED(ctx, "k_rs_hist", k_rs_hist<K><<<tiles, kRsThreads, 0, st>>>(ka, n, p * width, dmask, hist));
        if (tot)
            VLR_TIMED(ctx, "k_rs_offsets",
                      k_rs_offsets<<<256 / kRsCols, kRsCols * kRsRows, 0, st>>>(hist, tiles, tot));
        VLR_TIMED(ctx, "k_rs_scatter", k_rs_scatter<K><<<tiles, kRsThreads, 0, st>>>(ka, va, n, p * width, dmask,
                                                                                    tiles, hist, tot, kb, vb));
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    VLR_CUDA(ctx, cudaGetLastError());
    *keys_out = ka;
    *vals_out = va;
    return VLR_OK;
}

}  // namespace

size_t radix_scratch_bytes(int n, int key_bytes) {
    return (size_t)std::max(n, 0) * (key_bytes + 4) + ((size_t)256 * tiles_of(std::max(n, 0)) + 256) * 4 + 256;
}

int radix_sort(vlr_ctx* ctx, unsigned* keys, unsigned* vals, int n, int bits, void* scratch, unsigned** keys_out,
               unsigned** vals_out) {
    return sort_impl(ctx, keys, vals, n, bits, scratch, keys_out, vals_out);
}

int radix_sort(vlr_ctx* ctx, uint64_t* keys, unsigned* vals, int n, int bits, void* scratch, uint64_t** keys_out,
               unsigned** vals_out) {
    return sort_impl(ctx, keys, vals, n, bits, scratch, keys_out, vals_out);
}

}  // namespace vlr
