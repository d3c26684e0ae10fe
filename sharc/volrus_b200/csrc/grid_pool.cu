// Leaf-pool management: allocation, hash index, 27-neighbour table, scan and
// order-preserving compaction.  These replace the reference's pointer-chasing
// topology (RootNode HashMap -> InternalNode 16^3 -> boxed LeafNode,
// src/tree/root.rs:55-72, src/tree/internal.rs:88-143) with flat device
// arrays that the stencil kernels index directly.
#include <algorithm>
#include <pthread.h>
#include <unistd.h>

#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "vlr_host.hpp"

namespace vlr {

int set_error(vlr_ctx* ctx, int code, const std::string& msg) {
    if (ctx) ctx->last_error = msg;
    return code;
}

int check_cuda(vlr_ctx* ctx, cudaError_t e, const char* what) {
    cudaGetLastError();  // reported here: the next launch's check must not find it again
    int code = (e == cudaErrorMemoryAllocation) ? VLR_ERR_NOMEM : VLR_ERR_CUDA;
    return set_error(ctx, code, std::string(what) + ": " + cudaGetErrorString(e));
}

size_t value_bytes(int kind) { return kind == VLR_KIND_F16_VOXEL ? 2 : 4; }

int ctx_scratch(vlr_ctx* ctx, size_t bytes, void** out) {
    if (bytes > ctx->scratch_bytes) {
        if (ctx->scratch) {
            cudaStreamSynchronize(ctx->stream);
            cudaFree(ctx->scratch);
            ctx->scratch = nullptr;
            ctx->scratch_bytes = 0;
        }
        size_t want = std::max<size_t>(bytes, 1 << 20);
        VLR_CUDA(ctx, cudaMalloc(&ctx->scratch, want));
        ctx->scratch_bytes = want;
    }
    *out = ctx->scratch;
    return VLR_OK;
}

int read_int(vlr_ctx* ctx, const int* d_ptr, int* out) {
    int* h = (int*)ctx->pinned;
    VLR_CUDA(ctx, cudaMemcpyAsync(h, d_ptr, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    VLR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *out = *h;
    return VLR_OK;
}

static cudaEvent_t timer_event(vlr_ctx* ctx) {
    auto& t = ctx->timer;
    if (!t.free_events.empty()) {
        cudaEvent_t e = t.free_events.back();
        t.free_events.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
}

void timer_begin(vlr_ctx* ctx, const char* name) {
    auto& t = ctx->timer;
    if (!t.enabled) return;
    vlr_kernel_timer::Pending p{name, timer_event(ctx), timer_event(ctx)};
    cudaEventRecord(p.a, ctx->stream);
    t.pending.push_back(p);
}

void timer_end(vlr_ctx* ctx) {
    auto& t = ctx->timer;
    if (!t.enabled || t.pending.empty()) return;
    cudaEventRecord(t.pending.back().b, ctx->stream);
}

int timer_collect(vlr_ctx* ctx) {
    auto& t = ctx->timer;
    if (t.pending.empty()) return VLR_OK;
    VLR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (auto& p : t.pending) {
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, p.a, p.b);
        bool found = false;
        for (auto& kv : t.totals)
            if (kv.first == p.name) {
                kv.second.first += ms;
                kv.second.second += 1;
                found = true;
                break;
            }
        if (!found) t.totals.push_back({std::string(p.name), {(double)ms, 1ll}});
        t.free_events.push_back(p.a);
        t.free_events.push_back(p.b);
    }
    t.pending.clear();
    return VLR_OK;
}

// Copies between pageable host memory and the device.  A fresh result array is
// untouched memory, so writing it costs a page fault per 4 KB (or the clearing
// of 2 MB pages) beside the copy itself: a few GB/s for one thread, against
// 55 GB/s of the link.  The copy is cut into kCopyShares contiguous shares, so
// that threads do not fault the same page; each share passes through two pinned
// buffers of its own, one filled or emptied while the DMA of the other runs.
// The calling thread takes the first share, the context's copy threads the
// others.  7.3 MB into a fresh array: 1550-2200 us by one thread through two
// buffers, 760-970 us here; 300k particles there and back (16 MB each way)
// 6.9 -> 1.5 ms with the caller's own copy gone (2.1 ms when the threads split
// every chunk instead, 2.8 ms when eight did).  Into memory that is in use the
// driver's copy and this meet at 2 MB (152 and 157 us), at 3 MB 210 and 175 us,
// at 7.3 MB 477 and 251 us: the line is at 3 MB.
constexpr size_t kCopyChunk = 1u << 20;
constexpr int kCopyShares = 4;
constexpr size_t kCopyMin = 3u << 20;  // below, one driver call

static bool host_pageable(const void* p) {
    cudaPointerAttributes at{};
    const bool known = cudaPointerGetAttributes(&at, p) == cudaSuccess && at.type != cudaMemoryTypeUnregistered;
    cudaGetLastError();  // a pageable pointer may leave an error behind on older drivers
    return !known;
}

// One share, through pinned buffers b[0], b[1] with events ev[0], ev[1].
static cudaError_t copy_share(char* host, char* dev, size_t bytes, bool up, char* b, cudaEvent_t* ev, cudaStream_t st) {
    const size_t n = (bytes + kCopyChunk - 1) / kCopyChunk;
    cudaError_t e = cudaSuccess;
    auto length = [&](size_t k) { return std::min(kCopyChunk, bytes - k * kCopyChunk); };
    auto send = [&](size_t k) {
        char* d = dev + k * kCopyChunk;
        char* r = b + (k & 1) * kCopyChunk;
        e = up ? cudaMemcpyAsync(d, r, length(k), cudaMemcpyHostToDevice, st)
               : cudaMemcpyAsync(r, d, length(k), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(ev[k & 1], st);
    };
    for (size_t k = 0; !up && k < std::min<size_t>(n, 2) && e == cudaSuccess; ++k) send(k);
    for (size_t k = 0; k < n && e == cudaSuccess; ++k) {
        if (!up || k >= 2) e = cudaEventSynchronize(ev[k & 1]);  // landed (down), or its buffer is free (up)
        if (e != cudaSuccess) break;
        char* h = host + k * kCopyChunk;
        char* r = b + (k & 1) * kCopyChunk;
        std::memcpy(up ? r : h, up ? h : r, length(k));
        if (up) send(k);
        else if (k + 2 < n) send(k + 2);
    }
    for (size_t k = n > 2 ? n - 2 : 0; up && k < n && e == cudaSuccess; ++k) e = cudaEventSynchronize(ev[k & 1]);
    return e;
}

// The threads beside the caller, kept with the context from its first large
// copy: started and joined per copy they cost 30-50 us, and what they allocate
// in the caller's heap made glibc give its top back to the system and fault it
// in again on each call (meshing 2.1 -> 2.9 ms).  They are joined when the
// context goes (idle by then), so none of them is in the library's code after
// that; a forked child, which has no such threads, leaves the state be.
struct CopyThreads {
    std::mutex m;
    std::condition_variable go, idle;
    void (*job)(void*, int) = nullptr;
    void* arg = nullptr;
    unsigned long turn = 0;
    int running = 0;  // threads still at the current job
    bool quit = false;
    const pid_t owner = getpid();
    std::vector<std::thread> threads;
};

static void copy_thread(CopyThreads* s, int t, int device) {
    pthread_setname_np(pthread_self(), "vlr-copy");
    const bool ok = cudaSetDevice(device) == cudaSuccess;
    std::unique_lock<std::mutex> lock(s->m);
    for (unsigned long seen = 0;;) {
        s->go.wait(lock, [&] { return s->quit || s->turn != seen; });
        if (s->quit) return;
        seen = s->turn;
        lock.unlock();
        s->job(s->arg, ok ? t : -t);
        lock.lock();
        if (--s->running == 0) s->idle.notify_one();
    }
}

void copy_threads_stop(vlr_ctx* ctx) {
    CopyThreads* s = ctx->copy_threads;
    ctx->copy_threads = nullptr;
    if (!s || s->owner != getpid()) return;
    {
        std::lock_guard<std::mutex> lock(s->m);
        s->quit = true;
    }
    s->go.notify_all();
    for (std::thread& t : s->threads) t.join();
    delete s;
}

static int staged_copy(vlr_ctx* ctx, char* host, char* dev, size_t bytes, bool up) {
    cudaStream_t st = ctx->stream;
    if (!ctx->stage) {
        VLR_CUDA(ctx, cudaMallocHost(&ctx->stage, 2 * kCopyShares * kCopyChunk));
        for (cudaEvent_t& e : ctx->stage_ev) VLR_CUDA(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    if (!ctx->copy_threads) {
        try {
            CopyThreads* s = ctx->copy_threads = new CopyThreads;
            s->threads.reserve(kCopyShares - 1);
            for (int t = 1; t < kCopyShares; ++t) s->threads.emplace_back(copy_thread, s, t, ctx->device);
        } catch (...) {  // no more threads: the caller takes the shares that are left
        }
    }
    const size_t step = ((bytes + kCopyShares - 1) / kCopyShares + 4095) & ~(size_t)4095;
    cudaError_t err[kCopyShares] = {};
    auto share = [&](int t) {
        const size_t a = std::min(bytes, step * std::abs(t)), z = std::min(bytes, a + step);
        if (t < 0) err[-t] = cudaErrorInvalidDevice;  // the thread could not take the context's device
        else if (a < z)
            err[t] = copy_share(host + a, dev + a, z - a, up, static_cast<char*>(ctx->stage) + 2 * t * kCopyChunk,
                                ctx->stage_ev + 2 * t, st);
    };
    CopyThreads* pool = ctx->copy_threads;
    const int others = pool && pool->owner == getpid() ? (int)pool->threads.size() : 0;
    if (others) {
        std::lock_guard<std::mutex> lock(pool->m);
        pool->job = [](void* f, int t) { (*static_cast<decltype(share)*>(f))(t); };
        pool->arg = &share;
        pool->running = others;
        ++pool->turn;
    }
    if (others) pool->go.notify_all();
    share(0);
    for (int t = others + 1; t < kCopyShares; ++t) share(t);
    if (others) {
        std::unique_lock<std::mutex> lock(pool->m);
        pool->idle.wait(lock, [&] { return pool->running == 0; });
    }
    for (const cudaError_t e : err)
        if (e != cudaSuccess) return check_cuda(ctx, e, "staged copy");
    return VLR_OK;
}

int d2h_copy(vlr_ctx* ctx, void* dst, const void* src, size_t bytes) {
    if (!bytes) return VLR_OK;
    if (bytes >= kCopyMin && host_pageable(dst))
        return staged_copy(ctx, static_cast<char*>(dst), static_cast<char*>(const_cast<void*>(src)), bytes, false);
    VLR_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    VLR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return VLR_OK;
}

int h2d_copy(vlr_ctx* ctx, void* dst, const void* src, size_t bytes) {
    if (!bytes) return VLR_OK;
    if (bytes >= kCopyMin && host_pageable(src))
        return staged_copy(ctx, static_cast<char*>(const_cast<void*>(src)), static_cast<char*>(dst), bytes, true);
    VLR_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
    return VLR_OK;
}

// The status of error word e, reported as `what`; clears the word on the device.
static int map_device_errors(vlr_ctx* ctx, unsigned e, const char* what) {
    if (!e) return VLR_OK;
    VLR_CUDA(ctx, cudaMemsetAsync(ctx->d_errword, 0, sizeof(unsigned), ctx->stream));
    std::string m = std::string(what) + ": device reported";
    int code = VLR_ERR_CUDA;
    if (e & kErrReach) { m += " backtrace outside the staged neighbourhood;"; code = VLR_ERR_REACH; }
    if (e & kErrExtent) { m += " leaf outside the hashable extent;"; code = VLR_ERR_EXTENT; }
    if (e & kErrCapacity) { m += " leaf capacity exceeded;"; code = VLR_ERR_CAPACITY; }
    if (e & kErrHashFull) { m += " hash table full;"; code = VLR_ERR_CAPACITY; }
    if (e & kErrTimeout) { m += " bounded wait timed out;"; code = VLR_ERR_TIMEOUT; }
    if (e & kErrInput) {
        m += " device input failed a check (a leaf origin off the 8-voxel lattice, a leaf listed twice or a list "
             "position out of range);";
        code = VLR_ERR_INVALID;
    }
    return set_error(ctx, code, m);
}

int consume_device_errors(vlr_ctx* ctx, const char* what) {
    unsigned* h = (unsigned*)ctx->pinned;
    VLR_CUDA(ctx, cudaMemcpyAsync(h, ctx->d_errword, sizeof(unsigned), cudaMemcpyDeviceToHost, ctx->stream));
    VLR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return map_device_errors(ctx, *h, what);
}

int read_int_checked(vlr_ctx* ctx, const int* d_ptr, int* out, const char* what) {
    unsigned* h = (unsigned*)ctx->pinned;
    VLR_CUDA(ctx, cudaMemcpyAsync(h + 1, d_ptr, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    VLR_CUDA(ctx, cudaMemcpyAsync(h, ctx->d_errword, sizeof(unsigned), cudaMemcpyDeviceToHost, ctx->stream));
    VLR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *out = (int)h[1];
    return map_device_errors(ctx, h[0], what);
}

void grid_free_arrays(vlr_grid* g) {
    if (g->block) {
        // stream-ordered: later work on the context stream may reuse the memory
        if (g->ctx && g->ctx->stream) cudaFreeAsync(g->block, g->ctx->stream);
        else cudaFree(g->block);
    }
    g->block = nullptr;
    g->origin = nullptr;
    g->mask = nullptr;
    g->values = nullptr;
    g->nbr = nullptr;
    g->hkey = nullptr;
    g->hval = nullptr;
    g->hcap = 0;
    g->cap = 0;
}

static int next_pow2(long long v) {
    int p = 64;
    while ((long long)p < v && p < (1 << 30)) p <<= 1;
    return p;
}

// The grid's arrays in one allocation from the context's pool (256-byte
// aligned pieces): a step that makes a new grid costs no synchronising
// cudaMalloc.
int grid_alloc(vlr_ctx* ctx, vlr_grid* g, int cap) {
    grid_free_arrays(g);
    if (!g->ctx) g->ctx = ctx;
    int c = std::max(cap, 1);
    size_t vb = value_bytes(g->kind);
    g->hcap = next_pow2(2ll * c);
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t s_origin = up(sizeof(int4) * c), s_mask = up(sizeof(uint64_t) * 8 * c),
                 s_values = up(vb * kLeafVoxels * c), s_nbr = up(sizeof(int) * kNbr * (size_t)c),
                 s_hkey = up(sizeof(uint64_t) * g->hcap), s_hval = up(sizeof(int) * g->hcap);
    char* p = nullptr;
    VLR_CUDA(ctx, cudaMallocFromPoolAsync((void**)&p, s_origin + s_mask + s_values + s_nbr + s_hkey + s_hval, ctx->pool,
                                          ctx->stream));
    g->block = p;
    g->origin = (int4*)p;
    p += s_origin;
    g->mask = (uint64_t*)p;
    p += s_mask;
    g->values = p;
    p += s_values;
    g->nbr = (int*)p;
    p += s_nbr;
    g->hkey = (uint64_t*)p;
    p += s_hkey;
    g->hval = (int*)p;
    g->cap = c;
    return VLR_OK;
}

int choose_base(vlr_ctx* ctx, const int32_t* origins, size_t n, long long base[3], int* box) {
    if (n == 0) {
        if (box) std::fill(box, box + 6, 0);
        base[0] = base[1] = base[2] = -kKeyHalf;
        return VLR_OK;
    }
    for (int a = 0; a < 3; ++a) {
        long long lo = LLONG_MAX, hi = LLONG_MIN;
        for (size_t i = 0; i < n; ++i) {
            long long l = (long long)(origins[3 * i + a] >> 3);
            lo = std::min(lo, l);
            hi = std::max(hi, l);
        }
        if (hi - lo >= (1ll << kKeyBits) - 2)
            return set_error(ctx, VLR_ERR_EXTENT, "grid spans more than 2^24 voxels along an axis");
        base[a] = (lo + hi) / 2 - kKeyHalf;
        if (box) {
            box[a] = (int)lo;
            box[3 + a] = (int)hi;
        }
    }
    return VLR_OK;
}

// ---------------------------------------------------------------- kernels

// Empty keys, values that every inserted slot is below (atomicMin), and the
// duplicate flag.
__global__ void k_hash_clear(uint64_t* key, int* val, int cap, int* dup) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += gridDim.x * blockDim.x) {
        key[i] = kEmptyKey;
        val[i] = INT_MAX;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *dup = 0;
}

__global__ void k_hash_insert(const int4* origin, int n, uint64_t* hkey, int* hval, int hcap, long long b0,
                              long long b1, long long b2, unsigned* err) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    long long base[3] = {b0, b1, b2};
    int4 o = origin[i];
    uint64_t key = pack_key(o.x >> 3, o.y >> 3, o.z >> 3, base);
    if (key == kEmptyKey) {
        atomicOr(err, kErrExtent);
        return;
    }
    uint32_t m = (uint32_t)hcap - 1u;
    uint32_t p = (uint32_t)mix64(key) & m;
    for (int probe = 0; probe < hcap; ++probe) {
        unsigned long long prev =
            atomicCAS((unsigned long long*)&hkey[p], (unsigned long long)kEmptyKey, (unsigned long long)key);
        if (prev == kEmptyKey || prev == key) {
            // Duplicates keep the smallest slot (deterministic).
            atomicMin(&hval[p] , i) ;
            return;
        }
        p = (p + 1u) & m;
    }
    atomicOr(err, kErrHashFull);
}

__global__ void k_nbr_build(const int4* origin, int n, const uint64_t* hkey, const int* hval, int hcap, long long b0,
                            long long b1, long long b2, int* nbr, int* dup_flag) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    int i = t / kNbr, d = t % kNbr;
    if (i >= n) return;
    HashView h{hkey, hval, hcap, {b0, b1, b2}};
    int4 o = origin[i];
    int dx = d / 9 - 1, dy = (d / 3) % 3 - 1, dz = d % 3 - 1;
    int s = hash_find_leaf(h, (long long)(o.x >> 3) + dx, (long long)(o.y >> 3) + dy, (long long)(o.z >> 3) + dz);
    nbr[i * kNbr + d] = s;
    if (d == 13 && s != i) atomicOr(dup_flag, 1);  // a duplicate origin maps to another slot
}

int grid_index(vlr_ctx* ctx, vlr_grid* g) {
    int hc = g->hcap;
    int thr = 256;
    int blocks = std::min((hc + thr - 1) / thr, ctx->sm_count * 8);
    void* sp;
    int rc = ctx_scratch(ctx, sizeof(int), &sp);
    if (rc) return rc;
    int* dup = (int*)sp;
    k_hash_clear<<<blocks, thr, 0, ctx->stream>>>(g->hkey, g->hval, hc, dup);
    if (g->n > 0) {
        k_hash_insert<<<(g->n + thr - 1) / thr, thr, 0, ctx->stream>>>(g->origin, g->n, g->hkey, g->hval, hc,
                                                                     g->base[0], g->base[1], g->base[2],
                                                                     ctx->d_errword);
        long long tot = (long long)g->n * kNbr;
        k_nbr_build<<<(unsigned)((tot + thr - 1) / thr), thr, 0, ctx->stream>>>(
            g->origin, g->n, g->hkey, g->hval, hc, g->base[0], g->base[1], g->base[2], g->nbr, dup);
    }
    VLR_CUDA(ctx, cudaGetLastError());
    int h_dup = 0;
    rc = read_int_checked(ctx, dup, &h_dup, "grid index");
    if (h_dup) return set_error(ctx, VLR_ERR_INVALID, "duplicate leaf origin");
    return rc;
}

// ------------------------------------------------------------------ scan

// Exclusive scan in tiles of 8192 (1024 threads, 8 consecutive values each).
// More than one tile: k_scan_sums first writes the tiles' sums, and each block
// of k_scan_tiles adds up the sums of the tiles before its own, so no block
// waits on another and nothing is allocated per level.  A scan was two
// launches, five from 1025 values up (about 8 us of launches and gaps); it is
// one up to 8192 values (2.2 us) and two beyond.
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

// Block-wide inclusive scan of one int per thread; *total = the block's sum.
__device__ inline int block_incl_scan(int v, int* warp_sums, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
        int s = warp_sums[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        warp_sums[lane] = s;
    }
    __syncthreads();
    *total = warp_sums[31];
    return x + (w ? warp_sums[w - 1] : 0);
}

__global__ void __launch_bounds__(kScanThreads) k_scan_sums(const int* __restrict__ in, long long n, int* __restrict__ sums) {
    __shared__ int ws[32];
    const size_t base = (size_t)blockIdx.x * kScanTile;
    int v = 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        const size_t i = base + q * kScanThreads + threadIdx.x;
        if (i < (size_t)n) v += in[i];
    }
    int tot;
    block_incl_scan(v, ws, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const int* in, int* out, long long n,
                                                            const int* __restrict__ sums, int* total) {
    __shared__ int ws[32];
    int before = 0;
    if (blockIdx.x > 0) {  // one tile: sums is null
        int v = 0;
        for (int t = threadIdx.x; t < (int)blockIdx.x; t += kScanThreads) v += sums[t];
        block_incl_scan(v, ws, &before);
        __syncthreads();
    }
    const size_t i0 = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
    int v[kScanItems], s = 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        v[q] = i0 + q < (size_t)n ? in[i0 + q] : 0;
        s += v[q];
    }
    int tot;
    int run = before + block_incl_scan(s, ws, &tot) - s;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        if (i0 + q < (size_t)n) out[i0 + q] = run;
        run += v[q];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total = before + tot;
}

// Exclusive scan of n ints on the context stream; *d_total (device) = their sum.
int scan_exclusive(vlr_ctx* ctx, const int* d_in, int* d_out, long long n, int* d_total) {
    if (n <= 0) {
        VLR_CUDA(ctx, cudaMemsetAsync(d_total, 0, sizeof(int), ctx->stream));
        return VLR_OK;
    }
    const int nb = (int)((n + kScanTile - 1) / kScanTile);
    int* sums = nullptr;
    if (nb > 1) {
        VLR_CUDA(ctx, cudaMallocFromPoolAsync(&sums, sizeof(int) * nb, ctx->pool, ctx->stream));
        k_scan_sums<<<nb, kScanThreads, 0, ctx->stream>>>(d_in, n, sums);
    }
    k_scan_tiles<<<nb, kScanThreads, 0, ctx->stream>>>(d_in, d_out, n, sums, d_total);
    VLR_CUDA(ctx, cudaGetLastError());
    if (sums) VLR_CUDA(ctx, cudaFreeAsync(sums, ctx->stream));
    return VLR_OK;
}

// ------------------------------------------------------------ compaction

template <typename T>
__global__ void k_compact_leaves(int n, const int* flags, const int* pos, const int4* o_in, const uint64_t* m_in,
                                 const T* v_in, int4* o_out, uint64_t* m_out, T* v_out) {
    int i = blockIdx.x;
    if (i >= n || !flags[i]) return;
    int j = pos[i];
    if (threadIdx.x == 0) o_out[j] = o_in[i];
    if (threadIdx.x < 8) m_out[(size_t)j * 8 + threadIdx.x] = m_in[(size_t)i * 8 + threadIdx.x];
    const uint4* src = (const uint4*)(v_in + (size_t)i * kLeafVoxels);
    uint4* dst = (uint4*)(v_out + (size_t)j * kLeafVoxels);
    constexpr int kVec = kLeafVoxels * sizeof(T) / 16;
    for (int t = threadIdx.x; t < kVec; t += blockDim.x) dst[t] = src[t];
}

int grid_compact(vlr_ctx* ctx, vlr_grid* g, const int* d_flags, const char* what, const vlr_grid* index) {
    if (g->n == 0) return VLR_OK;
    int* pos = nullptr;
    VLR_CUDA(ctx, cudaMallocFromPoolAsync(&pos, sizeof(int) * (g->n + 1), ctx->pool, ctx->stream));
    vlr_grid tmp;
    tmp.ctx = ctx;
    tmp.kind = g->kind;
    int total = 0;
    auto run = [&]() -> int {
        int rc = scan_exclusive(ctx, d_flags, pos, g->n, pos + g->n);
        if (!rc) rc = read_int_checked(ctx, pos + g->n, &total, what);
        if (rc || total == g->n) return rc;
        rc = grid_alloc(ctx, &tmp, std::max(total, 1));
        if (rc) return rc;
        if (g->kind == VLR_KIND_F16_VOXEL)
            k_compact_leaves<__half><<<g->n, 64, 0, ctx->stream>>>(g->n, d_flags, pos, g->origin, g->mask,
                                                                  (const __half*)g->values, tmp.origin, tmp.mask,
                                                                  (__half*)tmp.values);
        else
            k_compact_leaves<float><<<g->n, 128, 0, ctx->stream>>>(g->n, d_flags, pos, g->origin, g->mask,
                                                                  (const float*)g->values, tmp.origin, tmp.mask,
                                                                  (float*)tmp.values);
        VLR_CUDA(ctx, cudaGetLastError());
        return VLR_OK;
    };
    const int rc = run();
    cudaFreeAsync(pos, ctx->stream);
    if (rc) {
        grid_free_arrays(&tmp);
        return rc;
    }
    if (total == g->n) {
        if (!index) return VLR_OK;
        if (index->hcap != g->hcap) return grid_index(ctx, g);
        VLR_CUDA(ctx, cudaMemcpyAsync(g->nbr, index->nbr, sizeof(int) * kNbr * (size_t)g->n, cudaMemcpyDeviceToDevice,
                                      ctx->stream));
        VLR_CUDA(ctx, cudaMemcpyAsync(g->hkey, index->hkey, sizeof(uint64_t) * g->hcap, cudaMemcpyDeviceToDevice,
                                      ctx->stream));
        VLR_CUDA(ctx, cudaMemcpyAsync(g->hval, index->hval, sizeof(int) * g->hcap, cudaMemcpyDeviceToDevice,
                                      ctx->stream));
        return VLR_OK;
    }
    std::swap(g->block, tmp.block);
    std::swap(g->origin, tmp.origin);
    std::swap(g->mask, tmp.mask);
    std::swap(g->values, tmp.values);
    std::swap(g->nbr, tmp.nbr);
    std::swap(g->hkey, tmp.hkey);
    std::swap(g->hval, tmp.hval);
    std::swap(g->hcap, tmp.hcap);
    std::swap(g->cap, tmp.cap);
    grid_free_arrays(&tmp);  // stream-ordered: after the copy
    g->n = total;
    return grid_index(ctx, g);
}

}  // namespace vlr
