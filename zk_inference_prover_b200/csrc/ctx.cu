// Context lifetime, device memory helpers, the twiddle tower and small utilities.
#include <climits>
#include <cstdarg>
#include <unordered_map>
#include <utility>
#include <vector>

#include "common.cuh"
#include "fri_tail.hpp"
#include "side_stream.hpp"
#include "gather_blocks.hpp"

namespace zk {

int set_error(zkb_ctx* ctx, int code, const char* fmt, ...) {
    if (ctx) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(ctx->err, sizeof(ctx->err), fmt, ap);
        va_end(ap);
    }
    return code;
}

// The ring is used from its start again: earlier slots may still be in flight, so drain the stream, and forget what they held.
static int stage_wrap(zkb_ctx* ctx) {
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (ctx->other_stream) ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->other_stream));
    ctx->ring_pos = 0;
    for (auto& t : ctx->staged) t.n = 0;
    return ZKB_OK;
}

int stage_reserve(zkb_ctx* ctx, size_t slots) {
    if (slots > ctx->ring_cap) return set_error(ctx, ZKB_EINVAL, "stage_reserve: the tables of one call (%zu slots) exceed the staging ring", slots);
    return ctx->ring_pos + slots > ctx->ring_cap ? stage_wrap(ctx) : ZKB_OK;
}

// Device memory of a proof's small arrays (tree layers, FRI layers, coordinate columns): a proof allocates hundreds of them, and
// the stream-ordered allocator takes 0.6-0.8 us of host time for each allocation and each release (716 us of a ten-column proof
// were 230 of them). Blocks of up to 2^MAX_LOG bytes are rounded up to a power of two and kept per size when they are freed,
// up to KEPT_BYTES in all; they go back to the pool beyond that, when an allocation fails and with the context. A context's work is
// ordered on one stream, so a kept block is as reusable as one the pool would hand out on that stream.
struct BlockCache {
    static constexpr int MIN_LOG = 8, MAX_LOG = 24;
    static constexpr size_t KEPT_BYTES = (size_t)256 << 20;
    std::unordered_map<void*, int> live;  // block -> log2 of its size
    std::vector<void*> kept[MAX_LOG + 1];
    size_t kept_bytes = 0;
    static int log_of(size_t bytes) {
        int l = MIN_LOG;
        while (((size_t)1 << l) < bytes) l++;
        return l;
    }
    void release(cudaStream_t stream) {
        for (auto& k : kept) {
            for (void* p : k) cudaFreeAsync(p, stream);
            k.clear();
        }
        kept_bytes = 0;
    }
};

// Copies the table into the ring, unless the same table is still there from an earlier call: a tree's columns are named by the
// interpolation, the extension, the hashing, the sampling, the numerators and the decommitment in turn, and a copy of a table in
// between two kernels costs 2-3 us of the stream. (What was handed out stays in place until the ring is used from its start again: an
// operator with several tables has their room reserved first.)
static const zkb_ctx::StagedTable* find_staged(const zkb_ctx* ctx, const void* const* h_ptrs, size_t n) {
    for (const auto& t : ctx->staged)
        if (t.n == n && ctx->h_ring[t.pos] == h_ptrs[0] && !memcmp(ctx->h_ring + t.pos, h_ptrs, n * sizeof(void*))) return &t;
    return nullptr;
}
static void remember_staged(zkb_ctx* ctx, size_t pos, size_t n) {
    ctx->staged[ctx->staged_next] = {pos, n};
    ctx->staged_next = (ctx->staged_next + 1) % zkb_ctx::STAGED_TABLES;
}
int stage_ptrs(zkb_ctx* ctx, const void* const* h_ptrs, int n, void*** out) {
    if (n < 0 || (size_t)n > ctx->ring_cap) return set_error(ctx, ZKB_EINVAL, "stage_ptrs: %d pointers exceed the staging ring", n);
    if (n == 0) { *out = ctx->d_ring; return ZKB_OK; }
    if (const auto* t = find_staged(ctx, h_ptrs, (size_t)n)) {
        *out = ctx->d_ring + t->pos;
        return ZKB_OK;
    }
    if (ctx->ring_pos + (size_t)n > ctx->ring_cap) {
        if (int rc = stage_wrap(ctx)) return rc;
    }
    void** h = ctx->h_ring + ctx->ring_pos;
    void** d = ctx->d_ring + ctx->ring_pos;
    memcpy(h, h_ptrs, (size_t)n * sizeof(void*));
    ZKB_CUDA(ctx, cudaMemcpyAsync(d, h, (size_t)n * sizeof(void*), cudaMemcpyHostToDevice, ctx->stream));
    if (!ctx->on_side) remember_staged(ctx, ctx->ring_pos, (size_t)n);  // a table copied on the side is not there yet for the work outside
    ctx->ring_pos += (size_t)n;
    *out = d;
    return ZKB_OK;
}

int side_begin(zkb_ctx* ctx) {
    DeviceGuard g(ctx);
    if (!ctx->other_stream) {
        // what goes there is long and narrow (chains of a few warps): its CTAs are placed before those of the wide work beside it
        int low = 0, high = 0;
        ZKB_CUDA(ctx, cudaDeviceGetStreamPriorityRange(&low, &high));
        ZKB_CUDA(ctx, cudaStreamCreateWithPriority(&ctx->other_stream, cudaStreamNonBlocking, high));
        for (auto& e : ctx->side_events) ZKB_CUDA(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    ZKB_CUDA(ctx, cudaEventRecord(ctx->side_events[0], ctx->stream));
    ZKB_CUDA(ctx, cudaStreamWaitEvent(ctx->other_stream, ctx->side_events[0], 0));
    std::swap(ctx->stream, ctx->other_stream);
    ctx->on_side = true;
    return ZKB_OK;
}
int side_end(zkb_ctx* ctx) {
    if (!ctx->on_side) return ZKB_OK;
    DeviceGuard g(ctx);
    std::swap(ctx->stream, ctx->other_stream);
    ctx->on_side = false;
    ctx->side_pending = true;
    ZKB_CUDA(ctx, cudaEventRecord(ctx->side_events[1], ctx->other_stream));
    return ZKB_OK;
}
int side_join(zkb_ctx* ctx) {
    if (int rc = side_end(ctx)) return rc;
    if (!ctx->side_pending) return ZKB_OK;
    DeviceGuard g(ctx);
    ctx->side_pending = false;
    ZKB_CUDA(ctx, cudaStreamWaitEvent(ctx->stream, ctx->side_events[1], 0));
    return ZKB_OK;
}

// A block's place in the ring, its bytes copied to the page-locked side.
static int stage_place(zkb_ctx* ctx, const void* h_data, size_t bytes, size_t* at) {
    const size_t slots = (bytes + sizeof(void*) - 1) / sizeof(void*);
    if (slots + 1 > ctx->ring_cap) return set_error(ctx, ZKB_EINVAL, "stage_blob: %zu bytes exceed the staging ring", bytes);
    size_t pos = (ctx->ring_pos + 1) & ~(size_t)1;  // slots are 8 bytes and the ring's base is aligned: even slots are 16-byte aligned
    if (pos + slots > ctx->ring_cap) {
        if (int rc = stage_wrap(ctx)) return rc;
        pos = 0;
    }
    memcpy(ctx->h_ring + pos, h_data, bytes);
    ctx->ring_pos = pos + slots;
    *at = pos;
    return ZKB_OK;
}
int stage_blob(zkb_ctx* ctx, const void* h_data, size_t bytes, void** out) {
    size_t pos = 0;
    if (int rc = stage_place(ctx, h_data, bytes, &pos)) return rc;
    ZKB_CUDA(ctx, cudaMemcpyAsync(ctx->d_ring + pos, ctx->h_ring + pos, bytes, cudaMemcpyHostToDevice, ctx->stream));
    *out = ctx->d_ring + pos;
    return ZKB_OK;
}
int upload_small(zkb_ctx* ctx, uint32_t* dst, const uint32_t* h, size_t words) {
    DeviceGuard g(ctx);
    size_t pos = 0;
    if (int rc = stage_place(ctx, h, words * 4, &pos)) return rc;
    ZKB_CUDA(ctx, cudaMemcpyAsync(dst, ctx->h_ring + pos, words * 4, cudaMemcpyHostToDevice, ctx->stream));
    return ZKB_OK;
}

// G * 2^b for the generator G of the order-2^31 circle group over M31
// (nitroo/crates/stwo/src/core/circle.rs:202-205).
__constant__ cpoint c_gen_pow2[31];

__device__ __forceinline__ cpoint circle_point_from_index(uint32_t idx) {
    cpoint r{1u, 0u};
#pragma unroll 1
    for (int b = 0; b < 31; b++)
        if ((idx >> b) & 1u) r = cpoint_add(r, c_gen_pow2[b]);
    return r;
}

// tw[t], t in [1, len): k = floor(log2 t) + 1, h = t - 2^(k-1);
// value = x( half_odds(k).at(bitrev_{k-1}(h)) ), index 2^(29-k) + j * 2^(31-k).
__global__ void twiddle_tower_kernel(uint32_t* __restrict__ tw, uint32_t* __restrict__ itw, size_t len) {
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= len) return;
    if (t == 0) { tw[0] = 1u; itw[0] = 1u; return; }
    int k = 32 - __clz((uint32_t)t);
    uint32_t h = (uint32_t)t - (1u << (k - 1));
    uint32_t j = (k > 1) ? (__brev(h) >> (32 - (k - 1))) : 0u;
    uint32_t index = (1u << (29 - k)) + (j << (31 - k));
    cpoint p = circle_point_from_index(index & 0x7fffffffu);
    tw[t] = p.x;
    itw[t] = m31_inv(p.x);
}

__global__ void twice_signed_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, size_t len) {
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < len) out[t] = m31_twice_signed(in[t]);
}

__global__ void gather_multi_kernel(const uint32_t* const* __restrict__ cols, int ncols, const uint32_t* __restrict__ idx,
                                    int nidx, uint32_t* __restrict__ out) {
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)ncols * nidx) return;
    int i = (int)(t / ncols), c = (int)(t % ncols);
    out[t] = cols[c][idx[i]];
}

__global__ void gather_hashes_kernel(const uint4* __restrict__ hashes, const uint32_t* __restrict__ idx, int nidx,
                                     uint4* __restrict__ out) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * nidx) return;
    out[t] = hashes[2 * (size_t)idx[t >> 1] + (t & 1)];
}

__global__ void gather_words_kernel(const uint32_t* const* __restrict__ addrs, size_t n, uint32_t* __restrict__ out) {
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) out[t] = *addrs[t];
}

// Everything a read plan asks for (gather_plan). Thread t < n_cells: cell t of the blocks (their out_off ascending; a CTA's first warp finds the block its
// cells begin in, the threads go on from there); then a word per word address; then eight words per hash address. The plan begins with
// the word addresses. With a launch a block beyond 2^20 cells, the 54 blocks of a micro segment took 119 us and as much in the gaps between them, now 14; 56 blocks of
// 12 million cells 236 us and the gaps, now 120.
struct PlanBlock { const uint32_t* const* cols; uint64_t out_off; uint32_t ncols, idx, here, pad; };  // idx: where its row indices start; here: cols is an offset into the plan
__host__ __device__ __forceinline__ const uint32_t* const* plan_cols(const PlanBlock& b, const void* plan) {
    return b.here ? reinterpret_cast<const uint32_t* const*>(static_cast<const char*>(plan) + reinterpret_cast<uintptr_t>(b.cols)) : b.cols;
}
__global__ void __launch_bounds__(256) gather_plan_kernel(const PlanBlock* __restrict__ blocks, int n_blocks, const uint32_t* __restrict__ idx, uint64_t n_cells,
                                                          const uint32_t* const* __restrict__ words, uint64_t n_words,
                                                          const uint32_t* const* __restrict__ hashes, uint64_t n_hashes, uint32_t* __restrict__ out) {
    __shared__ int first;
    const uint64_t t0 = blockIdx.x * 256ull, t = t0 + threadIdx.x;
    if (t0 < n_cells) {
        if (threadIdx.x < 32) {  // the last block that begins at t0 or before, of all that have cells
            int n = 0;
            for (int b = threadIdx.x; b < n_blocks; b += 32) n += blocks[b].out_off <= t0;
            n = __reduce_add_sync(0xffffffffu, n);
            if (threadIdx.x == 0) first = n - 1;
        }
        __syncthreads();
    }
    if (t < n_cells) {
        int b = first;
        while (b + 1 < n_blocks && blocks[b + 1].out_off <= t) b++;
        const PlanBlock pb = blocks[b];
        const uint32_t e = (uint32_t)(t - pb.out_off);
        out[t] = plan_cols(pb, words)[e % pb.ncols][idx[pb.idx + e / pb.ncols]];
        return;
    }
    if (t < n_cells + n_words) {
        out[t] = *words[t - n_cells];
        return;
    }
    const uint64_t h = t - n_cells - n_words;
    if (h < 8 * n_hashes) out[t] = hashes[h >> 3][h & 7];
}

}  // namespace zk

using namespace zk;

extern "C" int zk_set_error_public(zkb_ctx* ctx, int code, const char* msg) { return set_error(ctx, code, "%s", msg); }

extern "C" {

int zkb_init(int device, int max_log_size, zkb_ctx** out) {
    if (!out) return ZKB_EINVAL;
    *out = nullptr;
    if (max_log_size < 3 || max_log_size > 28) return ZKB_EINVAL;
    zkb_ctx* ctx = new (std::nothrow) zkb_ctx();
    if (!ctx) return ZKB_ENOMEM;
    ctx->device = device;
    ctx->max_log = max_log_size;
    ctx->blocks = new (std::nothrow) BlockCache();
    if (!ctx->blocks) { delete ctx; return ZKB_ENOMEM; }
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) { delete ctx->blocks; delete ctx; return ZKB_ECUDA; }
    auto fail = [&](int code) { zkb_destroy(ctx); return code; };
    if (cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(ZKB_ECUDA);
    ctx->tw_len = (size_t)1 << (max_log_size - 1);
    if (cudaMalloc(&ctx->tw, ctx->tw_len * 4) != cudaSuccess) return fail(ZKB_ENOMEM);
    if (cudaMalloc(&ctx->itw, ctx->tw_len * 4) != cudaSuccess) return fail(ZKB_ENOMEM);
    if (cudaMalloc(&ctx->tw2, ctx->tw_len * 4) != cudaSuccess) return fail(ZKB_ENOMEM);
    if (cudaMalloc(&ctx->itw2, ctx->tw_len * 4) != cudaSuccess) return fail(ZKB_ENOMEM);
    if (cudaMalloc(&ctx->dev_err, 64) != cudaSuccess) return fail(ZKB_ENOMEM);
    if (cudaMemsetAsync(ctx->dev_err, 0, 64, ctx->stream) != cudaSuccess) return fail(ZKB_ECUDA);
    ctx->ring_cap = RING_SLOTS;
    if (cudaMallocHost(&ctx->h_ring, ctx->ring_cap * sizeof(void*)) != cudaSuccess) return fail(ZKB_ENOMEM);
    if (cudaMalloc(&ctx->d_ring, ctx->ring_cap * sizeof(void*)) != cudaSuccess) return fail(ZKB_ENOMEM);
    ctx->scratch_words = SCRATCH_WORDS;
    if (cudaMalloc(&ctx->scratch, ctx->scratch_words * 4) != cudaSuccess) return fail(ZKB_ENOMEM);
    if (cudaMalloc(&ctx->ticket, 64) != cudaSuccess) return fail(ZKB_ENOMEM);
    if (cudaMemsetAsync(ctx->ticket, 0, 64, ctx->stream) != cudaSuccess) return fail(ZKB_ECUDA);
    if (cudaMallocHost(&ctx->h_small, (SMALL_WORDS + 16) * 4) != cudaSuccess) return fail(ZKB_ENOMEM);

    {
        cudaMemPool_t pool;
        if (cudaDeviceGetDefaultMemPool(&pool, device) != cudaSuccess) return fail(ZKB_ECUDA);
        unsigned long long keep = ~0ull;
        if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) return fail(ZKB_ECUDA);
    }
    // Generator doublings on the host, then the tower on the device.
    cpoint g[31];
    g[0] = {2u, 1268011823u};
    for (int b = 1; b < 31; b++) g[b] = cpoint_add(g[b - 1], g[b - 1]);
    if (cudaMemcpyToSymbolAsync(c_gen_pow2, g, sizeof(g), 0, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess) return fail(ZKB_ECUDA);
    unsigned blocks = (unsigned)((ctx->tw_len + 255) / 256);
    twiddle_tower_kernel<<<blocks, 256, 0, ctx->stream>>>(ctx->tw, ctx->itw, ctx->tw_len);
    twice_signed_kernel<<<blocks, 256, 0, ctx->stream>>>(ctx->tw, ctx->tw2, ctx->tw_len);
    twice_signed_kernel<<<blocks, 256, 0, ctx->stream>>>(ctx->itw, ctx->itw2, ctx->tw_len);
    if (cudaGetLastError() != cudaSuccess) return fail(ZKB_ECUDA);
    if (cudaStreamSynchronize(ctx->stream) != cudaSuccess) return fail(ZKB_ECUDA);
    *out = ctx;
    return ZKB_OK;
}

int zkb_destroy(zkb_ctx* ctx) {
    if (!ctx) return ZKB_EINVAL;
    cudaSetDevice(ctx->device);
    if (ctx->stream) {
        ctx->blocks->release(ctx->stream);
        cudaStreamSynchronize(ctx->stream);
    }
    delete ctx->blocks;
    if (ctx->tw) cudaFree(ctx->tw);
    if (ctx->itw) cudaFree(ctx->itw);
    if (ctx->tw2) cudaFree(ctx->tw2);
    if (ctx->itw2) cudaFree(ctx->itw2);
    if (ctx->dev_err) cudaFree(ctx->dev_err);
    if (ctx->h_ring) cudaFreeHost(ctx->h_ring);
    if (ctx->d_ring) cudaFree(ctx->d_ring);
    if (ctx->scratch) cudaFree(ctx->scratch);
    if (ctx->ticket) cudaFree(ctx->ticket);
    if (ctx->h_small) cudaFreeHost(ctx->h_small);
    if (ctx->h_batch) cudaFreeHost(ctx->h_batch);
    if (ctx->batch_tickets) cudaFree(ctx->batch_tickets);
    for (int i = 0; i < 64; i++)
        if (ctx->events[i]) cudaEventDestroy(ctx->events[i]);
    if (ctx->prof) {
        for (int i = 0; i < ctx->prof_cap; i++)
            if (ctx->prof[i].a) { cudaEventDestroy(ctx->prof[i].a); cudaEventDestroy(ctx->prof[i].b); }
        delete[] ctx->prof;
    }
    for (int i = 0; i < 64; i++)
        if (ctx->fences[i]) cudaEventDestroy(ctx->fences[i]);
    if (ctx->copy_gate) cudaEventDestroy(ctx->copy_gate);
    if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
    for (auto e : ctx->side_events)
        if (e) cudaEventDestroy(e);
    if (ctx->other_stream) cudaStreamDestroy(ctx->other_stream);
    for (auto st : ctx->peer_streams)
        if (st) cudaStreamDestroy(st);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
    return ZKB_OK;
}

const char* zkb_last_error(zkb_ctx* ctx) { return ctx ? ctx->err : "null context"; }

int zkb_sync(zkb_ctx* ctx) {
    if (!ctx) return ZKB_EINVAL;
    DeviceGuard g(ctx);
    if (ctx->copy_stream) ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->copy_stream));
    if (ctx->other_stream) ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->other_stream));
    // a kernel whose bounded wait ran out has set the error word; report it here, where the host waits anyway
    ZKB_CUDA(ctx, cudaMemcpyAsync(ctx->h_small + SMALL_WORDS, ctx->dev_err, 4, cudaMemcpyDeviceToHost, ctx->stream));
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (ctx->h_small[SMALL_WORDS] != 0) {
        unsigned code = ctx->h_small[SMALL_WORDS];
        cudaMemsetAsync(ctx->dev_err, 0, 4, ctx->stream);
        return set_error(ctx, ZKB_ETIMEOUT, "zkb_sync: a device-side wait ran out of its iteration limit (code 0x%x); results of the calls since the last sync are not valid", code);
    }
    return ZKB_OK;
}

int zkb_get_stream(zkb_ctx* ctx, void** stream) {
    if (!ctx || !stream) return ZKB_EINVAL;
    *stream = (void*)ctx->stream;
    return ZKB_OK;
}

int zkb_event_record(zkb_ctx* ctx, int slot) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, slot >= 0 && slot < 64);
    DeviceGuard g(ctx);
    if (!ctx->events[slot]) ZKB_CUDA(ctx, cudaEventCreate(&ctx->events[slot]));
    ZKB_CUDA(ctx, cudaEventRecord(ctx->events[slot], ctx->stream));
    return ZKB_OK;
}

int zkb_event_elapsed_ms(zkb_ctx* ctx, int a, int b, float* h_ms) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, a >= 0 && a < 64 && b >= 0 && b < 64 && h_ms && ctx->events[a] && ctx->events[b]);
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaEventSynchronize(ctx->events[b]));
    ZKB_CUDA(ctx, cudaEventElapsedTime(h_ms, ctx->events[a], ctx->events[b]));
    return ZKB_OK;
}

int zkb_profile_begin(zkb_ctx* ctx) {
    if (!ctx) return ZKB_EINVAL;
    DeviceGuard g(ctx);
    if (!ctx->prof) {
        ctx->prof_cap = 8192;
        ctx->prof = new (std::nothrow) zkb_ctx::ProfRec[ctx->prof_cap]();
        if (!ctx->prof) { ctx->prof_cap = 0; return set_error(ctx, ZKB_ENOMEM, "zkb_profile_begin: out of host memory"); }
    }
    ctx->prof_n = 0;
    ctx->prof_on = true;
    return ZKB_OK;
}

int zkb_profile_end(zkb_ctx* ctx, const char** h_names, float* h_ms, int* h_count, int cap, int* n) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, h_names && h_ms && h_count && n && cap > 0);
    DeviceGuard g(ctx);
    ctx->prof_on = false;
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    int k = 0;
    for (int i = 0; i < ctx->prof_n; i++) {
        float ms = 0.f;
        ZKB_CUDA(ctx, cudaEventElapsedTime(&ms, ctx->prof[i].a, ctx->prof[i].b));
        int j = 0;
        while (j < k && h_names[j] != ctx->prof[i].name) j++;
        if (j == k) {
            if (k == cap) continue;
            h_names[k] = ctx->prof[i].name; h_ms[k] = 0.f; h_count[k] = 0; k++;
        }
        h_ms[j] += ms;
        h_count[j] += 1;
    }
    *n = k;
    return ZKB_OK;
}

int zkb_max_log_size(zkb_ctx* ctx) { return ctx ? ctx->max_log : ZKB_EINVAL; }

int zkb_malloc(zkb_ctx* ctx, size_t bytes, void** dptr) {
    if (!ctx || !dptr) return ZKB_EINVAL;
    DeviceGuard g(ctx);
    *dptr = nullptr;
    if (bytes == 0) return ZKB_OK;
    // Stream-ordered allocation from the device's default pool (kept warm: the release threshold
    // is raised in zkb_init), so neither allocation nor release synchronises the device.
    BlockCache& bc = *ctx->blocks;
    const bool small = bytes <= ((size_t)1 << BlockCache::MAX_LOG);
    const int log = small ? BlockCache::log_of(bytes) : 0;
    if (small && !bc.kept[log].empty()) {
        *dptr = bc.kept[log].back();
        bc.kept[log].pop_back();
        bc.kept_bytes -= (size_t)1 << log;
        bc.live[*dptr] = log;
        return ZKB_OK;
    }
    const size_t want = small ? (size_t)1 << log : bytes;
    cudaError_t e = cudaMallocAsync(dptr, want, ctx->stream);
    if (e == cudaErrorMemoryAllocation && bc.kept_bytes) {
        (void)cudaGetLastError();
        bc.release(ctx->stream);
        e = cudaMallocAsync(dptr, want, ctx->stream);
    }
    ZKB_CUDA(ctx, e);
    if (small) bc.live[*dptr] = log;
    return ZKB_OK;
}

int zkb_free(zkb_ctx* ctx, void* dptr) {
    if (!ctx) return ZKB_EINVAL;
    if (!dptr) return ZKB_OK;
    DeviceGuard g(ctx);
    BlockCache& bc = *ctx->blocks;
    auto it = bc.live.find(dptr);
    if (it != bc.live.end()) {
        const int log = it->second;
        bc.live.erase(it);
        if (bc.kept_bytes + ((size_t)1 << log) <= BlockCache::KEPT_BYTES) {
            bc.kept[log].push_back(dptr);
            bc.kept_bytes += (size_t)1 << log;
            return ZKB_OK;
        }
    }
    ZKB_CUDA(ctx, cudaFreeAsync(dptr, ctx->stream));
    return ZKB_OK;
}

int zkb_memset_zero(zkb_ctx* ctx, void* dptr, size_t bytes) {
    if (!ctx) return ZKB_EINVAL;
    if (bytes == 0) return ZKB_OK;
    ZKB_CHECK_ARG(ctx, dptr != nullptr);
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaMemsetAsync(dptr, 0, bytes, ctx->stream));
    return ZKB_OK;
}

int zkb_h2d(zkb_ctx* ctx, void* dptr, const void* h_src, size_t bytes) {
    if (!ctx) return ZKB_EINVAL;
    if (bytes == 0) return ZKB_OK;
    ZKB_CHECK_ARG(ctx, dptr != nullptr && h_src != nullptr);
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaMemcpyAsync(dptr, h_src, bytes, cudaMemcpyHostToDevice, ctx->stream));
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return ZKB_OK;
}

int zkb_d2h(zkb_ctx* ctx, void* h_dst, const void* dptr, size_t bytes) {
    if (!ctx) return ZKB_EINVAL;
    if (bytes == 0) return ZKB_OK;
    ZKB_CHECK_ARG(ctx, dptr != nullptr && h_dst != nullptr);
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaMemcpyAsync(h_dst, dptr, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return ZKB_OK;
}

int zkb_h2d_async(zkb_ctx* ctx, void* dptr, const void* h_pinned_src, size_t bytes) {
    if (!ctx) return ZKB_EINVAL;
    if (bytes == 0) return ZKB_OK;
    ZKB_CHECK_ARG(ctx, dptr != nullptr && h_pinned_src != nullptr);
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaMemcpyAsync(dptr, h_pinned_src, bytes, cudaMemcpyHostToDevice, ctx->stream));
    return ZKB_OK;
}

int zkb_h2d_overlapped(zkb_ctx* ctx, void* dptr, const void* h_pinned_src, size_t bytes, int fence) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, fence >= -1 && fence < 64 && (bytes == 0 || (dptr != nullptr && h_pinned_src != nullptr)));
    DeviceGuard g(ctx);
    if (!ctx->copy_stream) ZKB_CUDA(ctx, cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
    if (!ctx->copy_gate) ZKB_CUDA(ctx, cudaEventCreateWithFlags(&ctx->copy_gate, cudaEventDisableTiming));
    // the destination may have been allocated (stream-ordered) on the compute stream just now
    ZKB_CUDA(ctx, cudaEventRecord(ctx->copy_gate, ctx->stream));
    ZKB_CUDA(ctx, cudaStreamWaitEvent(ctx->copy_stream, ctx->copy_gate, 0));
    if (bytes) ZKB_CUDA(ctx, cudaMemcpyAsync(dptr, h_pinned_src, bytes, cudaMemcpyHostToDevice, ctx->copy_stream));
    if (fence >= 0) {
        if (!ctx->fences[fence]) ZKB_CUDA(ctx, cudaEventCreateWithFlags(&ctx->fences[fence], cudaEventDisableTiming));
        ZKB_CUDA(ctx, cudaEventRecord(ctx->fences[fence], ctx->copy_stream));
    }
    return ZKB_OK;
}

int zkb_wait_fence(zkb_ctx* ctx, int fence) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, fence >= 0 && fence < 64 && ctx->fences[fence] != nullptr);
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaStreamWaitEvent(ctx->stream, ctx->fences[fence], 0));
    return ZKB_OK;
}

// ---- buffers another process's GPU can write into (one process per GPU on one host) -----------------------------
// The stream-ordered pool's memory can not be shared between processes, so these come from cudaMalloc. A peer opens the
// handle and copies into the buffer with the copy engines (zkb_copy_to_peer): no SM is used, which is what lets the
// exchange of a sharded commitment run under the transform kernels (a collective's copy kernels wait for SMs the
// persistent transform passes hold).
int zkb_peer_buffer_alloc(zkb_ctx* ctx, size_t bytes, void** dptr, unsigned char handle[64]) {
    if (!ctx || !dptr || !handle || bytes == 0) return ZKB_EINVAL;
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "handle size");
    DeviceGuard g(ctx);
    *dptr = nullptr;
    ZKB_CUDA(ctx, cudaMalloc(dptr, bytes));
    cudaIpcMemHandle_t h;
    cudaError_t e = cudaIpcGetMemHandle(&h, *dptr);
    if (e != cudaSuccess) {
        cudaFree(*dptr);
        *dptr = nullptr;
        return set_error(ctx, ZKB_ECUDA, "zkb_peer_buffer_alloc: %s", cudaGetErrorString(e));
    }
    memcpy(handle, &h, 64);
    return ZKB_OK;
}
int zkb_peer_buffer_free(zkb_ctx* ctx, void* dptr) {
    if (!ctx) return ZKB_EINVAL;
    if (!dptr) return ZKB_OK;
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    ZKB_CUDA(ctx, cudaFree(dptr));
    return ZKB_OK;
}
int zkb_peer_buffer_open(zkb_ctx* ctx, const unsigned char handle[64], void** peer_ptr) {
    if (!ctx || !handle || !peer_ptr) return ZKB_EINVAL;
    DeviceGuard g(ctx);
    cudaIpcMemHandle_t h;
    memcpy(&h, handle, 64);
    *peer_ptr = nullptr;
    ZKB_CUDA(ctx, cudaIpcOpenMemHandle(peer_ptr, h, cudaIpcMemLazyEnablePeerAccess));
    return ZKB_OK;
}
int zkb_peer_buffer_close(zkb_ctx* ctx, void* peer_ptr) {
    if (!ctx) return ZKB_EINVAL;
    if (!peer_ptr) return ZKB_OK;
    DeviceGuard g(ctx);
    for (auto st : ctx->peer_streams)
        if (st) ZKB_CUDA(ctx, cudaStreamSynchronize(st));
    ZKB_CUDA(ctx, cudaIpcCloseMemHandle(peer_ptr));
    return ZKB_OK;
}
int zkb_copy_to_peer(zkb_ctx* ctx, void* dst, const void* src, size_t bytes, int lane) {
    if (!ctx || !dst || !src || lane < 0) return ZKB_EINVAL;
    DeviceGuard g(ctx);
    cudaStream_t& st = ctx->peer_streams[lane & 3];
    if (!st) ZKB_CUDA(ctx, cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    if (!ctx->copy_gate) ZKB_CUDA(ctx, cudaEventCreateWithFlags(&ctx->copy_gate, cudaEventDisableTiming));
    // after everything enqueued on the compute stream so far (the source has just been written there)
    ZKB_CUDA(ctx, cudaEventRecord(ctx->copy_gate, ctx->stream));
    ZKB_CUDA(ctx, cudaStreamWaitEvent(st, ctx->copy_gate, 0));
    if (bytes) ZKB_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, st));
    return ZKB_OK;
}
int zkb_peer_copies_wait(zkb_ctx* ctx) {
    if (!ctx) return ZKB_EINVAL;
    DeviceGuard g(ctx);
    for (auto st : ctx->peer_streams)
        if (st) ZKB_CUDA(ctx, cudaStreamSynchronize(st));
    return ZKB_OK;
}

int zkb_d2h_async(zkb_ctx* ctx, void* h_pinned_dst, const void* dptr, size_t bytes) {
    if (!ctx) return ZKB_EINVAL;
    if (bytes == 0) return ZKB_OK;
    ZKB_CHECK_ARG(ctx, dptr != nullptr && h_pinned_dst != nullptr);
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaMemcpyAsync(h_pinned_dst, dptr, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    return ZKB_OK;
}

int zkb_d2d(zkb_ctx* ctx, void* dst, const void* src, size_t bytes) {
    if (!ctx) return ZKB_EINVAL;
    if (bytes == 0) return ZKB_OK;
    ZKB_CHECK_ARG(ctx, dst != nullptr && src != nullptr);
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    return ZKB_OK;
}

int zkb_host_alloc_pinned(zkb_ctx* ctx, size_t bytes, void** h_ptr) {
    if (!ctx || !h_ptr) return ZKB_EINVAL;
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaMallocHost(h_ptr, bytes ? bytes : 1));
    return ZKB_OK;
}

int zkb_host_free_pinned(zkb_ctx* ctx, void* h_ptr) {
    if (!ctx) return ZKB_EINVAL;
    if (!h_ptr) return ZKB_OK;
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaFreeHost(h_ptr));
    return ZKB_OK;
}

int zkb_gather_multi(zkb_ctx* ctx, const uint32_t* const* cols, int ncols, const uint32_t* h_idx, int nidx,
                     uint32_t* h_out) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, ncols >= 0 && nidx >= 0);
    if (ncols == 0 || nidx == 0) return ZKB_OK;
    ZKB_CHECK_ARG(ctx, cols != nullptr && h_idx != nullptr && h_out != nullptr);
    size_t total = (size_t)ncols * nidx;
    ZKB_CHECK_ARG(ctx, total + (size_t)nidx <= ctx->scratch_words);
    DeviceGuard g(ctx);
    void** d_cols;
    int rc = stage_ptrs(ctx, (const void* const*)cols, ncols, &d_cols);
    if (rc) return rc;
    uint32_t* d_idx = ctx->scratch;
    uint32_t* d_out = ctx->scratch + nidx;
    ZKB_CUDA(ctx, cudaMemcpyAsync(d_idx, h_idx, (size_t)nidx * 4, cudaMemcpyHostToDevice, ctx->stream));
    gather_multi_kernel<<<(unsigned)((total + 255) / 256), 256, 0, ctx->stream>>>((const uint32_t* const*)d_cols, ncols,
                                                                                  d_idx, nidx, d_out);
    ZKB_LAUNCH_CHECK(ctx);
    ZKB_CUDA(ctx, cudaMemcpyAsync(h_out, d_out, total * 4, cudaMemcpyDeviceToHost, ctx->stream));
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return ZKB_OK;
}

int zkb_gather_words(zkb_ctx* ctx, const uint32_t* const* h_addrs, size_t n, uint32_t* h_out) {
    if (!ctx) return ZKB_EINVAL;
    if (n == 0) return ZKB_OK;
    ZKB_CHECK_ARG(ctx, h_addrs != nullptr && h_out != nullptr);
    DeviceGuard g(ctx);
    // addresses (2 words each) and results share the scratch buffer; large requests go in slices
    const size_t slice = ctx->scratch_words / 3;
    for (size_t off = 0; off < n; off += slice) {
        size_t m = n - off < slice ? n - off : slice;
        const uint32_t** d_addrs = reinterpret_cast<const uint32_t**>(ctx->scratch);
        uint32_t* d_out = ctx->scratch + 2 * slice;
        ZKB_CUDA(ctx, cudaMemcpyAsync(d_addrs, h_addrs + off, m * sizeof(void*), cudaMemcpyHostToDevice, ctx->stream));
        gather_words_kernel<<<(unsigned)((m + 255) / 256), 256, 0, ctx->stream>>>(d_addrs, m, d_out);
        ZKB_LAUNCH_CHECK(ctx);
        ZKB_CUDA(ctx, cudaMemcpyAsync(h_out + off, d_out, m * 4, cudaMemcpyDeviceToHost, ctx->stream));
        ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    return ZKB_OK;
}

int zkb_gather_hashes(zkb_ctx* ctx, const uint32_t* hashes, const uint32_t* h_idx, int nidx, uint32_t* h_out) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, nidx >= 0);
    if (nidx == 0) return ZKB_OK;
    ZKB_CHECK_ARG(ctx, hashes != nullptr && h_idx != nullptr && h_out != nullptr && ((uintptr_t)hashes & 15) == 0);
    ZKB_CHECK_ARG(ctx, (size_t)nidx * 9 + 4 <= ctx->scratch_words);
    DeviceGuard g(ctx);
    uint32_t* d_out = ctx->scratch;  // 8 words per hash, 16-byte aligned
    uint32_t* d_idx = ctx->scratch + 8 * (size_t)nidx;
    ZKB_CUDA(ctx, cudaMemcpyAsync(d_idx, h_idx, (size_t)nidx * 4, cudaMemcpyHostToDevice, ctx->stream));
    gather_hashes_kernel<<<(2 * nidx + 127) / 128, 128, 0, ctx->stream>>>(reinterpret_cast<const uint4*>(hashes), d_idx, nidx,
                                                                        reinterpret_cast<uint4*>(d_out));
    ZKB_LAUNCH_CHECK(ctx);
    ZKB_CUDA(ctx, cudaMemcpyAsync(h_out, d_out, (size_t)nidx * 32, cudaMemcpyDeviceToHost, ctx->stream));
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return ZKB_OK;
}

int zkb_twiddles_d2h(zkb_ctx* ctx, int log_size, uint32_t* h_tw, uint32_t* h_itw) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, h_tw != nullptr && log_size >= 0 && log_size <= ctx->max_log - 1);
    DeviceGuard g(ctx);
    // Level j of the reference layout is T_{log_size - j}: 2^(log_size-j-1) words at offset
    // 2^log_size - 2^(log_size-j); the last word is the padding value 1.
    size_t n = (size_t)1 << log_size;
    for (int j = 0; j < log_size; j++) {
        int k = log_size - j;
        size_t len = (size_t)1 << (k - 1), off = n - ((size_t)1 << k);
        ZKB_CUDA(ctx, cudaMemcpyAsync(h_tw + off, ctx->tw + len, len * 4, cudaMemcpyDeviceToHost, ctx->stream));
        if (h_itw) ZKB_CUDA(ctx, cudaMemcpyAsync(h_itw + off, ctx->itw + len, len * 4, cudaMemcpyDeviceToHost, ctx->stream));
    }
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    h_tw[n - 1] = 1u;
    if (h_itw) h_itw[n - 1] = 1u;
    return ZKB_OK;
}

int zkb_secure_powers(zkb_ctx* ctx, const uint32_t h_felt[4], size_t n, uint32_t* h_out) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, h_felt != nullptr && (n == 0 || h_out != nullptr));
    qm31 f{{h_felt[0], h_felt[1], h_felt[2], h_felt[3]}}, acc = qm31_one();
    for (size_t i = 0; i < n; i++) {
        for (int k = 0; k < 4; k++) h_out[4 * i + k] = acc.c[k];
        acc = qm31_mul(acc, f);
    }
    return ZKB_OK;
}

}  // extern "C"

namespace zk {

int stage_table(zkb_ctx* ctx, const uint32_t* const* ptrs, int n) {
    DeviceGuard g(ctx);
    void** d = nullptr;
    return stage_ptrs(ctx, (const void* const*)ptrs, n, &d);
}

int stage_tables(zkb_ctx* ctx, const std::pair<const uint32_t* const*, size_t>* tables, size_t n_tables) {
    if (ctx->on_side) return ZKB_OK;  // whoever wants one copies it
    DeviceGuard g(ctx);
    size_t total = 0;
    for (size_t k = 0; k < n_tables; k++) total += tables[k].second;
    if (total > ctx->ring_cap / 2) return ZKB_OK;
    if (int rc = stage_reserve(ctx, total)) return rc;
    const size_t first = ctx->ring_pos;
    size_t end = first;
    std::vector<std::pair<size_t, size_t>> placed;  // remembered when the copy is on its way: a table that is found has to be there
    for (size_t k = 0; k < n_tables; k++) {
        const void* const* const p = (const void* const*)tables[k].first;
        const size_t n = tables[k].second;
        if (!n || find_staged(ctx, p, n)) continue;
        memcpy(ctx->h_ring + end, p, n * sizeof(void*));
        placed.push_back({end, n});
        end += n;
    }
    if (placed.empty()) return ZKB_OK;
    ZKB_CUDA(ctx, cudaMemcpyAsync(ctx->d_ring + first, ctx->h_ring + first, (end - first) * sizeof(void*), cudaMemcpyHostToDevice, ctx->stream));
    ctx->ring_pos = end;
    for (const auto& t : placed) remember_staged(ctx, t.first, t.second);
    return ZKB_OK;
}

int gather_plan(zkb_ctx* ctx, const GatherBlock* blocks, int n_blocks, size_t total_words, const uint32_t* const* word_addrs, size_t n_words,
                const uint32_t* const* hash_addrs, size_t n_hashes, uint32_t* h_out) {
    const size_t results = total_words + n_words + 8 * n_hashes;
    if (results == 0) return ZKB_OK;
    DeviceGuard g(ctx);
    // The column tables of short blocks (a FRI layer's four columns) travel in the plan; those of a tree's columns are the ones its
    // commitment staged.
    int own_cols = 64;
    size_t n_idx = 0, n_own = 0, n_wide = 0;
    for (int b = 0; b < n_blocks; b++) {
        n_idx += (size_t)blocks[b].nidx;
        (blocks[b].ncols <= own_cols ? n_own : n_wide) += (size_t)blocks[b].ncols;
    }
    if (n_wide > ctx->ring_cap / 2) {  // too many to be in the ring together: all travel in the plan
        own_cols = INT_MAX;
        n_own += n_wide;
        n_wide = 0;
    }
    // [word addresses | hash addresses | short tables | block descriptors | row indices]
    const size_t at_hash = 8 * n_words, at_own = at_hash + 8 * n_hashes, at_blocks = at_own + 8 * n_own, at_idx = at_blocks + sizeof(PlanBlock) * (size_t)n_blocks;
    std::vector<unsigned char> blob(at_idx + 4 * n_idx);
    const bool in_ring = blob.size() <= sizeof(void*) * (ctx->ring_cap / 8);  // a longer plan brings its own memory
    if (int rc = stage_reserve(ctx, n_wide + (in_ring ? blob_slots(blob.size()) : 0))) return rc;
    if (n_words) memcpy(blob.data(), word_addrs, 8 * n_words);
    if (n_hashes) memcpy(blob.data() + at_hash, hash_addrs, 8 * n_hashes);
    PlanBlock* pb = reinterpret_cast<PlanBlock*>(blob.data() + at_blocks);
    uint32_t* pi = reinterpret_cast<uint32_t*>(blob.data() + at_idx);
    size_t first_idx = 0, own = 0;
    for (int b = 0; b < n_blocks; b++) {
        const GatherBlock& g = blocks[b];
        void** cols = nullptr;
        const bool here = g.ncols <= own_cols;
        if (here) {  // as an offset into the plan
            memcpy(blob.data() + at_own + 8 * own, g.cols, 8 * (size_t)g.ncols);
            cols = reinterpret_cast<void**>(at_own + 8 * own);
            own += (size_t)g.ncols;
        } else if (int rc = stage_ptrs(ctx, (const void* const*)g.cols, g.ncols, &cols)) {
            return rc;
        }
        if (g.nidx) memcpy(pi + first_idx, g.idx, 4 * (size_t)g.nidx);
        pb[b] = {(const uint32_t* const*)cols, g.out_off, (uint32_t)g.ncols, (uint32_t)first_idx, here ? 1u : 0u, 0u};
        first_idx += (size_t)g.nidx;
    }
    unsigned char *d_blob = nullptr, *d_own = nullptr;
    uint32_t* d_out = nullptr;
    cudaError_t e = cudaSuccess;
    int rc = ZKB_OK;
    if (in_ring) {
        rc = stage_blob(ctx, blob.data(), blob.size(), (void**)&d_blob);
    } else {
        rc = zkb_malloc(ctx, blob.size(), (void**)&d_own);
        d_blob = d_own;
        if (rc == ZKB_OK) e = cudaMemcpyAsync(d_blob, blob.data(), blob.size(), cudaMemcpyHostToDevice, ctx->stream);
    }
    if (rc == ZKB_OK) rc = zkb_malloc(ctx, results * 4, (void**)&d_out);
    if (rc == ZKB_OK && e == cudaSuccess) {
        const uint32_t* const* d_words = reinterpret_cast<const uint32_t* const*>(d_blob);
        const uint32_t* const* d_hashes = reinterpret_cast<const uint32_t* const*>(d_blob + at_hash);
        const PlanBlock* d_blocks = reinterpret_cast<const PlanBlock*>(d_blob + at_blocks);
        const uint32_t* d_idx = reinterpret_cast<const uint32_t*>(d_blob + at_idx);
        gather_plan_kernel<<<(unsigned)((results + 255) / 256), 256, 0, ctx->stream>>>(d_blocks, n_blocks, d_idx, total_words, d_words, n_words, d_hashes, n_hashes, d_out);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(h_out, d_out, results * 4, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    }
    zkb_free(ctx, d_out);
    zkb_free(ctx, d_own);
    if (rc != ZKB_OK) return rc;
    if (e != cudaSuccess) return set_error(ctx, ZKB_ECUDA, "gather_plan: %s", cudaGetErrorString(e));
    return ZKB_OK;
}

}  // namespace zk
