// MerkleOps::commit_on_layer with the Blake2s hasher, and the proof-of-work grind.
//
// A node's message is [left child hash | right child hash |] col_0[i] | col_1[i] | ... with every
// column value as one little-endian word (nitroo/crates/stwo/src/core/vcs/blake2_merkle.rs:18-39),
// hashed with Blake2s-256 (RFC 7693) and, for the M31 hasher, each digest word reduced mod 2^31-1
// (core/vcs/blake2_hash.rs:111-118). One thread hashes one node: the column words ARE the message
// words, so a 64-byte block is 16 coalesced loads (one per column) straight into registers.
#include <algorithm>

#include "blake2s.cuh"
#include "channel.cuh"
#include "common.cuh"

namespace zk {

__device__ __forceinline__ void store_hash(uint32_t* __restrict__ out, size_t i, const uint32_t h[8], bool m31_out) {
    uint32_t r[8];
#pragma unroll
    for (int k = 0; k < 8; k++) r[k] = m31_out ? reduce_word_m31(h[k]) : h[k];
    uint4* o = reinterpret_cast<uint4*>(out + 8 * i);
    o[0] = make_uint4(r[0], r[1], r[2], r[3]);
    o[1] = make_uint4(r[4], r[5], r[6], r[7]);
}

__global__ void __launch_bounds__(256) merkle_layer_kernel(int log_size, const uint32_t* __restrict__ prev,
                                                           const uint32_t* const* __restrict__ cols, int ncols,
                                                           int m31_out, uint32_t* __restrict__ out) {
    const size_t n = (size_t)1 << log_size;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t h[8], m[16];
    blake2s_init(h);
    const uint32_t total = (prev ? 64u : 0u) + 4u * (uint32_t)ncols;
    uint32_t t = 0;
    int c = 0;
    if (prev) {
        const uint4* p = reinterpret_cast<const uint4*>(prev + 16 * i);
        uint4 a = p[0], b = p[1], cc = p[2], d = p[3];
        m[0] = a.x; m[1] = a.y; m[2] = a.z; m[3] = a.w; m[4] = b.x; m[5] = b.y; m[6] = b.z; m[7] = b.w;
        m[8] = cc.x; m[9] = cc.y; m[10] = cc.z; m[11] = cc.w; m[12] = d.x; m[13] = d.y; m[14] = d.z; m[15] = d.w;
        t = 64;
        blake2s_compress(h, m, t, total == 64u);
    }
    // full blocks of 16 columns that are not the last block
    while (ncols - c > 16) {
#pragma unroll
        for (int k = 0; k < 16; k++) m[k] = cols[c + k][i];
        c += 16;
        t += 64;
        blake2s_compress(h, m, t, false);
    }
    // last block: 1..16 remaining columns, or the empty message when nothing was hashed yet
    if (ncols - c > 0 || total == 0u) {
        int rem = ncols - c;
#pragma unroll
        for (int k = 0; k < 16; k++) m[k] = (k < rem) ? cols[c + k][i] : 0u;
        t += 4u * (uint32_t)rem;
        blake2s_compress(h, m, t, true);
    }
    store_hash(out, i, h, m31_out != 0);
}

// The same node hash for layers of at most 2^13 nodes and few columns (chain_min_cols), four lanes to a node (b2s_compress_quad in channel.cuh). Such a layer is
// bound by the latency of its compressions, and by fetching their code where it is one of a few: a quad issues a quarter of
// a thread's instructions from a quarter of the code. A lane brings four of a block's sixteen words; a block's words
// and the addresses of the next one's are on their way while the block before is hashed. A tree of 2^16 leaves built layer by
// layer, with the next launch started early (below): 5.4 -> 4.2 us a layer.
constexpr int QUAD_THREADS = 64, QUAD_MAX_LOG = 13;
__global__ void __launch_bounds__(QUAD_THREADS) merkle_layer_quad_kernel(int log_size, const uint32_t* prev,
                                                                         const uint32_t* const* __restrict__ cols, int ncols, int m31_out,
                                                                         uint32_t* out) {
    __shared__ uint32_t sched[40];
    __shared__ alignas(16) uint32_t msg[QUAD_THREADS / 4][PAIR_WORDS];
    const uint32_t node = blockIdx.x * (QUAD_THREADS / 4) + (threadIdx.x >> 2), l = threadIdx.x & 3u;
    const bool live = (node >> log_size) == 0;
    const uint32_t i = live ? node : 0u;
    const int col_blocks = (ncols + 15) / 16, first = prev ? 0 : 1, end = prev || ncols ? 1 + col_blocks : 2;  // block 0: the children
    const uint32_t* at[4] = {nullptr, nullptr, nullptr, nullptr};
    uint32_t next[4] = {0u, 0u, 0u, 0u};
    auto addresses = [&](int b) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int c = 16 * b + 4 * (int)l + u;
            at[u] = c < ncols ? cols[c] : nullptr;
        }
    };
    auto values = [&] {
#pragma unroll
        for (int u = 0; u < 4; u++) next[u] = at[u] ? at[u][i] : 0u;
    };
    quad_make_schedule(sched, threadIdx.x, QUAD_THREADS);
    __syncthreads();
    uint32_t* const m = msg[threadIdx.x >> 2];
    const QuadWords word(m, sched);
    const QuadConst k;
    // A tree built layer by layer is a chain of launches of a microsecond or two: the next one may start now (programmatic dependent
    // launch) and wait here for this grid to end. (What that grid writes while this one already runs, the children and the columns, is
    // read by plain loads: a read-only load is for memory that nobody writes during a kernel's life.)
    let_next_start();
    follow_previous();
    addresses(0);
    uint4 cur = make_uint4(0u, 0u, 0u, 0u);
    if (prev) cur = reinterpret_cast<const uint4*>(prev)[4 * (size_t)i + l];
    values();
    addresses(1);
    uint2 h = make_uint2(k.h0, k.h1);
#pragma unroll 1
    for (int b = first; b < end; b++) {
        if (b > 0) cur = make_uint4(next[0], next[1], next[2], next[3]);
        *reinterpret_cast<uint4*>(m + 4 * l) = cur;
        __syncwarp();
        if (b > 0) {
            values();
            addresses(b + 1);
        }
        const bool last = b + 1 == end;
        const uint32_t bytes = (prev ? 64u : 0u) + 4u * (uint32_t)(16 * b < ncols ? 16 * b : ncols);
        h = b2s_compress_quad(h, word, k, bytes, last ? 0xffffffffu : 0u);
        __syncwarp();
    }
    if (live) {
        out[8 * (size_t)node + l] = m31_out ? reduce_word_m31(h.x) : h.x;
        out[8 * (size_t)node + 4 + l] = m31_out ? reduce_word_m31(h.y) : h.y;
    }
}

// The same for layers of many columns, a chain of up to 2,000 compressions a node: sixteen nodes' quads in two warps, and a third warp that brings
// their blocks, so that a hash meets no load from memory and none of the instructions around one (some 250 of 1,500 cycles a
// block). While block k is hashed the loader puts block k + 1 into the other buffer, its words asked for two blocks before and
// their columns' addresses three; one CTA barrier a block.
constexpr int CHAIN_NODES = 16, CHAIN_THREADS = 4 * CHAIN_NODES + 32;
// From how many columns on. The third warp costs a start of its own and a barrier a block, which some six blocks make up for; where a CTA shares its SM
// with another, from 2^12 nodes on, it shares schedulers too and takes longer to. Quads -> chain, a layer alone, columns not in L2: 2^8 nodes of 64
// columns 10.3 -> 10.7 us, 80 10.5 -> 10.7, 96 11.2 -> 10.7, 256 18.8 -> 17.6, 4,096 203 -> 176; 2^11 of 80 10.6 -> 10.8, 96 11.4 -> 11.0, 1,024 55.7 -> 53.4;
// 2^12 of 256 19.1 -> 21.0, 512 32.4 -> 33.2, 1,024 57.3 -> 57.4, 2,048 106.3 -> 105.2, 16,000 777 -> 764; 2^13 of 128 14.8 -> 16.0, 144 18.4 -> 16.5, 300 25.6 ->
// 25.1, 4,096 244 -> 224.
static int chain_min_cols(int log_size) { return log_size <= 11 ? 96 : log_size == 12 ? 1536 : 144; }
__global__ void __launch_bounds__(CHAIN_THREADS) merkle_layer_chain_kernel(int log_size, const uint32_t* prev, const uint32_t* const* __restrict__ cols, int ncols,
                                                                           int m31_out, uint32_t* out) {
    __shared__ uint32_t sched[40];
    __shared__ alignas(16) uint32_t msg[2][CHAIN_NODES][PAIR_WORDS];
    const int children = prev ? 1 : 0, n_blocks = children + (ncols + 15) / 16;
    quad_make_schedule(sched, threadIdx.x, CHAIN_THREADS);
    __syncthreads();
    let_next_start();
    follow_previous();
    if (threadIdx.x >= 4 * CHAIN_NODES) {
        // lane: eight words of a node's block
        const uint32_t mine = threadIdx.x & 15u, half = (threadIdx.x >> 4) & 1u, node = blockIdx.x * CHAIN_NODES + mine;
        const uint32_t i = (node >> log_size) == 0 ? node : 0u;
        const uint32_t* at[8];
        auto addresses = [&](int k) {  // of block k
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int c = 16 * (k - children) + 8 * (int)half + u;
                at[u] = c >= 0 && c < ncols ? cols[c] : nullptr;
            }
        };
        auto fetch = [&](int k, uint32_t (&v)[8]) {  // block k, whose addresses are there; then the next one's addresses
            if (k < children) {
                const uint4* const p = reinterpret_cast<const uint4*>(prev) + 4 * (size_t)i + 2 * half;
                const uint4 x = p[0], y = p[1];
                v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
            } else {
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = at[u] ? at[u][i] : 0u;
            }
            addresses(k + 1);
        };
        auto put = [&](int k, const uint32_t (&v)[8]) {
            uint4* const o = reinterpret_cast<uint4*>(&msg[k & 1][mine][8 * half]);
            o[0] = make_uint4(v[0], v[1], v[2], v[3]);
            o[1] = make_uint4(v[4], v[5], v[6], v[7]);
        };
        uint32_t v0[8], v1[8];
        addresses(0);
        fetch(0, v0);
        fetch(1, v1);
        put(0, v0);
        fetch(2, v0);
        __syncthreads();
        // block k is being hashed: v1 holds block k + 1, v0 block k + 2 (blocks past the end are zeros that nobody hashes)
        for (int k = 0; k < n_blocks; k += 2) {
            put(k + 1, v1);
            fetch(k + 3, v1);
            __syncthreads();
            if (k + 1 == n_blocks) break;
            put(k + 2, v0);
            fetch(k + 4, v0);
            __syncthreads();
        }
        return;
    }
    const uint32_t l = threadIdx.x & 3u, mine = threadIdx.x >> 2, node = blockIdx.x * CHAIN_NODES + mine;
    QuadWords word(msg[0][mine], sched);
    const QuadConst q;
    uint2 h = make_uint2(q.h0, q.h1);
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < n_blocks; k++) {
        const bool last = k + 1 == n_blocks;
        const uint32_t bytes = last ? 64u * children + 4u * (uint32_t)ncols : 64u * (uint32_t)(k + 1);
        word.at = (k & 1) * (uint32_t)sizeof(msg[0]);
        h = b2s_compress_quad(h, word, q, bytes, last ? 0xffffffffu : 0u);
        __syncthreads();
    }
    if ((node >> log_size) == 0) {
        out[8 * (size_t)node + l] = m31_out ? reduce_word_m31(h.x) : h.x;
        out[8 * (size_t)node + 4 + l] = m31_out ? reduce_word_m31(h.y) : h.y;
    }
}

// One thread a node for layers of few rows and many columns (a segment's trees hold tens of thousands of columns of
// 2^8 ... 2^11 rows: a leaf is then a chain of up to 2,000 compressions on a few hundred threads, and what a thread waits for
// is the memory latency of its next sixteen column words, not the arithmetic). A warp issues in order, so a word whose column
// pointer has not arrived holds up the compression behind it: the loads therefore run two blocks deep. During the compression
// of block b the sixteen words of block b + 1 are in flight (their pointers arrived during block b - 1) and so are the sixteen
// pointers of block b + 2.
__global__ void __launch_bounds__(256) merkle_layer_prefetch_kernel(int log_size, const uint32_t* __restrict__ prev,
                                                                    const uint32_t* const* __restrict__ cols, int ncols, int m31_out,
                                                                    uint32_t* __restrict__ out) {
    const size_t n = (size_t)1 << log_size;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t h[8], m[16], nx[16];
    const uint32_t* pp[16];
    blake2s_init(h);
    const uint32_t total = (prev ? 64u : 0u) + 4u * (uint32_t)ncols;
    uint32_t t = 0;
    const int full = ncols > 0 ? (ncols - 1) / 16 : 0;  // blocks of sixteen columns that are not the last block
    if (full > 0) {
#pragma unroll
        for (int k = 0; k < 16; k++) pp[k] = cols[k];
#pragma unroll
        for (int k = 0; k < 16; k++) nx[k] = __ldg(pp[k] + i);
    }
    if (full > 1) {
#pragma unroll
        for (int k = 0; k < 16; k++) pp[k] = cols[16 + k];
    }
    if (prev) {
        const uint4* p = reinterpret_cast<const uint4*>(prev + 16 * i);
        uint4 a = p[0], b = p[1], cc = p[2], d = p[3];
        m[0] = a.x; m[1] = a.y; m[2] = a.z; m[3] = a.w; m[4] = b.x; m[5] = b.y; m[6] = b.z; m[7] = b.w;
        m[8] = cc.x; m[9] = cc.y; m[10] = cc.z; m[11] = cc.w; m[12] = d.x; m[13] = d.y; m[14] = d.z; m[15] = d.w;
        t = 64;
        blake2s_compress(h, m, t, total == 64u);
    }
    for (int b = 0; b < full; b++) {
#pragma unroll
        for (int k = 0; k < 16; k++) m[k] = nx[k];
        if (b + 1 < full) {
#pragma unroll
            for (int k = 0; k < 16; k++) nx[k] = __ldg(pp[k] + i);
        }
        if (b + 2 < full) {
            const uint32_t* const* cp = cols + 16 * (b + 2);
#pragma unroll
            for (int k = 0; k < 16; k++) pp[k] = cp[k];
        }
        t += 64;
        blake2s_compress(h, m, t, false);
    }
    const int c = 16 * full;
    if (ncols - c > 0 || total == 0u) {
        int rem = ncols - c;
#pragma unroll
        for (int k = 0; k < 16; k++) m[k] = (k < rem) ? cols[c + k][i] : 0u;
        t += 4u * (uint32_t)rem;
        blake2s_compress(h, m, t, true);
    }
    store_hash(out, i, h, m31_out != 0);
}

// A leaf layer (no children) hashed in several calls, a run of columns at a time, so that hashing can
// start while later columns are still being produced. `out` carries the chaining value between calls
// (8 words per leaf, exactly the space of the final hash). A call that is not the last one absorbs
// whole 64-byte blocks only (ncols a multiple of 16); the last call pads and finalises.
__global__ void __launch_bounds__(256) merkle_leaves_partial_kernel(int log_size, const uint32_t* const* __restrict__ cols,
                                                                    int ncols, uint32_t cols_before, int is_last, int m31_out,
                                                                    uint32_t* __restrict__ out) {
    const size_t n = (size_t)1 << log_size;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t h[8], m[16];
    uint4* o = reinterpret_cast<uint4*>(out + 8 * i);
    if (cols_before == 0) {
        blake2s_init(h);
    } else {
        uint4 a = o[0], b = o[1];
        h[0] = a.x; h[1] = a.y; h[2] = a.z; h[3] = a.w; h[4] = b.x; h[5] = b.y; h[6] = b.z; h[7] = b.w;
    }
    uint32_t t = 4u * cols_before;
    int c = 0;
    while (ncols - c > 16 || (!is_last && ncols - c == 16)) {
#pragma unroll
        for (int k = 0; k < 16; k++) m[k] = cols[c + k][i];
        c += 16;
        t += 64;
        blake2s_compress(h, m, t, false);
    }
    if (is_last) {
        int rem = ncols - c;
#pragma unroll
        for (int k = 0; k < 16; k++) m[k] = (k < rem) ? cols[c + k][i] : 0u;
        t += 4u * (uint32_t)rem;
        blake2s_compress(h, m, t, true);
        store_hash(out, i, h, m31_out != 0);
    } else {
        o[0] = make_uint4(h[0], h[1], h[2], h[3]);
        o[1] = make_uint4(h[4], h[5], h[6], h[7]);
    }
}

// The top of a tree in one launch: layers 2^(top_log-1) ... 2^0 from layer 2^top_log, nodes only
// (no columns are injected). One CTA; a barrier separates the levels.
constexpr int MERKLE_TOP_MAX_LOG = 10;
struct MerkleTopArgs { uint32_t* layer[MERKLE_TOP_MAX_LOG + 1]; };  // layer[k]: 2^k hashes


// Several consecutive layers of nodes (no columns) in one launch: a CTA takes 512 child hashes and builds up to nine levels
// above them, every level written to its own layer array and kept in shared memory for the next one. A layer of a tree is
// one compression per node whatever the launch shape; what this saves is a launch (and its drain and refill of the whole
// GPU) per layer, for the layers between the leaves and the last ten, which merkle_top_kernel builds.
constexpr int MERKLE_LEVELS_MAX = 9;
// From 2^20 children on the GPU is full with three levels of whole warps (eight, four and two of them), and the six above, where a CTA has at most
// one warp's work and waits for its latency, are left to the next launch: nine levels of 2^22 children in one launch are 227 us, 18.5 M
// hashes a ms, the first three alone 152, 24.2 M. At 2^18 the six levels as a launch of their own (12 us) cost more than they save (9).
constexpr int MERKLE_LEVELS_SPLIT_LOG = 20, MERKLE_LEVELS_SPLIT = 3;
struct MerkleLevelsArgs {
    const uint32_t* children;             // 2^child_log hashes
    uint32_t* out[MERKLE_LEVELS_MAX + 1];  // out[j]: the layer j levels above the children (2^(child_log - j) hashes), j = 1..levels
};
__global__ void __launch_bounds__(256) merkle_levels_kernel(MerkleLevelsArgs a, int levels, int m31_out) {
    __shared__ uint32_t sh[2][256][8];
    const size_t cta = blockIdx.x;
    let_next_start();
    follow_previous();
    uint32_t h[8], m[16];
    {
        blake2s_init(h);
        const uint4* p = reinterpret_cast<const uint4*>(a.children + 16 * (cta * 256 + threadIdx.x));
        uint4 x0 = p[0], x1 = p[1], x2 = p[2], x3 = p[3];
        m[0] = x0.x; m[1] = x0.y; m[2] = x0.z; m[3] = x0.w; m[4] = x1.x; m[5] = x1.y; m[6] = x1.z; m[7] = x1.w;
        m[8] = x2.x; m[9] = x2.y; m[10] = x2.z; m[11] = x2.w; m[12] = x3.x; m[13] = x3.y; m[14] = x3.z; m[15] = x3.w;
        blake2s_compress(h, m, 64u, true);
#pragma unroll
        for (int k = 0; k < 8; k++) { h[k] = m31_out ? reduce_word_m31(h[k]) : h[k]; sh[1][threadIdx.x][k] = h[k]; }
        store_hash(a.out[1], cta * 256 + threadIdx.x, h, false);
    }
    for (int j = 2; j <= levels; j++) {
        __syncthreads();
        const uint32_t n = 512u >> j;  // nodes of this level in the CTA
        if (threadIdx.x < n) {
            const uint32_t(*src)[8] = sh[(j - 1) & 1];
            blake2s_init(h);
#pragma unroll
            for (int k = 0; k < 8; k++) { m[k] = src[2 * threadIdx.x][k]; m[8 + k] = src[2 * threadIdx.x + 1][k]; }
            blake2s_compress(h, m, 64u, true);
#pragma unroll
            for (int k = 0; k < 8; k++) { h[k] = m31_out ? reduce_word_m31(h[k]) : h[k]; sh[j & 1][threadIdx.x][k] = h[k]; }
            store_hash(a.out[j], cta * n + threadIdx.x, h, false);
        }
    }
}

// Blake2sM31Channel on the device, for protocol loops whose next launch only needs a challenge
// (FRI: mix the layer's root, draw the folding challenge). State: chan[0..8) = digest, chan[8] = n_draws.
// mix_root is H(digest || root) (core/vcs/blake2_merkle.rs:53-58); draw_secure_felt is chan_step's.
__global__ void channel_mix_root_draw_kernel(uint32_t* __restrict__ chan, const uint32_t* __restrict__ root,
                                             uint32_t* __restrict__ alpha_out, uint32_t* __restrict__ root_copy) {
    __shared__ ChanSm ch;
    __shared__ uint32_t felt[4];
    const int lane = threadIdx.x;
    chan_make_schedule(ch, lane, 32);
    const uint32_t w = lane < 8 ? root[lane] : 0u;
    ch.msg[lane] = lane < 8 ? chan[lane] : 0u;
    __syncwarp();
    if (lane < 8) {
        ch.msg[8 + lane] = w;
        if (root_copy) root_copy[lane] = w;
    }
    if (lane == 0) ch.n_draws = chan[8];
    chan_step(ch, 8, 1, felt);
    if (lane < 8) chan[lane] = ch.msg[lane];
    if (lane == 8) chan[8] = ch.n_draws;
    if (lane < 4) alpha_out[lane] = felt[lane];
}

// The last (at most ten) layers of a tree in one CTA. Every level is written to its layer array and kept in shared memory
// for the next one (a level read back from global memory costs an L2 round trip on top of the compression; ten levels are a
// chain of ten dependent hashes either way, which is what bounds it). Levels of 2^8 and 2^9 nodes are a thread a node, bound by
// issue; from 2^7 down a node is a quad's (channel.cuh). When `chan` is
// given, the last warp goes on with the channel step of a FRI layer (mix the root, draw the folding challenge), which would otherwise
// be a launch of its own. Eight levels and the step: 14.0 us with the schedule looked up in shared memory and a handful of branches a level, now 12.7.
__global__ void __launch_bounds__(512, 1) merkle_top_kernel(const __grid_constant__ MerkleTopArgs a, int top_log, int m31_out, uint32_t* __restrict__ chan,
                                                         uint32_t* __restrict__ alpha_out, uint32_t* __restrict__ root_copy) {
    __shared__ alignas(16) uint32_t sh[2][256 * PAIR_WORDS];
    __shared__ ChanSm ch;
    __shared__ uint32_t felt[4];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, l = tid & 3u;
    chan_make_schedule(ch, (int)tid, (int)blockDim.x);
    let_next_start();  // one CTA: whatever comes next finds room
    follow_previous();
    if (chan && tid < 32) {
        ch.msg[tid] = tid < 8 ? chan[tid] : 0u;
        if (tid == 0) ch.n_draws = chan[8];
    }
    int lg = top_log - 1;
    if (top_log <= 8)
        for (uint32_t i = tid; i < (2u << top_log); i += blockDim.x)
            *reinterpret_cast<uint4*>(&sh[(lg + 1) & 1][(i >> 2) * PAIR_WORDS + (i & 3u) * 4u]) = reinterpret_cast<const uint4*>(a.layer[top_log])[i];
    __syncthreads();
#pragma unroll 1
    for (; lg >= 8; lg--) {
        if (tid < (1u << lg)) {
            uint32_t h[8], m[16];
            blake2s_init(h);
            const uint4* p = lg == top_log - 1 ? reinterpret_cast<const uint4*>(a.layer[lg + 1] + 16 * (size_t)tid)
                                               : reinterpret_cast<const uint4*>(&sh[(lg + 1) & 1][tid * PAIR_WORDS]);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint4 x = p[q];
                m[4 * q] = x.x; m[4 * q + 1] = x.y; m[4 * q + 2] = x.z; m[4 * q + 3] = x.w;
            }
            blake2s_compress(h, m, 64u, true);
#pragma unroll
            for (int k = 0; k < 8; k++) h[k] = m31_out ? reduce_word_m31(h[k]) : h[k];
            uint4* const o = reinterpret_cast<uint4*>(&sh[lg & 1][pair_at(tid)]);
            o[0] = make_uint4(h[0], h[1], h[2], h[3]);
            o[1] = make_uint4(h[4], h[5], h[6], h[7]);
            store_hash(a.layer[lg], tid, h, false);
        }
        __syncthreads();
    }
    // A hash's way to the next level is shared memory and a barrier; it goes to the layer's array behind that. A warp without a hash at a level
    // has none further up and leaves; quads of the last warp without one hash what is there, for nobody. (Every branch on the way is
    // some 25 cycles of a level's 1,400.)
    const QuadConst k;
    const uint32_t node = tid >> 2;
    QuadWords word(&sh[0][node * PAIR_WORDS], ch.sched);
    uint32_t* const parent = &sh[0][pair_at(node)] + l;
    if (warp * 8u >= (1u << lg)) return;
#pragma unroll 1
    while (true) {
        uint32_t* const g = a.layer[lg] + 8 * (size_t)node + l;
        uint32_t* const o = parent + (lg & 1) * (256 * PAIR_WORDS);
        const bool live = node < (1u << lg);
        word.at = ((lg + 1) & 1) * (uint32_t)sizeof(sh[0]);
        uint2 h = b2s_compress_quad(make_uint2(k.h0, k.h1), word, k, 64u, 0xffffffffu);
        if (m31_out) h = make_uint2(reduce_word_m31(h.x), reduce_word_m31(h.y));
        o[0] = h.x;
        o[4] = h.y;
        __syncthreads();
        if (live) {
            g[0] = h.x;
            g[4] = h.y;
        }
        if (--lg < 0 || warp * 8u >= (1u << lg)) break;
    }
    if (warp) return;
    if (!chan) return;
    if (lane < 8) {
        const uint32_t w = sh[0][lane];
        ch.msg[8 + lane] = w;
        if (root_copy) root_copy[lane] = w;
    }
    chan_step(ch, 8, 1, felt);
    if (lane < 8) chan[lane] = ch.msg[lane];
    if (lane == 8) chan[8] = ch.n_draws;
    if (lane < 4) alpha_out[lane] = felt[lane];
}

// Grind: thread `lo` tests nonce (hi << 32) | lo; the minimum passing lo is kept.
__global__ void grind_kernel(uint32_t d0, uint32_t d1, uint32_t d2, uint32_t d3, uint32_t d4, uint32_t d5, uint32_t d6,
                             uint32_t d7, uint32_t hi, int pow_bits, int m31_out, unsigned int* __restrict__ best) {
    uint32_t lo = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t h[8], m[16] = {d0, d1, d2, d3, d4, d5, d6, d7, lo, hi, 0, 0, 0, 0, 0, 0};
    blake2s_init(h);
    blake2s_compress(h, m, 40u, true);
    uint32_t w = m31_out ? reduce_word_m31(h[0]) : h[0];
    int tz = w ? __ffs(w) - 1 : 32;
    if (tz >= pow_bits) atomicMin(best, lo);
}

}  // namespace zk

using namespace zk;

extern "C" {

int zkb_merkle_layer(zkb_ctx* ctx, int log_size, const uint32_t* prev, const uint32_t* const* cols, int ncols,
                     int m31_out, uint32_t* out) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, log_size >= 0 && log_size <= 30 && ncols >= 0 && out != nullptr);
    ZKB_CHECK_ARG(ctx, ncols == 0 || cols != nullptr);
    ZKB_CHECK_ARG(ctx, ((uintptr_t)out & 15) == 0 && ((uintptr_t)prev & 15) == 0);
    DeviceGuard g(ctx);
    void** d_cols = nullptr;
    if (ncols) {
        int rc = stage_ptrs(ctx, (const void* const*)cols, ncols, &d_cols);
        if (rc) return rc;
    }
    const size_t n = (size_t)1 << log_size;
    if (log_size <= QUAD_MAX_LOG && ncols >= chain_min_cols(log_size)) {
        ProfScope prof(ctx, "merkle_layer_chain_kernel");
        ZKB_CUDA(ctx, launch_following(ctx, merkle_layer_chain_kernel, (unsigned)((n + CHAIN_NODES - 1) / CHAIN_NODES), CHAIN_THREADS, log_size, prev,
                                       (const uint32_t* const*)d_cols, ncols, m31_out, out));
        return ZKB_OK;
    }
    if (log_size <= QUAD_MAX_LOG) {
        // up to here there are no more than two warps of quads a scheduler, so a node's latency is what counts
        ProfScope prof(ctx, "merkle_layer_quad_kernel");
        ZKB_CUDA(ctx, launch_following(ctx, merkle_layer_quad_kernel, (unsigned)((4 * n + QUAD_THREADS - 1) / QUAD_THREADS), QUAD_THREADS, log_size, prev,
                                       (const uint32_t* const*)d_cols, ncols, m31_out, out));
        return ZKB_OK;
    }
    const unsigned threads = 256, blocks = (unsigned)(n / threads);
    if (ncols >= 64 && n <= ((size_t)1 << 17)) {
        // few rows (at 2^17 there are still only seven warps per scheduler), a long chain of compressions each: the next
        // block's loads are in flight during a compression; small CTAs so that the few rows spread over all SMs
        ProfScope prof(ctx, "merkle_layer_prefetch_kernel");
        merkle_layer_prefetch_kernel<<<(unsigned)((n + 31) / 32), 32, 0, ctx->stream>>>(log_size, prev, (const uint32_t* const*)d_cols, ncols, m31_out, out);
        ZKB_LAUNCH_CHECK(ctx);
        return ZKB_OK;
    }
    ProfScope prof(ctx, !ncols ? "merkle_layer_kernel(nodes only)" : (!prev && ncols > 16 ? "merkle_layer_kernel(leaves)" : "merkle_layer_kernel(columns)"));
    merkle_layer_kernel<<<blocks, threads, 0, ctx->stream>>>(log_size, prev, (const uint32_t* const*)d_cols, ncols, m31_out,
                                                             out);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

int zkb_merkle_leaves_partial(zkb_ctx* ctx, int log_size, const uint32_t* const* cols, int ncols, int cols_before, int total_cols,
                              int m31_out, uint32_t* out) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, log_size >= 0 && log_size <= 30 && cols != nullptr && out != nullptr && ((uintptr_t)out & 15) == 0);
    ZKB_CHECK_ARG(ctx, ncols >= 1 && cols_before >= 0 && cols_before % 16 == 0 && cols_before + ncols <= total_cols);
    const bool is_last = cols_before + ncols == total_cols;
    ZKB_CHECK_ARG(ctx, is_last || ncols % 16 == 0);
    DeviceGuard g(ctx);
    void** d_cols = nullptr;
    int rc = stage_ptrs(ctx, (const void* const*)cols, ncols, &d_cols);
    if (rc) return rc;
    size_t n = (size_t)1 << log_size;
    unsigned threads = n < 256 ? 32 : 256;
    ProfScope prof(ctx, "merkle_leaves_partial_kernel");
    merkle_leaves_partial_kernel<<<(unsigned)((n + threads - 1) / threads), threads, 0, ctx->stream>>>(
        log_size, (const uint32_t* const*)d_cols, ncols, (uint32_t)cols_before, is_last ? 1 : 0, m31_out, out);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

int zkb_merkle_levels(zkb_ctx* ctx, int child_log, const uint32_t* children, int levels, uint32_t* const* out_layers, int m31_out) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, children != nullptr && out_layers != nullptr && ((uintptr_t)children & 15) == 0);
    ZKB_CHECK_ARG(ctx, levels >= 1 && levels <= MERKLE_LEVELS_MAX && child_log >= 9 && child_log <= 31 && child_log - levels >= 0);
    for (int j = 1; j <= levels; j++) ZKB_CHECK_ARG(ctx, out_layers[j - 1] != nullptr && ((uintptr_t)out_layers[j - 1] & 15) == 0);
    DeviceGuard g(ctx);
    for (int done = 0; done < levels;) {
        const int log = child_log - done, left = levels - done, take = log >= MERKLE_LEVELS_SPLIT_LOG ? std::min(left, MERKLE_LEVELS_SPLIT) : left;
        MerkleLevelsArgs a{};
        a.children = done ? out_layers[done - 1] : children;
        for (int j = 1; j <= take; j++) a.out[j] = out_layers[done + j - 1];
        ProfScope prof(ctx, "merkle_levels_kernel");
        ZKB_CUDA(ctx, launch_following(ctx, merkle_levels_kernel, 1u << (log - 9), 256u, a, take, m31_out));
        done += take;
    }
    return ZKB_OK;
}

static int merkle_top_impl(zkb_ctx* ctx, int top_log, const uint32_t* top_layer, uint32_t* const* lower_layers, int m31_out, uint32_t* d_chan,
                           uint32_t* d_alpha, uint32_t* d_root_copy);
int zkb_merkle_top(zkb_ctx* ctx, int top_log, const uint32_t* top_layer, uint32_t* const* lower_layers, int m31_out) {
    return merkle_top_impl(ctx, top_log, top_layer, lower_layers, m31_out, nullptr, nullptr, nullptr);
}
int zkb_merkle_top_channel(zkb_ctx* ctx, int top_log, const uint32_t* top_layer, uint32_t* const* lower_layers, int m31_out, uint32_t* d_chan,
                           uint32_t* d_alpha, uint32_t* d_root_copy) {
    if (ctx && (!d_chan || !d_alpha || top_log < 1)) return zk::set_error(ctx, ZKB_EINVAL, "zkb_merkle_top_channel: needs a channel, a challenge slot and at least one layer to build");
    return merkle_top_impl(ctx, top_log, top_layer, lower_layers, m31_out, d_chan, d_alpha, d_root_copy);
}
static int merkle_top_impl(zkb_ctx* ctx, int top_log, const uint32_t* top_layer, uint32_t* const* lower_layers, int m31_out, uint32_t* d_chan,
                           uint32_t* d_alpha, uint32_t* d_root_copy) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, top_log >= 0 && top_log <= MERKLE_TOP_MAX_LOG && top_layer != nullptr && ((uintptr_t)top_layer & 15) == 0);
    if (top_log == 0) return ZKB_OK;
    ZKB_CHECK_ARG(ctx, lower_layers != nullptr);
    MerkleTopArgs a;
    a.layer[top_log] = const_cast<uint32_t*>(top_layer);
    for (int k = 0; k < top_log; k++) {
        ZKB_CHECK_ARG(ctx, lower_layers[k] != nullptr && ((uintptr_t)lower_layers[k] & 15) == 0);
        a.layer[k] = lower_layers[k];
    }
    DeviceGuard g(ctx);
    ProfScope prof(ctx, "merkle_top_kernel");
    ZKB_CUDA(ctx, launch_following(ctx, merkle_top_kernel, 1u, top_log >= 8 ? 512u : (unsigned)std::max(2 << top_log, 32), a, top_log, m31_out, d_chan, d_alpha, d_root_copy));
    return ZKB_OK;
}

int zkb_channel_mix_root_draw(zkb_ctx* ctx, uint32_t* d_chan, const uint32_t* d_root, uint32_t* d_alpha, uint32_t* d_root_copy) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, d_chan != nullptr && d_root != nullptr && d_alpha != nullptr);
    DeviceGuard g(ctx);
    ProfScope prof(ctx, "channel_mix_root_draw_kernel");
    channel_mix_root_draw_kernel<<<1, 32, 0, ctx->stream>>>(d_chan, d_root, d_alpha, d_root_copy);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

int zkb_grind(zkb_ctx* ctx, const uint32_t h_prefixed_digest[8], int pow_bits, int m31_out, uint64_t* h_nonce) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, h_prefixed_digest != nullptr && h_nonce != nullptr && pow_bits >= 0 && pow_bits <= 32);
    DeviceGuard g(ctx);
    const uint32_t* d = h_prefixed_digest;
    const unsigned LOW = 1u << 20;
    if (pow_bits == 0) {  // every nonce passes
        *h_nonce = 0;
        return ZKB_OK;
    }
    // Half of the first 2^20 nonces already pass a few bits: a first launch over 2^(pow_bits + 4) of them finds the smallest in all
    // but one case in nine million; the whole search follows otherwise.
    unsigned first = pow_bits + 4 < 12 ? 1u << 12 : pow_bits + 4 < 20 ? 1u << (pow_bits + 4) : LOW;
    // Bounded search: hi values are tried in order; a miss over 2^20 nonces has probability
    // (1 - 2^-pow_bits)^(2^20), so the bound of 2^12 rounds is never reached for pow_bits <= 32
    // in practice and keeps the loop finite.
    for (uint32_t hi = 0; hi < (1u << 12);) {
        ZKB_CUDA(ctx, cudaMemsetAsync(ctx->ticket + 8, 0xff, 4, ctx->stream));
        grind_kernel<<<first / 256, 256, 0, ctx->stream>>>(d[0], d[1], d[2], d[3], d[4], d[5], d[6], d[7], hi, pow_bits,
                                                         m31_out, ctx->ticket + 8);
        ZKB_LAUNCH_CHECK(ctx);
        ZKB_CUDA(ctx, cudaMemcpyAsync(ctx->h_small, ctx->ticket + 8, 4, cudaMemcpyDeviceToHost, ctx->stream));
        ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        const unsigned int best = ctx->h_small[0];
        if (best != 0xffffffffu) {
            *h_nonce = ((uint64_t)hi << 32) | best;
            return ZKB_OK;
        }
        if (first == LOW) hi++;
        first = LOW;
    }
    return set_error(ctx, ZKB_ETIMEOUT, "zkb_grind: no nonce found in 2^32 attempts");
}

}  // extern "C"
