// The last layers of a FRI commitment (FriProver::commit, nitroo/crates/stwo/src/prover/fri.rs:109-221), from a layer of at most
// 2^10 values down to the last one, in ONE launch of one CTA: per layer the leaf hashes, the tree, the channel step on its root
// (mix, draw the folding challenge) and the fold.
//
// What bounds it: dependency depth. A layer of 2^l values is a chain of l + 1 tree levels and two channel compressions, each some
// 0.75 us; at 2^10 values the leaves and the level above them are another 9 us of one SM's hashing. Levels of up to 2^7 hashes are
// four lanes a hash, their message's addresses in registers and no branch but the loop's on a hash's way to the next level: eight layers from
// 2^10 values 91 -> 86 us. As launches (fold and leaves, tree
// top with channel step) a layer also paid two launches, the gaps around them and a dozen allocations for its arrays: a ten-column
// proof of 2^8 rows spent 190 us of device time in them and as much on the host. Layers stay in shared memory; what the decommitment
// reads later (trees, folded layers) is written to memory on the side. Above 2^10 values a layer has enough hashes for more SMs: fri_mid_kernel below.
#include <cstdlib>
#include <cstring>

#include "channel.cuh"
#include "common.cuh"
#include "fri_tail.hpp"

namespace zk {

constexpr int TAIL_THREADS = 512;
constexpr size_t TAIL_N = (size_t)1 << FRI_TAIL_LOG;
static_assert(TAIL_N / 2 <= TAIL_THREADS && TAIL_N >= 256, "a layer folds to at most a value a thread; the messages of 128 quads have room");

__device__ __forceinline__ uint32_t bitrev_bits(uint32_t i, int bits) { return bits ? __brev(i) >> (32 - bits) : 0u; }

// Dynamic shared memory: two layers of values, word by word, and two of hashes, pair by pair (pair_at).
constexpr size_t TAIL_PAIRS = TAIL_N / 2 * PAIR_WORDS, TAIL_SMEM = (2 * 4 * TAIL_N + 2 * TAIL_PAIRS) * 4;

// The levels lv ... 0 of a tree, or of a subtree, by a CTA of TAIL_THREADS: leaves from ev where lv is leaf_lv (coordinate c of leaf i at ev[c * ev_stride + i]), else nodes of the
// pairs at `below`, which is ha or hb; one loop, so that the code of the hash is there once. Hash i of a level goes to out(level) + 8 i too. Returns
// where warp 0 finds the root; the other warps may still be on their way.
template <class Out>
__device__ __forceinline__ uint32_t* hash_levels(uint32_t* const ha, uint32_t* const hb, uint32_t* below, const uint32_t* ev, size_t ev_stride, int lv, int leaf_lv, QuadWords& word,
                                                 const QuadConst& qc, Out out) {
    const int tid = threadIdx.x, warp = tid >> 5, l = tid & 3, quad = tid >> 2;
    uint32_t* cur = below == ha ? hb : ha;
    auto leaf_word = [&](int c, uint32_t i) { return ev[c * ev_stride + i]; };
#pragma unroll 1
    for (; lv >= 8; lv--) {
        uint32_t* const o_level = out(lv);
        const bool leaf = lv == leaf_lv;
        for (uint32_t i = tid; i < (1u << lv); i += TAIL_THREADS) {
            uint32_t h[8], m[16];
            blake2s_init(h);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                uint4 x = make_uint4(0u, 0u, 0u, 0u);
                if (!leaf) x = *reinterpret_cast<const uint4*>(below + PAIR_WORDS * i + 4 * q);
                else if (q == 0) x = make_uint4(leaf_word(0, i), leaf_word(1, i), leaf_word(2, i), leaf_word(3, i));
                m[4 * q] = x.x; m[4 * q + 1] = x.y; m[4 * q + 2] = x.z; m[4 * q + 3] = x.w;
            }
            blake2s_compress(h, m, leaf ? 16u : 64u, true);
#pragma unroll
            for (int w = 0; w < 8; w++) h[w] = reduce_word_m31(h[w]);
            const uint4 lo = make_uint4(h[0], h[1], h[2], h[3]), hi = make_uint4(h[4], h[5], h[6], h[7]);
            uint4 *const c = reinterpret_cast<uint4*>(cur + pair_at(i)), *const o = reinterpret_cast<uint4*>(o_level + 8 * (size_t)i);
            c[0] = o[0] = lo;
            c[1] = o[1] = hi;
        }
        uint32_t* const swap = cur;
        cur = below;
        below = swap;
        __syncthreads();
    }
    // From 2^7 hashes down four lanes a hash, as in merkle_top_kernel; warps that have one meet at a barrier of their own, the others wait for
    // the challenge.
    if (lv == leaf_lv && 8 * warp < (1 << lv)) {
        const uint32_t i = quad < (1 << lv) ? quad : 0;
        *reinterpret_cast<uint4*>(below + PAIR_WORDS * quad + 4 * l) = l ? make_uint4(0u, 0u, 0u, 0u) : make_uint4(leaf_word(0, i), leaf_word(1, i), leaf_word(2, i), leaf_word(3, i));
        __syncwarp();
    }
    if (8 * warp < (1 << lv)) {
        uint32_t* const parent = ha + pair_at(quad) + l;
        const uint32_t apart = (uint32_t)(hb - ha);
        uint32_t side = below == ha ? 0u : 1u;  // which of the two the messages are in
#pragma unroll 1
        while (true) {
            uint32_t* const o = out(lv) + 8 * quad + l;
            const bool live = quad < (1 << lv);
            const int meet = lv >= 3 ? 4 << lv : 32;
            word.at = side * (apart * 4u);
            side ^= 1u;
            uint32_t* const c = parent + side * apart;
            uint2 h = b2s_compress_quad(make_uint2(qc.h0, qc.h1), word, qc, lv == leaf_lv ? 16u : 64u, 0xffffffffu);
            h = make_uint2(reduce_word_m31(h.x), reduce_word_m31(h.y));
            c[0] = h.x;
            c[4] = h.y;
            asm volatile("bar.sync 1, %0;" ::"r"(meet) : "memory");
            if (live) {
                o[0] = h.x;
                o[4] = h.y;
            }
            if (--lv < 0 || 8 * warp >= (1 << lv)) break;
        }
        below = side ? hb : ha;
    }
    return below;
}

__global__ void __launch_bounds__(TAIL_THREADS, 1) fri_tail_kernel(const __grid_constant__ FriTailArgs a, const uint32_t* __restrict__ itw) {
    extern __shared__ uint32_t dyn[];
    __shared__ ChanSm ch;
    __shared__ uint32_t alpha_w[4];
    uint32_t *ev = dyn, *ev_next = ev + 4 * TAIL_N, *const ha = ev_next + 4 * TAIL_N, *const hb = ha + TAIL_PAIRS;
    const int tid = threadIdx.x, lane = tid & 31, quad = tid >> 2;
    const QuadConst qc;
    chan_make_schedule(ch, tid, TAIL_THREADS);
    if (tid < 32) ch.msg[tid] = tid < 8 ? (a.chan ? a.chan[tid] : a.digest[tid]) : 0u;
    if (tid == 0) ch.n_draws = a.chan ? a.chan[8] : a.n_draws;
    for (int i = tid; i < 4 << a.first_log; i += TAIL_THREADS) {
        const int c = i >> a.first_log, r = i & ((1 << a.first_log) - 1);
        ev[c * TAIL_N + r] = a.src[c][r];
    }
    __syncthreads();
    QuadWords word(ha + PAIR_WORDS * quad, ch.sched);
    for (int k = 0; k < a.n_layers; k++) {
        const int log = a.first_log - k;
        // the fold's twiddle (a layer folds to at most a value a thread) is on its way while the tree is hashed
        const uint32_t half = 1u << (log - 1), mine = (uint32_t)tid < half ? (uint32_t)tid : 0u;
        uint32_t t, ix;
        if (a.circle && k == 0) half_coset_point(itw, log, mine, ix, t);
        else t = itw[half + mine];  // T_log^-1 starts at 2^(log - 1)
        const uint32_t* const below = hash_levels(ha, hb, hb, ev, TAIL_N, log, log, word, qc, [&](int lv) { return a.tree[k] + ((size_t)8 << lv); });
        // the root is in warp 0's below[0, 8): mix it in, draw the challenge
        if (tid < 32) {
            if (lane < 8) {
                const uint32_t w = below[lane];
                ch.msg[8 + lane] = w;
                a.out[FRI_TAIL_ROOTS + 8 * k + lane] = w;
            }
            chan_step(ch, 8, 1, alpha_w);
        }
        __syncthreads();
        const qm31 alpha{{alpha_w[0], alpha_w[1], alpha_w[2], alpha_w[3]}};
        const size_t stride = log - 1 < 2 ? 4 : half;
        if ((uint32_t)tid < half) {
            const uint32_t i = (uint32_t)tid;
            qm31 x, y;
#pragma unroll
            for (int c = 0; c < 4; c++) { x.c[c] = ev[c * TAIL_N + 2 * i]; y.c[c] = ev[c * TAIL_N + 2 * i + 1]; }
            const qm31 r = qm31_add(qm31_add(x, y), qm31_mul(alpha, qm31_mul_m31(qm31_sub(x, y), t)));
#pragma unroll
            for (int c = 0; c < 4; c++) { ev_next[c * TAIL_N + i] = r.c[c]; a.evals[k][c * stride + i] = r.c[c]; }
        }
        uint32_t* const swap = ev;
        ev = ev_next;
        ev_next = swap;
        __syncthreads();
    }
    if (tid >= 32) return;
    uint32_t too_high = 0u;
    if (a.last_bound >= 0) {
        // commit_last_layer (fri.rs:193-221): interpolate on the line domain of last_log, value `lane` of the natural order per lane
        const int log = a.last_log, lb = a.last_bound;
        const uint32_t n = 1u << log, pos = bitrev_bits((uint32_t)lane & (n - 1), log);
        qm31 v;
#pragma unroll
        for (int c = 0; c < 4; c++) v.c[c] = ev[c * TAIL_N + pos];
        for (int k = log; k > 0; k--) {
            const uint32_t half = 1u << (k - 1), p = (uint32_t)lane & (2 * half - 1);
            const bool low = p < half;
            qm31 o;
#pragma unroll
            for (int c = 0; c < 4; c++) o.c[c] = __shfl_xor_sync(0xffffffffu, v.c[c], half);
            const uint32_t xinv = itw[half + bitrev_bits(p & (half - 1), k - 1)];
            v = low ? qm31_add(v, o) : qm31_mul_m31(qm31_sub(o, v), xinv);
        }
        v = qm31_mul_m31(v, m31_inv(n));
        // lane l holds the coefficient at bitrev(l) of the bit-reversed order, of which only the first 2^lb may be non-zero
        const uint32_t j = pos;
        too_high = __any_sync(0xffffffffu, (uint32_t)lane < n && j >= (1u << lb) && !qm31_is_zero(v)) ? 1u : 0u;
        const uint32_t slot = bitrev_bits(j & ((1u << lb) - 1), lb);
        if ((uint32_t)lane < n && j < (1u << lb)) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                ch.msg[8 + 4 * slot + c] = v.c[c];
                a.out[32 + 4 * slot + c] = v.c[c];
            }
        }
        chan_step(ch, 4 << lb, 0, alpha_w);
        // the digest a proof of work is searched for: H(prefix, 12 zero bytes, digest, pow_bits), channel/blake2s.rs:124-133
        const uint32_t d = lane < 8 ? ch.msg[lane] : 0u;
        const uint32_t shifted = __shfl_sync(0xffffffffu, d, (lane - 4) & 31);
        uint32_t* const block = ch.msg + 16;
        if (lane < 16) block[lane] = lane == 0 ? 0x12345678u : lane < 4 ? 0u : lane < 12 ? shifted : lane == 12 ? a.pow_bits : 0u;
        __syncwarp();
        const QuadConst q;
        const uint2 h = b2s_compress_quad(make_uint2(q.h0, q.h1), ScheduledWords{block, ch.sched}, q, 52u, 0xffffffffu);
        if (lane < 4) { a.out[16 + lane] = reduce_word_m31(h.x); a.out[20 + lane] = reduce_word_m31(h.y); }
    }
    if (lane < 8) a.out[lane] = ch.msg[lane];
    if (lane == 8) a.out[8] = ch.n_draws;
    if (lane == 9) a.out[9] = too_high;
    if (lane == 10) a.out[10] = 0xffffffffu;
}

// The layers above those, of up to 2^FRI_MID_LOG values, in one cooperative launch of 32 CTAs. A fold takes neighbouring values, so a CTA keeps its slice of
// the values from layer to layer in shared memory and hashes the subtree above it; what goes round in a layer is the subtrees' roots, to CTA 0, and the
// challenge back, both with a bit in every word that says that it is there (words of a hash and coordinates are below 2^31; the bit's value changes with
// every use of the slot): neither waits for a fence or a count. CTA 0 hashes the levels above the subtrees and keeps the channel.
//
// As launches (fold and leaves, levels, top with the channel step) a layer of 2^11 ... 2^15 values took 16-24 us, whose chain of hashes is
// 9-12; a proof of four columns, domain 2^14: 470 us before, 428 with this launch. The waits end: every CTA is resident (the launch is refused otherwise), a wait is for what the others do before their own, and after MID_SPINS
// polls (a second) a CTA leaves, with the channel's failed word set: after the last challenge nobody waits for it any more, and CTA 0 may end well.
constexpr uint32_t MID_SPINS = 1u << 21;
constexpr size_t MID_N = (size_t)1 << (FRI_MID_LOG - FRI_MID_CTAS_LOG), MID_PAIRS = MID_N / 2 * PAIR_WORDS, MID_SMEM = (2 * 4 * MID_N + 2 * MID_PAIRS) * 4;  // the largest slice
static_assert(MID_N / 2 <= TAIL_THREADS && MID_N >= 256 && ((size_t)1 << FRI_MID_CTAS_LOG) <= MID_N, "a slice folds to at most a value a thread; quads and roots have room");
__device__ __forceinline__ bool mid_wait(const uint32_t* slot, uint32_t there, uint32_t polls, uint32_t& w) {
    for (uint32_t spin = 0; spin < polls; spin++) {
        w = *reinterpret_cast<const volatile uint32_t*>(slot);
        if (w >> 31 == there) {
            w &= 0x7fffffffu;
            return true;
        }
    }
    return false;
}
__global__ void __launch_bounds__(TAIL_THREADS, 1) fri_mid_kernel(const __grid_constant__ FriMidArgs a, const uint32_t* __restrict__ itw) {
    extern __shared__ uint32_t dyn[];
    __shared__ ChanSm ch;
    __shared__ uint32_t alpha_w[4];
    __shared__ bool gave_up;
    uint32_t *ev = dyn, *ev_next = ev + 4 * MID_N, *const ha = ev_next + 4 * MID_N, *const hb = ha + MID_PAIRS;
    const uint32_t tid = threadIdx.x, lane = tid & 31, cta = blockIdx.x, ctas = 1u << FRI_MID_CTAS_LOG;
    const QuadConst qc;
    chan_make_schedule(ch, (int)tid, TAIL_THREADS);
    if (tid == 0) gave_up = false;
    if (cta == 0) {
        if (tid < 32) ch.msg[tid] = tid < 8 ? a.chan[tid] : 0u;
        if (tid == 0) ch.n_draws = a.chan[8];
    }
    int slice_log = a.first_log - FRI_MID_CTAS_LOG;
    for (uint32_t i = tid; i < 4u << slice_log; i += TAIL_THREADS) {
        const uint32_t c = i >> slice_log, r = i & ((1u << slice_log) - 1);
        ev[c * MID_N + r] = a.src[c][((size_t)cta << slice_log) + r];
    }
    __syncthreads();
    QuadWords word(ha + PAIR_WORDS * (tid >> 2), ch.sched);
    for (int k = 0; k < a.n_layers; k++, slice_log--) {
        const int log = a.first_log - k;
        const uint32_t there = (k >> 1 & 1) ^ 1u;
        uint32_t *const root_slots = a.sync + (size_t)(k & 1) * 8 * ctas, *const alpha_slot = a.sync + 16 * ctas + 4 * (k & 1);
        const uint32_t half = 1u << (slice_log - 1), mine = tid < half ? tid : 0u, fold_at = (cta << (slice_log - 1)) + mine;
        uint32_t t, ix;
        if (a.circle && k == 0) half_coset_point(itw, log, fold_at, ix, t);
        else t = itw[(1u << (log - 1)) + fold_at];
        const uint32_t* below = hash_levels(ha, hb, hb, ev, MID_N, slice_log, slice_log, word, qc,
                                            [&](int lv) { return a.tree[k] + ((size_t)8 << (lv + FRI_MID_CTAS_LOG)) + (((size_t)8 * cta) << lv); });
        if (tid < 8) *reinterpret_cast<volatile uint32_t*>(root_slots + 8 * cta + tid) = below[tid] | there << 31;
        if (cta == 0) {
            __syncthreads();
            for (uint32_t i = tid; i < 8 * ctas; i += TAIL_THREADS) {
                uint32_t w = 0;
                if (!mid_wait(root_slots + i, there, MID_SPINS, w)) gave_up = true;
                ha[pair_at(i >> 3) + (i & 7u)] = w;
            }
            __syncthreads();
            if (gave_up) break;
            below = hash_levels(ha, hb, ha, ev, MID_N, FRI_MID_CTAS_LOG - 1, -1, word, qc, [&](int lv) { return a.tree[k] + ((size_t)8 << lv); });
            if (tid < 32) {
                if (lane < 8) {
                    const uint32_t w = below[lane];
                    ch.msg[8 + lane] = w;
                    a.roots[8 * k + lane] = w;
                }
                chan_step(ch, 8, 1, alpha_w);
                if (lane < 4) *reinterpret_cast<volatile uint32_t*>(alpha_slot + lane) = alpha_w[lane] | there << 31;
            }
        } else if (tid < 4) {
            uint32_t w = 0;
            if (!mid_wait(alpha_slot + tid, there, a.impatient ? 0u : MID_SPINS, w)) gave_up = true;
            alpha_w[tid] = w;
        }
        __syncthreads();
        if (gave_up) break;
        const qm31 alpha{{alpha_w[0], alpha_w[1], alpha_w[2], alpha_w[3]}};
        if (tid < half) {
            qm31 x, y;
#pragma unroll
            for (int c = 0; c < 4; c++) { x.c[c] = ev[c * MID_N + 2 * tid]; y.c[c] = ev[c * MID_N + 2 * tid + 1]; }
            const qm31 r = qm31_add(qm31_add(x, y), qm31_mul(alpha, qm31_mul_m31(qm31_sub(x, y), t)));
#pragma unroll
            for (int c = 0; c < 4; c++) { ev_next[c * MID_N + tid] = r.c[c]; a.evals[k][((size_t)c << (log - 1)) + fold_at] = r.c[c]; }
        }
        uint32_t* const swap = ev;
        ev = ev_next;
        ev_next = swap;
        __syncthreads();
    }
    if (gave_up && tid == 0) a.chan[FRI_MID_FAILED] = 1u;
    if (gave_up || cta || tid >= 32) return;
    if (lane < 8) a.chan[lane] = ch.msg[lane];
    if (lane == 8) a.chan[8] = ch.n_draws;
    if (lane == FRI_MID_DONE) a.chan[FRI_MID_DONE] = 1u;
}

__global__ void __launch_bounds__(256) grind_first_kernel(const uint32_t* __restrict__ prefixed, int pow_bits, unsigned int* __restrict__ best) {
    const uint32_t lo = blockIdx.x * 256u + threadIdx.x;
    uint32_t h[8], m[16];
#pragma unroll
    for (int w = 0; w < 16; w++) m[w] = w < 8 ? prefixed[w] : 0u;
    m[8] = lo;
    blake2s_init(h);
    blake2s_compress(h, m, 40u, true);
    const uint32_t w = reduce_word_m31(h[0]);
    const int tz = w ? __ffs(w) - 1 : 32;
    if (tz >= pow_bits) atomicMin(best, lo);
}

int fri_tail(zkb_ctx* ctx, const FriTailArgs& args) {
    ZKB_CHECK_ARG(ctx, args.n_layers >= 1 && args.first_log <= FRI_TAIL_LOG && args.first_log - args.n_layers >= 0);
    ZKB_CHECK_ARG(ctx, args.first_log <= ctx->max_log - (args.circle ? 0 : 1));
    ZKB_CHECK_ARG(ctx, !args.circle || args.first_log >= 3);
    ZKB_CHECK_ARG(ctx, args.last_bound < 0 || (args.last_log == args.first_log - args.n_layers && args.last_log <= FRI_TAIL_MAX_LAST &&
                                              args.last_bound <= FRI_TAIL_MAX_BOUND && args.last_bound <= args.last_log));
    DeviceGuard g(ctx);
    if (!ctx->fri_tail_ready) {
        ZKB_CUDA(ctx, cudaFuncSetAttribute(fri_tail_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TAIL_SMEM));
        ctx->fri_tail_ready = true;
    }
    ProfScope prof(ctx, "fri_tail_kernel");
    fri_tail_kernel<<<1, TAIL_THREADS, TAIL_SMEM, ctx->stream>>>(args, ctx->itw);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

int fri_mid(zkb_ctx* ctx, FriMidArgs args) {
    ZKB_CHECK_ARG(ctx, args.n_layers >= 1 && args.n_layers <= FRI_MID_LOG - FRI_MID_END && args.first_log <= FRI_MID_LOG && args.first_log - args.n_layers >= FRI_MID_END);
    ZKB_CHECK_ARG(ctx, args.first_log <= ctx->max_log - (args.circle ? 0 : 1));
    const char* const env = getenv("ZKB_FRI_MID");  // to be tried: as though the launch were refused; CTAs that give up at once
    if (env && !strcmp(env, "refused")) return FRI_MID_REFUSED;
    args.impatient = env && !strcmp(env, "impatient");
    DeviceGuard g(ctx);
    if (!ctx->fri_mid_ready) {
        ZKB_CUDA(ctx, cudaFuncSetAttribute(fri_mid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MID_SMEM));
        ctx->fri_mid_ready = true;
    }
    ProfScope prof(ctx, "fri_mid_kernel");
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;  // every CTA is resident, or the launch fails
    attr[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1u << FRI_MID_CTAS_LOG);
    cfg.blockDim = dim3(TAIL_THREADS);
    cfg.dynamicSmemBytes = MID_SMEM;
    cfg.stream = ctx->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, fri_mid_kernel, args, (const uint32_t*)ctx->itw);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        (void)cudaGetLastError();
        return FRI_MID_REFUSED;
    }
    ZKB_CUDA(ctx, e);
    return ZKB_OK;
}

int grind_first(zkb_ctx* ctx, const uint32_t* prefixed, int pow_bits, uint32_t* best) {
    // 2^(pow_bits + 4) nonces all fail with probability e^-16; zkb_grind then searches from the start
    const int log = pow_bits + 4 < 12 ? 12 : pow_bits + 4 > 20 ? 20 : pow_bits + 4;
    DeviceGuard g(ctx);
    ProfScope prof(ctx, "grind_kernel");
    grind_first_kernel<<<1u << (log - 8), 256, 0, ctx->stream>>>(prefixed, pow_bits, best);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

int read_small(zkb_ctx* ctx, const uint32_t* d, size_t words, const uint32_t** h) {
    ZKB_CHECK_ARG(ctx, words <= (size_t)SMALL_WORDS);
    DeviceGuard g(ctx);
    ZKB_CUDA(ctx, cudaMemcpyAsync(ctx->h_small, d, words * 4, cudaMemcpyDeviceToHost, ctx->stream));
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *h = ctx->h_small;
    return ZKB_OK;
}

}  // namespace zk
