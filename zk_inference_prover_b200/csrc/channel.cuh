// The Fiat-Shamir channel (Blake2sM31Channel, core/channel/blake2s.rs:20-141) run by ONE WARP on state in shared memory,
// for kernels that keep a protocol's transcript on the device.
//
// What bounds it: a compression is a chain of 240 dependent instructions (ten rounds of two G functions), so a transcript
// step is latency, not throughput. One thread that runs the four G functions of a half-round itself is limited by the
// issue of its 1,086 instructions and, in a launch that has not hashed before, by fetching them: 5,300 cycles measured for a
// first compression, 1,675 for the later ones. Here a compression is spread over the four lanes of a quad (all eight quads of
// the warp do the same, so nothing diverges), one column or diagonal each. Between the column and the diagonal step the lanes
// keep their `b` word and exchange a, c and d: those are final two to five instructions before b is, so most of the
// exchange's latency is hidden behind the end of the G function. Measured: 1,690 cycles for the first compression of a
// launch, 1,530-1,560 for the later ones. (An earlier form that moved b and looked the schedule up in constant memory, which a
// warp's lanes read at four addresses each, took 3,500.)
#pragma once
#include "blake2s.cuh"

namespace zk {

__constant__ uint8_t c_chan_sigma[10][16] = {
    {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15}, {14, 10, 4, 8, 9, 15, 13, 6, 1, 12, 0, 2, 11, 7, 5, 3},
    {11, 8, 12, 0, 5, 2, 15, 13, 10, 14, 3, 6, 7, 1, 9, 4}, {7, 9, 3, 1, 13, 12, 11, 14, 2, 6, 5, 10, 4, 0, 15, 8},
    {9, 0, 5, 7, 2, 4, 10, 15, 14, 1, 11, 12, 6, 8, 3, 13}, {2, 12, 6, 10, 0, 11, 8, 3, 4, 13, 7, 5, 15, 14, 1, 9},
    {12, 5, 1, 15, 14, 13, 4, 10, 0, 7, 6, 3, 9, 2, 8, 11}, {13, 11, 7, 14, 12, 1, 3, 9, 5, 0, 15, 4, 8, 6, 2, 10},
    {6, 15, 14, 9, 11, 3, 0, 8, 12, 2, 13, 7, 1, 4, 10, 5}, {10, 2, 8, 4, 7, 6, 1, 5, 15, 11, 9, 14, 3, 12, 13, 0}};

struct alignas(16) ChanSm {
    uint32_t sched[40];  // [round][lane of the quad]: byte offsets into the block of the lane's four words (column x, y, diagonal x, y)
    uint32_t msg[32];    // the message of the hash in flight: digest first, then the words mixed in, zero padded to whole blocks
    uint32_t n_draws, pad[7];
};

// Any set of threads; a barrier (of the warp or the CTA, whichever called) must follow.
__device__ __forceinline__ void quad_make_schedule(uint32_t* sched, int thread, int n_threads) {
    for (int t = thread; t < 40; t += n_threads) {
        const uint8_t* sg = c_chan_sigma[t >> 2];
        const int l = t & 3, g = (l + 3) & 3;  // in the diagonal step the lane that keeps v[4 + l] runs diagonal l - 1
        sched[t] = 4u * sg[2 * l] | (4u * sg[2 * l + 1]) << 8 | (4u * sg[8 + 2 * g]) << 16 | (4u * sg[9 + 2 * g]) << 24;
    }
}

__device__ __forceinline__ void chan_make_schedule(ChanSm& s, int thread, int n_threads) { quad_make_schedule(s.sched, thread, n_threads); }

// Where a lane finds its message words, in the order it takes them (word 4 r + u is the u-th of round r). By the schedule in shared memory,
// wherever the message is:
struct ScheduledWords {
    const uint32_t *m, *sched;
    __device__ __forceinline__ uint32_t operator()(int i) const {
        const uint32_t off = sched[(i & ~3) + (threadIdx.x & 3)] >> (8 * (i & 3)) & 255u;
        return *reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(m) + off);
    }
};
// By addresses in registers, for a kernel whose quads keep to one place, or to places `at` bytes apart: an instruction and a load less a word,
// and forty registers.
struct QuadWords {
    uint32_t address[40], at = 0;
    // sched: quad_make_schedule's, behind a barrier
    __device__ __forceinline__ QuadWords(const uint32_t* m, const uint32_t* sched) {
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(m);
#pragma unroll
        for (int r = 0; r < 10; r++) {
            const uint32_t pk = sched[4 * r + (threadIdx.x & 3)];
#pragma unroll
            for (int u = 0; u < 4; u++) address[4 * r + u] = base + ((pk >> (8 * u)) & 255u);
        }
    }
    __device__ __forceinline__ uint32_t operator()(int i) const { return *reinterpret_cast<const uint32_t*>(__cvta_shared_to_generic(address[i] + at)); }
};

// Where quads keep hashes of a tree level in shared memory: a pair of siblings is the 16-word message of their parent, the pairs are 20
// words apart (16-byte aligned, and the eight quads of a warp read their messages from different banks).
constexpr int PAIR_WORDS = 20;
__device__ __forceinline__ uint32_t pair_at(uint32_t node) { return (node >> 1) * PAIR_WORDS + (node & 1u) * 8u; }

// What a lane of the quad knows of the hash for good: its words of the initial state, and masks for the byte count and the last flag.
struct QuadConst {
    uint32_t h0, h1, c, d, t_mask, last_mask;
    __device__ __forceinline__ QuadConst() {
        const int l = threadIdx.x & 3;
        c = l == 0 ? B2S_IV0 : l == 1 ? B2S_IV1 : l == 2 ? B2S_IV2 : B2S_IV3;
        d = l == 0 ? B2S_IV4 : l == 1 ? B2S_IV5 : l == 2 ? B2S_IV6 : B2S_IV7;
        h0 = l == 0 ? (B2S_IV0 ^ 0x01010020u) : c;
        h1 = d;
        t_mask = l == 0 ? 0xffffffffu : 0u;
        last_mask = l == 2 ? 0xffffffffu : 0u;
    }
};

// Warp-collective compression: lane l of every quad holds h[l] in .x and h[4 + l] in .y. last: all ones for the last block.
template <class Words>
__device__ __forceinline__ uint2 b2s_compress_quad(uint2 h, const Words& word, const QuadConst& k, uint32_t t, uint32_t last) {
    const unsigned full = 0xffffffffu;
    const int l = threadIdx.x & 3, q = threadIdx.x & 28;
    const int up = q | ((l + 3) & 3), dn = q | ((l + 1) & 3);
    uint32_t a = h.x, b = h.y, c = k.c, d = k.d ^ (t & k.t_mask) ^ (last & k.last_mask);
#define CHAN_HALF_G(rot1, rot2, x) \
    a = (a + (x)) + b;             \
    d = rot1(d ^ a);               \
    c = c + d;                     \
    b = rot2(b ^ c);
// the second half of a G function with the exchange of a, d and c issued as each becomes final
#define CHAN_HALF_G_X(x, src_a, src_c)                          \
    a = (a + (x)) + b;                                          \
    {                                                           \
        const uint32_t na = __shfl_sync(full, a, src_a);        \
        d = rotr8(d ^ a);                                       \
        const uint32_t nd = __shfl_xor_sync(full, d, 2);        \
        c = c + d;                                              \
        const uint32_t nc = __shfl_sync(full, c, src_c);        \
        b = rotr7(b ^ c);                                       \
        a = na; d = nd; c = nc;                                 \
    }
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint32_t x0 = word(4 * r), x1 = word(4 * r + 1), x2 = word(4 * r + 2), x3 = word(4 * r + 3);
        CHAN_HALF_G(rotr16, rotr12, x0)
        CHAN_HALF_G_X(x1, up, dn)
        CHAN_HALF_G(rotr16, rotr12, x2)
        CHAN_HALF_G_X(x3, dn, up)
    }
#undef CHAN_HALF_G
#undef CHAN_HALF_G_X
    return make_uint2(h.x ^ a ^ c, h.y ^ b ^ d);
}

// Warp-collective transcript step. msg[0,8) is the digest. n >= 0: the caller has put n <= 24 words at msg[8, 8 + n) and zeros up
// to the block's end; digest <- H(digest || words), every word reduced mod p (channel/blake2s.rs:58-93), left at msg[0,8). Then
// `draws` secure felts (channel/blake2s.rs:34-52, 95-120): H(digest || n_draws || 0x00); the reference draws again while a word is
// >= 2p, which a reduced word never is. n < 0: draws only. msg[8,32) is zero on return. Felt j is left at felts[4 j, 4 j + 4) (and
// read back by any lane: a __syncwarp is the last thing done). One loop over the compressions with nothing but selections between
// them: the code of the hash is there once, and a taken branch costs more than the few instructions it would skip.
__device__ __forceinline__ void chan_step(ChanSm& s, int n, int draws, uint32_t* felts) {
    const int lane = threadIdx.x & 31;
    const QuadConst k;
    const uint32_t total = 4u * (uint32_t)(8 + n);
    int block = n < 0 ? 2 : n > 8 ? 0 : 1;  // 0: the first of two blocks; 1: the last block mixed; 2 ...: draws
    uint32_t drawn = n < 0 ? s.n_draws : 0u;
    const int end = 2 + draws;
    uint2 h = make_uint2(k.h0, k.h1);
    const uint32_t* m = s.msg;
    __syncwarp();
    if (lane == 8 && block == 2) s.msg[8] = drawn;
    __syncwarp();
#pragma unroll 1
    for (; block < end; block++) {
        h = b2s_compress_quad(h, ScheduledWords{m, s.sched}, k, block == 0 ? 64u : block == 1 ? total : 37u, block == 0 ? 0u : 0xffffffffu);
        const uint32_t rx = reduce_word_m31(h.x), ry = reduce_word_m31(h.y);
        const bool first = block == 0, mixed = block == 1;
        h.x = first ? h.x : k.h0;
        h.y = first ? h.y : k.h1;
        m = first ? s.msg + 16 : s.msg;
        drawn += block >= 2 ? 1u : 0u;
        uint32_t* const out = mixed ? s.msg : felts + 4 * (block - 2);
        __syncwarp();
        if (lane < 4 && !first) out[lane] = rx;
        if (lane < 4 && mixed) out[4 + lane] = ry;
        if (lane >= 8 && !first) s.msg[lane] = lane == 8 && block + 1 < end ? drawn : 0u;
        __syncwarp();
    }
    if (lane == 0) s.n_draws = drawn;
    __syncwarp();
}

// One hash of a sum-check's transcript and one draw after it (chan_step's steps), for a warp that does little else and keeps where its message words
// are. Every compression is code of its own and its words come by addresses in registers: 3,930 cycles for three compressions, 4,420 as chan_step.
// two_blocks: the message is msg[0, 32); otherwise it is msg[16, 32), the digest's copy (chan_copy_digest) and the words mixed in. bytes() is asked,
// and meanwhile() called, behind the first compression of two. draw: which of the draws after this hash is made (each hashes the digest and its number, so one that
// nobody reads need not be). Returns word (lane & 3) of the felt; msg[8, 32) is zero.
struct QuadWordsAt {
    const QuadWords& w;
    uint32_t bytes;  // a constant where it is used
    __device__ __forceinline__ uint32_t operator()(int i) const { return *reinterpret_cast<const uint32_t*>(__cvta_shared_to_generic(w.address[i] + bytes)); }
};
template <class Bytes, class Meanwhile>
__device__ __forceinline__ uint32_t chan_round(ChanSm& s, const QuadWords& w, const QuadConst& k, bool two_blocks, uint32_t draw, Bytes bytes, Meanwhile meanwhile) {
    const int lane = threadIdx.x & 31;
    uint2 h = make_uint2(k.h0, k.h1);
    if (two_blocks) h = b2s_compress_quad(h, QuadWordsAt{w, 0u}, k, 64u, 0u);
    meanwhile();
    h = b2s_compress_quad(h, QuadWordsAt{w, 64u}, k, bytes(), 0xffffffffu);
    h = make_uint2(reduce_word_m31(h.x), reduce_word_m31(h.y));
    if (lane < 4) { s.msg[lane] = h.x; s.msg[4 + lane] = h.y; }
    if (lane >= 8) s.msg[lane] = lane == 8 ? draw : 0u;
    if (lane == 0) s.n_draws = draw + 1u;
    __syncwarp();
    h = b2s_compress_quad(make_uint2(k.h0, k.h1), QuadWordsAt{w, 0u}, k, 37u, 0xffffffffu);
    if (lane == 8) s.msg[8] = 0u;
    return reduce_word_m31(h.x);
}
// For a message of one block, before its words: a __syncwarp must follow.
__device__ __forceinline__ void chan_copy_digest(ChanSm& s) {
    const int lane = threadIdx.x & 31;
    if (lane < 8) s.msg[16 + lane] = s.msg[lane];
}

// A product by y, a coordinate a lane (its two low bits): four multiply-adds and a reduction, where a lane that makes all four takes sixteen and four.
struct slice_by {
    uint32_t m[4];
    __device__ __forceinline__ slice_by(qm31 y) {
        const int k = threadIdx.x & 3;
        const uint32_t e0 = m31_sub(m31_dbl(y.c[2]), y.c[3]), e1 = m31_add(y.c[2], m31_dbl(y.c[3]));
        m[0] = k == 0 ? y.c[0] : k == 1 ? y.c[1] : k == 2 ? y.c[2] : y.c[3];
        m[1] = k == 0 ? P - y.c[1] : k == 1 ? y.c[0] : k == 2 ? P - y.c[3] : y.c[2];
        m[2] = k == 0 ? e0 : k == 1 ? e1 : k == 2 ? y.c[0] : y.c[1];
        m[3] = k == 0 ? P - e1 : k == 1 ? e0 : k == 2 ? P - y.c[1] : y.c[0];
    }
    // coordinate k of x y, and the word z added (qm31_add_products has the bound)
    __device__ __forceinline__ uint32_t mul_add(qm31 x, uint32_t z) const {
        return m31_reduce64(z + (uint64_t)x.c[0] * m[0] + (uint64_t)x.c[1] * m[1] + (uint64_t)x.c[2] * m[2] + (uint64_t)x.c[3] * m[3]);
    }
};
// The value whose coordinates are in lanes first ... first + 3.
__device__ __forceinline__ qm31 gather_q(uint32_t v, int first) {
    qm31 r;
#pragma unroll
    for (int c = 0; c < 4; c++) r.c[c] = __shfl_sync(0xffffffffu, v, first + c);
    return r;
}

// Sum mod p of one word over the warp, the same value in every lane: two integer warp reductions of 16-bit halves.
__device__ __forceinline__ uint32_t warp_sum_m31(uint32_t v) {
    const uint32_t lo = __reduce_add_sync(0xffffffffu, v & 0xffffu), hi = __reduce_add_sync(0xffffffffu, v >> 16);
    return m31_reduce64(((uint64_t)hi << 16) + lo);
}

}  // namespace zk
