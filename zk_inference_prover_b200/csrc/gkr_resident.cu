// GKR prove_batch with the Fiat-Shamir transcript resident on the device, for one or a few instances.
//
// The reference's prover (nitroo/crates/stwo/src/prover/lookups/gkr_prover.rs:657-882 with sumcheck.rs:96-176) returns to the
// host channel after every sum-check round: 276 round trips for one instance of 2^24 fractions. Which kernels run, on which
// sizes, in which order depends only on the instances' sizes, never on the transcript, so the host enqueues the whole proof
// without waiting and one copy brings it back.
//
// What bounds a proof is the chain of its rounds: each is three dependent Blake2s compressions (two to mix the round polynomial
// in, one to draw the challenge, some 0.8 us each, channel.cuh) between a pass over the layer and the next. Everything else is
// kept off that chain:
//   * Layers of at most 2^13 entries run in ONE CTA (res_chain_kernel): from the first fold on they live in its shared memory,
//     and as many whole layers as are small follow one another in the same launch, so a round costs no launch and no trip to L2.
//   * One oracle's rounds of at most 2^8 terms are worked out a round ahead (look_work): while a round's polynomial is hashed the other warps make
//     the next one as a function of the challenge to come. Between a challenge and the next hash are two products. The next layer's arrays and basis
//     are made ready under the hash of the mask, its first sums, linear in lambda, under the hash of the claims.
//   * In the other rounds what a polynomial depends on beside the two sums is prepared while the data warps work on the layer: the basis polynomials
//     of all rounds of a layer while its claims are mixed in, the claims, the corrections and the coefficients' share that does not depend on the sums
//     (one warp) while the others fold.
//   * Rounds on larger layers are one launch each (res_round_kernel): the fold by the round before's challenge, the sums of the
//     result, and, by the CTA that finishes last, the transcript step; the next launch is a programmatic dependent of it.
//   * eq(., point) is never written out for these: the terms are taken in chunks of at most 2^11 with one factor in common,
//     eq = A[low 11 bits] B[the rest], so a pass reads a table of 32 KB and multiplies by B once per chunk.
// Measured (one instance): 2^10 fractions 906 -> 317 -> 224 us, 2^24 fractions 7.95 -> 3.37 -> 3.21 ms (the last steps: rounds a round ahead, 12,000 ->
// 5,150 cycles each, of which the three compressions take 3,900; a layer's begin and end 22,000 -> 9,500). Code that runs once a layer is cold: some five
// cycles an instruction, so what is not on the transcript's path is better simple than short.
#include <algorithm>
#include <vector>

#include "channel.cuh"
#include "common.cuh"
#include "gkr_tower.cuh"
#include "gkr_resident.hpp"
#include "host/b200_backend.hpp"

namespace zk {

constexpr int RES_MAX_INST = 16;
constexpr int RES_MAX_VARS = 32;
constexpr int RES_THREADS = 512;          // the chain kernel's CTA
constexpr int RES_WARPS = RES_THREADS / 32;
// The chain kernel takes a layer over once its pass reads at most this many entries (log2): 2^13 entries folded to 2^12 of two
// columns are 128 KB of its shared memory, and the pass itself takes one SM about 5 us, what a launch of its own costs.
constexpr int CHAIN_LOG = 13;
constexpr int CHAIN_EQ_LOG = CHAIN_LOG - 2;                        // the most terms (log2) a pass of the chain kernel has
constexpr size_t CHAIN_EQ_BYTES = (size_t)16 << CHAIN_EQ_LOG;
constexpr size_t CHAIN_WORK_BYTES = (size_t)32 << (CHAIN_LOG - 1);
constexpr size_t CHAIN_SMEM = CHAIN_EQ_BYTES + CHAIN_WORK_BYTES;
constexpr int EQ_LOW = 11;                                         // low table of the launched rounds
constexpr int EQ_HIGH_MAX = 12;
constexpr int BASIS_Q = 16;                                        // (L0 - L1)[4], L1[4], L2[4], e0a, e2a, y, 1 - y
constexpr int POLY_WORDS = 20, MASK_WORDS = 16;
constexpr int STEP_LEVELS = 5;

__device__ __forceinline__ qm31 ldq_r(const void* p, size_t i) {
    uint4 v = reinterpret_cast<const uint4*>(p)[i];
    return {{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ void stq_r(void* p, size_t i, qm31 v) {
    reinterpret_cast<uint4*>(p)[i] = make_uint4(v.c[0], v.c[1], v.c[2], v.c[3]);
}
__device__ __forceinline__ qm31 shfl_q(qm31 v, int src) {
    qm31 r;
#pragma unroll
    for (int c = 0; c < 4; c++) r.c[c] = __shfl_sync(0xffffffffu, v.c[c], src);
    return r;
}
__device__ __forceinline__ qm31 warp_sum_q(qm31 v) {
    qm31 r;
#pragma unroll
    for (int c = 0; c < 4; c++) r.c[c] = warp_sum_m31(v.c[c]);
    return r;
}
// The steps of a transcript are run once a round by one warp, and what such code costs is as much the fetching of its instructions
// as the arithmetic: a taken branch to code that has left the instruction cache of the SM's quarter stalls some 70 cycles. (With
// every product inlined behind its own operand selection, or called, an update of three products in a row took 2,900-3,500 cycles
// and an empty loop over the oracles 550.) So there is one copy of the hash, one product for everything that is not on a round's
// path, and the products that are on it run from a table (step_level).
__device__ __noinline__ qm31 qmul(qm31 a, qm31 b) { return qm31_mul(a, b); }
__device__ __noinline__ void chan_step_shared(ChanSm& s, int n, int draws, qm31* felts) { chan_step(s, n, draws, reinterpret_cast<uint32_t*>(felts)); }
__device__ __forceinline__ qm31 one_minus(qm31 v) { return qm31_sub(qm31_one(), v); }

// ---- the transcript's state between launches, and its copy in shared memory while a kernel works on it
struct alignas(16) ResState {
    uint32_t digest[8];
    uint32_t n_draws, pad[3];
    qm31 alpha, lambda, challenge;       // (alpha and lambda are drawn together)
    qm31 ood[RES_MAX_VARS + 1];
    qm31 prefix[RES_MAX_VARS + 2];       // prefix[j] = prod_{i < j} (1 - ood[i])
    qm31 assign[RES_MAX_VARS + 1];       // the layer's challenges so far
    qm31 prefix_next[RES_MAX_VARS + 2];  // the same products over them: the next layer's prefix
    qm31 claims[RES_MAX_INST][2];
    qm31 out_claims[RES_MAX_INST][2];
    uint32_t n_claims[RES_MAX_INST], n_out_claims[RES_MAX_INST];
    qm31 sc[RES_MAX_INST];               // claims of the layer's oracles
    qm31 corr[RES_MAX_INST];             // eq(assignment, point) over the variables fixed so far
    qm31 apow[RES_MAX_INST];             // alpha^k
    uint32_t sums[RES_MAX_INST][8];
    uint4 steps[STEP_LEVELS][32];        // the products of a transcript step (step_level)
};
static_assert(sizeof(ResState) % 16 == 0, "ResState is copied in 16-byte pieces");

struct alignas(16) TrSm {
    ResState s;
    ChanSm ch;
    qm31 H0[RES_MAX_INST], H2[RES_MAX_INST];  // several oracles: corr e0a, corr e2a (r0 = sum0 H0, r2 = sum2 H2),
    qm31 G0[RES_MAX_INST], G2[RES_MAX_INST];  // and the same times alpha^k
    qm31 base[4];                             // the combined polynomial's share that does not depend on the sums
    qm31 coef[4];                             // the round's polynomial
    // one oracle: what a coefficient takes of the two sums (H0 (L0 - L1) and H2 L2), the round's H0 and H2, corr e0a and corr e2a of
    // the round after before its correction, the challenge and one minus it, the prefix product, intermediate values, zero
    qm31 A[8], H[2], next_h[2], r, omr, pcur, tmp[5], zero, sink[32];
    uint32_t n_vars[RES_MAX_INST];            // variables of the layer's oracles
    // rounds worked out ahead (look_rounds): the next polynomial's coefficients as cubics in the challenge, low first; the sums they are made
    // of; the challenges of this round and the last (and the two polynomials); the first round's sums (solo_begin)
    qm31 look_coef[2][4], ahead[16], look_sums[12], look_r[2], first_sums[32];
};

// Any set of threads; a barrier must follow (and precede tr_store's readers).
__device__ __forceinline__ void tr_load(TrSm& t, const ResState* st, int thread, int n_threads) {
    for (int i = thread; i < (int)(sizeof(ResState) / 16); i += n_threads) reinterpret_cast<uint4*>(&t.s)[i] = __ldcg(reinterpret_cast<const uint4*>(st) + i);
    chan_make_schedule(t.ch, thread, n_threads);
}
__device__ __forceinline__ void tr_open_channel(TrSm& t, int lane) {  // one warp, after tr_load's barrier
    t.ch.msg[lane] = lane < 8 ? t.s.digest[lane] : 0u;
    if (lane == 0) t.ch.n_draws = t.s.n_draws;
    __syncwarp();
}
__device__ __forceinline__ void tr_close_channel(TrSm& t, int lane) {
    __syncwarp();
    if (lane < 8) t.s.digest[lane] = t.ch.msg[lane];
    if (lane == 0) t.s.n_draws = t.ch.n_draws;
    __syncwarp();
}
__device__ __forceinline__ void tr_store(const TrSm& t, ResState* st, int thread, int n_threads) {
    for (int i = thread; i < (int)(sizeof(ResState) / 16); i += n_threads) reinterpret_cast<uint4*>(st)[i] = reinterpret_cast<const uint4*>(&t.s)[i];
}

// Basis of the rounds of a layer (correct_sum_as_poly_in_first_variable, gkr_prover.rs:884-923). With y = ood[n - k] the
// variable a round with k variables left fixes, an oracle's round polynomial goes through (0, r0), (1, r1), (2, r2), (b, 0) with
// b = (1 - y) / (1 - 2y), i.e. it is r0 L0 + r1 L1 + r2 L2; r0 = sum0 corr e0a, r2 = sum2 corr e2a with e0a = eq(0, y) / a and
// e2a = eq(2, y) / a, a = prod_{i <= n - k} eq(0, y_i). The inversions (of a, 1 - 2y, 1 - y, y, 1 - 3y; those of b, 1 - b and 2 - b
// follow) are one per thread.
// Rounds [first, n) of a layer, ys: their variables, prefix: the products before them.
__device__ __forceinline__ void basis_inverses(const qm31* ys, qm31* prefix, qm31* inv, int first, int n, int thread, int n_threads) {
    for (int i = 5 * first + thread; i < 5 * n; i += n_threads) {
        const int j = i / 5, w = i % 5;
        const qm31 y = ldq_r(ys, j), omy = one_minus(y), y2 = qm31_dbl(y);
        const qm31 a = qm31_mul(ldq_r(prefix, j), omy);
        if (w == 0) stq_r(prefix, j + 1, a);  // (what is there already, but for the last one)
        stq_r(inv, i, qm31_inv(w == 0 ? a : w == 1 ? one_minus(y2) : w == 2 ? omy : w == 3 ? y : qm31_sub(omy, y2)));
    }
}
// Every value is (p0 + p1 b) q, of lanes that all do the same: L1 = -t(t-2)(t-b) / (1-b), L2 = t(t-1)(t-b) / 2(2-b), L0 = -(t-1)(t-2)(t-b) / 2b, low
// coefficients first; 1/b = d / (1-y), -1/(1-b) = d / y, 1/(2-b) = d / (1-3y) with d = 1 - 2y. By whole warps.
__device__ __forceinline__ void basis_rounds(const qm31* ys, const qm31* inv, qm31* basis, int first, int n, int thread, int n_threads) {
    for (int i0 = BASIS_Q * first + (thread & ~31); i0 < BASIS_Q * n; i0 += n_threads) {
        const int i = i0 + (thread & 31), j = min(i / BASIS_Q, n - 1), w = i % BASIS_Q, c = w & 3;
        const qm31* iv = inv + 5 * j;
        const qm31 y = ldq_r(ys, j), omy = one_minus(y), y2 = qm31_dbl(y), d = one_minus(y2);
        const qm31 b = qm31_mul(omy, ldq_r(iv, 1)), q = qm31_mul(d, ldq_r(iv, w < 4 ? 2 : w < 8 ? 3 : 4)), b2 = qm31_dbl(b);
        auto small = [](uint32_t m) { return qm31_from_m31(m); };
        // the polynomials' numerators: t(t-2)(t-b), t(t-1)(t-b) and -(t-1)(t-2)(t-b)
        const qm31 p1 = c == 0 ? qm31_zero() : c == 1 ? b2 : c == 2 ? qm31_neg(qm31_add(small(2), b)) : qm31_one();
        const qm31 p2 = c == 0 ? qm31_zero() : c == 1 ? b : c == 2 ? qm31_neg(qm31_add(qm31_one(), b)) : qm31_one();
        const qm31 p0 = c == 0 ? b2 : c == 1 ? qm31_neg(qm31_add(small(2), qm31_add(b2, b))) : c == 2 ? qm31_add(small(3), b) : qm31_neg(qm31_one());
        // eq(0, y) / a and eq(2, y) / a, eq(2, y) = 3y - 1
        const qm31 x = w < 4 ? p0 : w < 8 ? p1 : w < 12 ? p2 : w == 12 ? omy : qm31_neg(qm31_sub(omy, y2));
        qm31 v = qm31_mul(x, w < 12 ? q : ldq_r(iv, 0));
        if (w < 4 || (w >= 8 && w < 12)) v = qm31_mul_m31(v, 1u << 30);
        const qm31 l1 = shfl_q(v, (thread + 4) & 31);
        if (w < 4) v = qm31_sub(v, l1);
        if (w >= 14) v = w == 14 ? y : omy;
        if (i < BASIS_Q * n) stq_r(basis, i, v);
    }
}

// The steps below are chains of a few dependent secure products on one warp. Each level of a chain is ONE product whose operands
// the lanes choose for themselves (a branch per product would run them one after the other).

// ---- one oracle. Its round polynomial is the batch's, so its next claim is that polynomial at the challenge, and everything a
// round needs beside its sums follows in three levels of products: the coefficients are sum0 A[c] + sum2 A[4 + c] + base[c].
//
// A level: every lane takes x (z + z') + a of four values in TrSm (and the basis behind it) and stores it; the byte offsets are in
// the level's table, so a level is the same thirty instructions and one product for all lanes whatever they compute, and the
// levels are one loop. z may move with the round (its offset in the basis).
__device__ __forceinline__ qm31 step_level(TrSm& t, const uint4 e, uint32_t basis_off) {
    char* const base = reinterpret_cast<char*>(&t);
    const qm31 x = ldq_r(base + e.x, 0);
    const qm31 z = qm31_add(ldq_r(base + (e.y & 0xffffu) + e.w * basis_off, 0), ldq_r(base + (e.y >> 16), 0));
    const qm31 m = qm31_mul_add(x, z, ldq_r(base + (e.z & 0xffffu), 0));
    stq_r(base + (e.z >> 16), 0, m);
    __syncwarp();
    return m;
}
// basis_at: byte offset of the basis of round 0 from TrSm.
__device__ __forceinline__ void step_tables(TrSm& t, uint32_t basis_at, int thread, int n_threads) {
    for (int i = thread; i < STEP_LEVELS * 32; i += n_threads) {
        const int level = i >> 5, l = i & 31;
        auto off = [&](const void* p) { return (uint32_t)(reinterpret_cast<const char*>(p) - reinterpret_cast<const char*>(&t)); };
        const uint32_t zero = off(&t.zero);
        uint32_t x = zero, z = zero, z2 = zero, a = zero, out = off(&t.sink[l]), moving = 0;
        auto B = [&](int ahead, int q) { moving = 1; return basis_at + 16u * (uint32_t)(BASIS_Q * ahead + q); };
        if (level == 0) {         // prepare a layer's first round: claim L1, corr e0a, corr e2a, and those of the round after
            if (l < 4) { x = off(&t.s.sc[0]); z = B(0, 4 + l); out = off(&t.base[l]); }
            else if (l < 6) { x = off(&t.s.corr[0]); z = B(0, 8 + l); out = off(&t.H[l - 4]); }
            else if (l < 8) { x = off(&t.s.corr[0]); z = B(1, 6 + l); out = off(&t.next_h[l - 6]); }
        } else if (level == 1) {
            if (l < 8) { x = off(&t.H[l >> 2]); z = B(0, l < 4 ? l : 4 + l); out = off(&t.A[l]); }
        } else if (level == 2) {  // after a challenge: (c3 r + c2), (c1 r + c0), r^2, the two parts of eq(r, y), the prefix product
            if (l < 2) { x = off(&t.coef[3 - 2 * l]); z = off(&t.r); a = off(&t.coef[2 - 2 * l]); out = off(&t.tmp[l]); }
            else if (l == 2) { x = off(&t.r); z = off(&t.r); out = off(&t.tmp[2]); }
            else if (l == 3) { x = off(&t.r); z = B(0, 14); out = off(&t.tmp[3]); }
            else if (l == 4) { x = off(&t.omr); z = B(0, 15); out = off(&t.tmp[4]); }
            else if (l == 5) { x = off(&t.pcur); z = off(&t.omr); out = off(&t.pcur); }
        } else if (level == 3) {  // the claim; the next round's H, the correction
            if (l == 0) { x = off(&t.tmp[0]); z = off(&t.tmp[2]); a = off(&t.tmp[1]); out = off(&t.s.sc[0]); }
            else if (l < 4) { x = l < 3 ? off(&t.next_h[l - 1]) : off(&t.s.corr[0]); z = off(&t.tmp[3]); z2 = off(&t.tmp[4]); out = l < 3 ? off(&t.H[l - 1]) : x; }
        } else {                  // prepare the next round, and the H of the round after it
            if (l < 8) { x = off(&t.H[l >> 2]); z = B(1, l < 4 ? l : 4 + l); out = off(&t.A[l]); }
            else if (l < 12) { x = off(&t.s.sc[0]); z = B(1, 4 + l - 8); out = off(&t.base[l - 8]); }
            else if (l < 14) { x = off(&t.s.corr[0]); z = B(2, l); out = off(&t.next_h[l - 12]); }
        }
        t.s.steps[level][l] = make_uint4(x, z | z2 << 16, a | out << 16, moving);
    }
}

// ---- several oracles, taken eight at a time: lane = 8 q + k, q saying which of up to four products of oracle k the lane has
__device__ __noinline__ void many_prepare(TrSm& t, const qm31* B, int K, uint32_t n_rem) {
    const int lane = threadIdx.x & 31, q = lane >> 3;
    qm31 ac_sum = qm31_zero(), cw_sum = qm31_zero();
    for (int kb = 0; kb < K; kb += 8) {
        const int k = kb + (lane & 7);
        const bool live = k < K, act = live && n_rem <= t.n_vars[k];
        const qm31 a = live ? t.s.apow[k] : qm31_zero(), sc = live ? t.s.sc[k] : qm31_zero(), corr = live ? t.s.corr[k] : qm31_zero();
        // a * claim (half of it when the oracle waits: it contributes the constant claim / 2), corr * e0a, corr * e2a
        const qm31 m = qmul(q == 0 ? a : corr, q == 0 ? (act ? sc : qm31_mul_m31(sc, 1u << 30)) : q == 1 ? B[12] : B[13]);
        const qm31 g = qmul(a, m);
        if (act && q == 1) { t.H0[k] = m; t.G0[k] = g; }
        if (act && q == 2) { t.H2[k] = m; t.G2[k] = g; }
        ac_sum = qm31_add(ac_sum, warp_sum_q(q == 0 && act ? m : qm31_zero()));
        cw_sum = qm31_add(cw_sum, warp_sum_q(q == 0 && live && !act ? m : qm31_zero()));
    }
    qm31 v = qmul(ac_sum, B[4 + (lane & 3)]);
    if (lane == 0) v = qm31_add(v, cw_sum);
    if (lane < 4) t.base[lane] = v;
    __syncwarp();
}
// The length of the combination when its leading coefficient vanishes: it keeps the length of its longest term (every term trimmed,
// their sum not), so the terms' own lengths decide.
__device__ __noinline__ int many_length(const TrSm& t, const qm31* B, int K, uint32_t n_rem) {
    const int lane = threadIdx.x & 31;
    int len = 0;
    if (lane < K) {
        if (n_rem <= t.n_vars[lane]) {
            const qm31 r0 = qmul(ldq_r(t.s.sums[lane], 0), t.H0[lane]), r2 = qmul(ldq_r(t.s.sums[lane], 1), t.H2[lane]);
            for (int c = 0; c < 4; c++)  // r0 L0 + (claim - r0) L1 + r2 L2
                if (!qm31_is_zero(qm31_add(qm31_add(qmul(r0, B[c]), qmul(t.s.sc[lane], B[4 + c])), qmul(r2, B[8 + c])))) len = c + 1;
        } else if (!qm31_is_zero(t.s.sc[lane])) {
            len = 1;
        }
    }
    return __reduce_max_sync(0xffffffffu, len);
}
// Coefficient (lane & 3) of the batch's polynomial: r1 = claim - r0, so the sums enter as S0 (L0 - L1) + S2 L2.
__device__ __noinline__ qm31 many_coefficients(const TrSm& t, const qm31* B, int K, uint32_t n_rem) {
    const int lane = threadIdx.x & 31, k = lane >> 1;
    const bool act = k < K && n_rem <= t.n_vars[k];
    const qm31 part = qmul(act ? ldq_r(t.s.sums[k], lane & 1) : qm31_zero(), act ? ((lane & 1) ? t.G2[k] : t.G0[k]) : qm31_zero());
    const qm31 S0 = warp_sum_q((lane & 1) ? qm31_zero() : part), S2 = warp_sum_q((lane & 1) ? part : qm31_zero());
    return qmul((lane & 4) ? S2 : S0, B[(lane & 3) + ((lane & 4) ? 8 : 0)]);
}
// Claims and corrections at the round's challenge (sumcheck.rs:150-171), and the next layer's prefix product.
__device__ __noinline__ void many_update(TrSm& t, const qm31* B, int K, uint32_t n_rem, int round) {
    const int lane = threadIdx.x & 31, q = lane >> 3;
    const qm31 r = t.s.challenge, y = B[14];
    // the basis at r, (L3 r + L2) r^2 + (L1 r + L0) (lanes 0-2 and 4-6), r^2 (8), eq(r, y) (9, 10), the prefix product (11)
    const int w = lane & 3;
    auto L = [&](int c) { return w == 0 ? qm31_add(B[c], B[4 + c]) : B[4 * w + c]; };
    qm31 x = r, z = r;
    if (lane < 8 && w < 3) x = L(lane < 4 ? 3 : 1);
    if (lane == 9) x = y;
    if (lane == 10) { x = one_minus(y); z = one_minus(r); }
    if (lane == 11) { x = t.s.prefix_next[round]; z = one_minus(r); }
    qm31 m = qmul(x, z);
    if (lane == 11) t.s.prefix_next[round + 1] = m;
    const qm31 step = qm31_add(shfl_q(m, 9), shfl_q(m, 10)), r2v = shfl_q(m, 8);
    if (lane < 8 && w < 3) m = qm31_add(m, L(lane < 4 ? 2 : 0));
    const qm31 at = qm31_add(qmul(m, r2v), shfl_q(m, (lane + 4) & 31));
    const qm31 l0 = shfl_q(at, 0), l1 = shfl_q(at, 1), l2 = shfl_q(at, 2);
    for (int kb = 0; kb < K; kb += 8) {
        const int k = kb + (lane & 7);
        const bool live = k < K, act = live && n_rem <= t.n_vars[k];
        const qm31 sc = live ? t.s.sc[k] : qm31_zero();
        // round values: r0 (q = 0), r2 (q = 2), r1 = claim - r0 (q = 1)
        const qm31 rv = qmul(act && !(q & 1) ? ldq_r(t.s.sums[k], q >> 1) : qm31_zero(), act ? (q == 0 ? t.H0[k] : t.H2[k]) : qm31_zero());
        const qm31 r0 = shfl_q(rv, lane & 7);
        const qm31 v = qmul(q == 0 ? r0 : q == 1 ? qm31_sub(sc, r0) : q == 2 ? rv : live ? t.s.corr[k] : qm31_zero(), q == 0 ? l0 : q == 1 ? l1 : q == 2 ? l2 : step);
        const qm31 sum = qm31_add(qm31_add(v, shfl_q(v, (lane + 8) & 31)), shfl_q(v, (lane + 16) & 31));
        if (act && q == 0) t.s.sc[k] = sum;
        if (act && q == 3) t.s.corr[k] = v;
        if (live && !act && q == 0) t.s.sc[k] = qm31_mul_m31(sc, 1u << 30);
    }
    __syncwarp();
}

// ---- the three parts of a round's transcript, each by one warp
// B: the round's basis, basis_off its byte offset from the first round's.
__device__ __forceinline__ void tr_prepare(TrSm& t, const qm31* B, uint32_t basis_off, int K, uint32_t n_rem) {
    if (K > 1) { many_prepare(t, B, K, n_rem); return; }
    const int lane = threadIdx.x & 31;
    uint4 e = t.s.steps[0][lane];
#pragma unroll 1
    for (int level = 0; level < 2; level++) {
        const uint4 next = t.s.steps[1][lane];
        step_level(t, e, basis_off);
        e = next;
    }
}
// The round polynomial of the batch from the oracles' sums (sumcheck.rs:139-149), mixed into the channel, and the round's
// challenge. poly: POLY_WORDS words of the proof.
__device__ __forceinline__ void tr_round(TrSm& t, const qm31* B, int K, uint32_t n_rem, int round, uint32_t* poly) {
    const int lane = threadIdx.x & 31;
    qm31 p;
    if (K == 1) p = qm31_mul(ldq_r(t.s.sums[0], (lane >> 2) & 1), t.A[lane & 7]);
    else p = many_coefficients(t, B, K, n_rem);
    const qm31 c = qm31_add(qm31_add(p, shfl_q(p, (lane + 4) & 31)), t.base[lane & 3]);
    if (lane < 4) {
        stq_r(t.ch.msg + 8, lane, c);
        stq_r(poly, lane, c);
        t.coef[lane] = c;
    }
    const unsigned nonzero = __ballot_sync(0xffffffffu, lane < 4 && !qm31_is_zero(c));
    int len = 32 - __clz(nonzero);
    if (K > 1 && len < 4) len = many_length(t, B, K, n_rem);
    if (lane == 0) poly[16] = (uint32_t)len;
    chan_step_shared(t.ch, 4 * len, 1, &t.r);
    if (lane == 0) { const qm31 r = t.r; t.s.challenge = r; t.omr = one_minus(r); t.s.assign[round] = r; }
    __syncwarp();
}
// Reads up to two bases after B (the rounds' whose H it prepares), whatever is there after the last one.
__device__ __forceinline__ void tr_update(TrSm& t, const qm31* B, uint32_t basis_off, int K, uint32_t n_rem, int round, bool prepare_next) {
    if (K > 1) {
        many_update(t, B, K, n_rem, round);
        if (prepare_next && n_rem > 1) many_prepare(t, B + BASIS_Q, K, n_rem - 1);
        return;
    }
    const int lane = threadIdx.x & 31;
    uint4 e = t.s.steps[2][lane];
#pragma unroll 1
    for (int level = 2; level < (prepare_next ? 5 : 4); level++) {
        const uint4 next = t.s.steps[level < 4 ? level + 1 : 4][lane];
        const qm31 m = step_level(t, e, basis_off);
        if (level == 2 && lane == 5) t.s.prefix_next[round + 1] = m;
        e = next;
    }
    __syncwarp();
}

// ---- one term of the round sums: t0 and t2 of sum_as_poly_in_first_variable (cpu/lookups/gkr.rs:39-211) from the denominators
// (and numerators) at (0, i, {0, 1}) and (1, i, {0, 1}); n0 d1 + n1 d0 + lambda d0 d1 taken as (n0 + lambda d0) d1 + n1 d0
template <int KIND>
__device__ __forceinline__ qm31 term_at(qm31 d0, qm31 d1, qm31 n0, qm31 n1, qm31 lambda) {
    if (KIND == ZKB_GKR_GRAND_PRODUCT) return qm31_mul(d0, d1);
    if (KIND == ZKB_GKR_LOGUP_SINGLES) return qm31_mul_add(lambda, qm31_mul(d0, d1), qm31_add(d0, d1));
    return qm31_dot2(qm31_mul_add(lambda, d0, n0), d1, n1, d0);
}
__device__ __forceinline__ qm31 at_two(qm31 v0, qm31 v1) { return qm31_sub(qm31_dbl(v1), v0); }
__device__ __forceinline__ qm31 fold_q(qm31 r, qm31 a, qm31 b) { return qm31_mul_add(r, qm31_sub(b, a), a); }
__device__ __forceinline__ qm31 fold_m(qm31 r, uint32_t a, uint32_t b) {
    qm31 v = qm31_mul_m31(r, m31_sub(b, a));
    v.c[0] = m31_add(v.c[0], a);
    return v;
}

// Term i of a layer's pass. FOLD: the layer (n entries) is first fixed at r, entries o and o + n/2 of every column giving entry o
// of the outputs; a thread reads and writes only the entries of its own terms, so the outputs may be the inputs' first half.
// nt: terms of the pass.
template <int KIND, bool FOLD, bool AHEAD>
__device__ __forceinline__ void pass_term(const void* num, const void* den, void* num_out, void* den_out, size_t nt, size_t i, qm31 r, qm31 lambda,
                                          qm31& t0, qm31& t2) {
    const size_t o[4] = {2 * i, 2 * i + 1, 2 * (nt + i), 2 * (nt + i) + 1};
    const size_t half = 4 * nt;  // entries after the fold
    constexpr bool QNUM = KIND == ZKB_GKR_LOGUP_GENERIC, BNUM = KIND == ZKB_GKR_LOGUP_MULTIPLICITIES;
    qm31 d[4], u[4];
    // AHEAD: all loads before the first store. As far as the compiler knows a store may be to what the next load reads, so that a term
    // waited for memory eight times over (2^24 entries: 3.82 -> 3.61 ms). A layer in one CTA's reach is better off entry by entry, with
    // fewer values held (2^10 entries: 317 us, 324 ahead).
    if (FOLD && !AHEAD) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            d[q] = fold_q(r, ldq_r(den, o[q]), ldq_r(den, o[q] + half));
            stq_r(den_out, o[q], d[q]);
            u[q] = qm31_zero();
            if (QNUM) u[q] = fold_q(r, ldq_r(num, o[q]), ldq_r(num, o[q] + half));
            if (BNUM) u[q] = fold_m(r, static_cast<const uint32_t*>(num)[o[q]], static_cast<const uint32_t*>(num)[o[q] + half]);
            if (QNUM || BNUM) stq_r(num_out, o[q], u[q]);
        }
        t0 = term_at<KIND>(d[0], d[1], u[0], u[1], lambda);
        t2 = term_at<KIND>(at_two(d[0], d[2]), at_two(d[1], d[3]), at_two(u[0], u[2]), at_two(u[1], u[3]), lambda);
        return;
    }
    qm31 d1[4], u1[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        d[q] = ldq_r(den, o[q]);
        if (FOLD) d1[q] = ldq_r(den, o[q] + half);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        u[q] = QNUM ? ldq_r(num, o[q]) : BNUM ? qm31_from_m31(static_cast<const uint32_t*>(num)[o[q]]) : qm31_zero();
        if (FOLD && QNUM) u1[q] = ldq_r(num, o[q] + half);
        if (FOLD && BNUM) u1[q].c[0] = static_cast<const uint32_t*>(num)[o[q] + half];
    }
    if (FOLD) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            d[q] = fold_q(r, d[q], d1[q]);
            stq_r(den_out, o[q], d[q]);
        }
        if (QNUM || BNUM) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                u[q] = QNUM ? fold_q(r, u[q], u1[q]) : fold_m(r, u[q].c[0], u1[q].c[0]);
                stq_r(num_out, o[q], u[q]);
            }
        }
    }
    t0 = term_at<KIND>(d[0], d[1], u[0], u[1], lambda);
    t2 = term_at<KIND>(at_two(d[0], d[2]), at_two(d[1], d[3]), at_two(u[0], u[2]), at_two(u[1], u[3]), lambda);
}

// ---- towers: gkr_tower.cuh's levels, the launches a chain of programmatic dependents
struct TowerArgs {
    const uint32_t *num, *den;  // 2^log entries
    uint32_t *num_out[TOWER_LEVELS], *den_out[TOWER_LEVELS];
    int levels, cta_log;        // a CTA takes 2^cta_log entries, levels <= cta_log
};
template <int KIND>
__global__ void __launch_bounds__(TOWER_THREADS) tower_kernel(TowerArgs a) {
    __shared__ uint4 sd[512], sn[KIND != ZKB_GKR_GRAND_PRODUCT ? 512 : 1];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    tower_cta<KIND>(a.num, a.den, blockIdx.x, a.cta_log, a.levels, sd, sn, [&](int l, uint32_t*& num, uint32_t*& den) { num = a.num_out[l]; den = a.den_out[l]; }, nullptr);
}

// ---- rounds on large layers, one launch each
struct RoundArgs {
    const uint32_t *num, *den;
    uint32_t *num_out, *den_out;
    const uint32_t *eq_low, *eq_high;  // eq = low[i mod 2^EQ_LOW] high[i >> EQ_LOW]
    size_t nt;                          // terms of the pass
    uint32_t chunk_log;                 // terms a CTA takes at a time: 2^chunk_log <= 2^EQ_LOW
    uint32_t* partials;
    unsigned int* ticket;
    ResState* st;
    const qm31* basis;                  // of the round whose sums these are; the next round's follows
    uint32_t* poly;
    int oracle;                         // whose sums these are
    int n_oracles, n_rem, round, transcript;  // transcript: this launch completes the round's sums and runs its step
    uint32_t n_vars[RES_MAX_INST];
};
constexpr int ROUND_THREADS = 256;
constexpr int ROUND_MAX_CTAS = 148 * 4;
template <int KIND, bool FOLD>
__global__ void __launch_bounds__(ROUND_THREADS, 2) res_round_kernel(const __grid_constant__ RoundArgs a) {
    __shared__ struct alignas(16) { TrSm tr; qm31 basis[3 * BASIS_Q]; } sm;
    TrSm& tr = sm.tr;
    __shared__ uint32_t red[ROUND_THREADS / 32][8];
    __shared__ bool is_last;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const qm31 lambda = ldq_r(&a.st->lambda, 0);
    const qm31 r = FOLD ? ldq_r(&a.st->challenge, 0) : qm31_zero();
    qm31 s0 = qm31_zero(), s2 = qm31_zero();
    const size_t n_chunks = a.nt >> a.chunk_log;
    for (size_t ck = blockIdx.x; ck < n_chunks; ck += gridDim.x) {
        const size_t begin = ck << a.chunk_log;
        qm31_sum c0 = qm31_sum_zero(), c2 = qm31_sum_zero();
        for (size_t i = begin + tid; i < begin + ((size_t)1 << a.chunk_log); i += ROUND_THREADS) {
            qm31 t0, t2;
            const qm31 e = ldq_r(a.eq_low, i & ((1u << EQ_LOW) - 1));
            pass_term<KIND, FOLD, true>(a.num, a.den, a.num_out, a.den_out, a.nt, i, r, lambda, t0, t2);
            c0.add_product(e, t0);
            c2.add_product(e, t2);
        }
        const qm31 eh = ldq_r(a.eq_high, begin >> EQ_LOW);
        s0 = qm31_add(s0, qm31_mul(eh, c0.value()));
        s2 = qm31_add(s2, qm31_mul(eh, c2.value()));
    }
    s0 = warp_sum_q(s0);
    s2 = warp_sum_q(s2);
    if (lane == 0) { stq_r(red[warp], 0, s0); stq_r(red[warp], 1, s2); }
    __syncthreads();
    if (tid < 8) {
        uint32_t acc = 0;
#pragma unroll
        for (int w = 0; w < ROUND_THREADS / 32; w++) acc = m31_add(acc, red[w][tid]);
        a.partials[8 * blockIdx.x + tid] = acc;
        __threadfence();
    }
    __syncthreads();
    if (tid == 0) is_last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!is_last) return;
    // every other CTA has ended or is about to: the next launch may be scheduled and run up to its wait
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __threadfence();
    if (tid == 0) *a.ticket = 0u;
    // the partial sums: word tid & 7 of every 32nd CTA per thread, then over the threads (eight threads that walk the CTAs one
    // after the other take 20 us for 592 of them)
    {
        uint32_t acc = 0;
        for (unsigned b = tid >> 3; b < gridDim.x; b += ROUND_THREADS / 8) acc = m31_add(acc, __ldcg(&a.partials[8 * b + (tid & 7)]));
        acc = m31_add(acc, __shfl_xor_sync(0xffffffffu, acc, 8));
        acc = m31_add(acc, __shfl_xor_sync(0xffffffffu, acc, 16));
        __syncthreads();
        if (lane < 8) red[warp][lane] = acc;
    }
    if (a.transcript) {
        tr_load(tr, a.st, tid, ROUND_THREADS);
        if (tid == 32) tr.zero = qm31_zero();
        if (tid < RES_MAX_INST) tr.n_vars[tid] = a.n_vars[tid];
        if (tid >= 64 && tid < 64 + 2 * BASIS_Q) sm.basis[tid - 64] = ldq_r(a.basis, tid - 64);  // this round's and the next one's
    }
    __syncthreads();
    uint32_t mine = 0;
    if (tid < 8) {
#pragma unroll
        for (int w = 0; w < ROUND_THREADS / 32; w++) mine = m31_add(mine, red[w][tid]);
        if (a.transcript) tr.s.sums[a.oracle][tid] = mine;
        else a.st->sums[a.oracle][tid] = mine;
    }
    if (!a.transcript) return;
    __syncthreads();
    if (warp == 0) {
        tr_open_channel(tr, lane);
        if (lane == 0) tr.pcur = tr.s.prefix_next[a.round];
        tr_prepare(tr, sm.basis, 0u, a.n_oracles, (uint32_t)a.n_rem);
        tr_round(tr, sm.basis, a.n_oracles, (uint32_t)a.n_rem, a.round, a.poly);
        tr_close_channel(tr, lane);
        tr_update(tr, sm.basis, 0u, a.n_oracles, (uint32_t)a.n_rem, a.round, false);
    }
    __syncthreads();
    tr_store(tr, a.st, tid, ROUND_THREADS);
}

// ---- whole layers in one CTA
enum : uint32_t { CHAIN_BEGIN = 1, CHAIN_ROUNDS = 2, CHAIN_END = 4 };
struct alignas(16) ChainLayer {
    uint32_t flags;
    int nv, round_start;               // rounds of the layer; the first the chain kernel runs
    int n_inst, n_oracles, last_active;
    int table_bits;                    // CHAIN_BEGIN without CHAIN_ROUNDS: bits of the high table (the low one has EQ_LOW)
    uint32_t *eq_low, *eq_high;        // where the two tables go
    qm31* basis;                       // the layer's basis in device memory (written with the tables, read when the rounds resume)
    uint32_t* polys;                   // POLY_WORDS per round of this layer
    uint32_t* masks;                   // MASK_WORDS per oracle
    // instances: the kind of the output layer of those that start here, -1 otherwise; its entry; whether the instance is active
    int start_kind[RES_MAX_INST], active[RES_MAX_INST];
    const uint32_t *out_num[RES_MAX_INST], *out_den[RES_MAX_INST];
    // oracles: instance, variables, the arrays the first pass of the launch reads and their kind, where folded layers go (a byte
    // offset into the CTA's work area, or, with work_global, an address)
    int inst[RES_MAX_INST], kind[RES_MAX_INST];
    uint32_t n_vars[RES_MAX_INST];
    const uint32_t *num[RES_MAX_INST], *den[RES_MAX_INST];
    uint64_t num_work[RES_MAX_INST], den_work[RES_MAX_INST];
    uint64_t work_global;
};
static_assert(sizeof(ChainLayer) % 16 == 0, "ChainLayer is copied in 16-byte pieces");

// While the first warp hashes at the start of a layer, the warps after it form the basis of its rounds and the rest eq(., point).
constexpr int BASIS_THREADS = 160, EQ_THREADS = RES_THREADS - 32 - BASIS_THREADS;
__device__ __forceinline__ void basis_bar() { asm volatile("bar.sync 1, %0;" ::"n"(BASIS_THREADS) : "memory"); }
__device__ __forceinline__ void eq_bar() { asm volatile("bar.sync 2, %0;" ::"n"(EQ_THREADS) : "memory"); }

// table[x] = v prod_{k < bits} (bit k of x ? y_k : 1 - y_k), y_k = ood[ny - first_bit - k] (gen_eq_evals: index bit k pairs with the
// k-th variable from the end). By the EQ_THREADS last threads.
__device__ __forceinline__ void eq_build(void* table, const qm31* ood, int ny, int first_bit, int bits, qm31 v) {
    const int th = threadIdx.x - (RES_THREADS - EQ_THREADS);
    if (th == 0) stq_r(table, 0, v);
    eq_bar();
    for (int k = 0; k < bits; k++) {
        const uint32_t len = 1u << k;
        const qm31 y = ood[ny - first_bit - k];
        for (uint32_t j = th; j < len; j += EQ_THREADS) {
            const qm31 e = ldq_r(table, j), hi = qmul(e, y);
            stq_r(table, j, qm31_sub(e, hi));
            stq_r(table, j + len, hi);
        }
        eq_bar();
    }
}

// The claims of the instances that start here, every active instance's claims into the channel, alpha and lambda, the oracles'
// claims (gkr_prover.rs:669-735). Warp-collective.
__device__ __forceinline__ void tr_begin(TrSm& t, const ChainLayer& L) {
    const int lane = threadIdx.x & 31;
    if (lane < L.n_inst && L.start_kind[lane] >= 0) {
        const int kind = L.start_kind[lane];
        const qm31 den0 = ldq_r(L.out_den[lane], 0);
        int n = 2;
        qm31 first = qm31_one();
        if (kind == ZKB_GKR_GRAND_PRODUCT) { first = den0; n = 1; }
        else if (kind == ZKB_GKR_LOGUP_GENERIC) first = ldq_r(L.out_num[lane], 0);
        else if (kind == ZKB_GKR_LOGUP_MULTIPLICITIES) first = qm31_from_m31(L.out_num[lane][0]);
        t.s.claims[lane][0] = first;
        t.s.claims[lane][1] = den0;
        t.s.n_claims[lane] = n;
        t.s.out_claims[lane][0] = first;
        t.s.out_claims[lane][1] = den0;
        t.s.n_out_claims[lane] = n;
    }
    __syncwarp();
    for (int i = 0; i < L.n_inst; i++)
        if (L.active[i]) {
            const int n = 4 * (int)t.s.n_claims[i];
            if (lane < n) t.ch.msg[8 + lane] = reinterpret_cast<const uint32_t*>(t.s.claims[i])[lane];
            chan_step_shared(t.ch, n, i == L.last_active ? 2 : 0, &t.s.alpha);
        }
    const qm31 alpha = t.s.alpha, lambda = t.s.lambda;
    if (lane == 0) { t.s.prefix_next[0] = qm31_one(); t.pcur = qm31_one(); }
    const int K = L.n_oracles, k = lane & 15;
    qm31 pw = qm31_one();
    if (K > 1) {  // alpha^k by the bits of k
        qm31 sq = alpha;
        for (int b = 0; (1 << b) < K; b++) {
            const qm31 m = qmul(pw, sq);
            if ((k >> b) & 1) pw = m;
            sq = qmul(sq, sq);
        }
    }
    const int i = k < K ? L.inst[k] : 0;
    const bool two = t.s.n_claims[i] == 2;
    const qm31 h = qmul(lambda, t.s.claims[i][1]);
    if (lane < K) {
        t.s.apow[k] = pw;
        t.s.corr[k] = qm31_one();
        t.s.sc[k] = qm31_mul_m31(two ? qm31_add(h, t.s.claims[i][0]) : t.s.claims[i][0], 1u << (L.nv - (int)L.n_vars[k]));
    }
    __syncwarp();
}

// The masks into the channel, the next layer's point and claims (gkr_prover.rs:745-800). Warp-collective. Oracle k's two entries
// per column are at num(k) / den(k), of kind kind(k): what the folds have made of the layer.
template <class Kind, class Num, class Den>
__device__ __forceinline__ void tr_end(TrSm& t, const ChainLayer& L, Kind kind, Num num, Den den) {
    const int lane = threadIdx.x & 31, K = L.n_oracles, nv = L.nv;
    for (int k = 0; k < K; k++) {
        uint32_t* out = L.masks + (size_t)MASK_WORDS * k;
        const bool one_col = kind(k) == ZKB_GKR_GRAND_PRODUCT;
        if (lane < 16) {
            uint32_t v = 0u;
            const uint32_t* d = static_cast<const uint32_t*>(den(k));
            if (one_col) v = lane < 8 ? d[lane] : 0u;
            else if (lane >= 8) v = d[lane - 8];
            else if (kind(k) == ZKB_GKR_LOGUP_GENERIC) v = static_cast<const uint32_t*>(num(k))[lane];
            else v = (lane & 3) == 0 ? 1u : 0u;
            t.ch.msg[8 + lane] = v;
            out[lane] = v;
        }
        chan_step_shared(t.ch, one_col ? 8 : 16, k == K - 1 ? 1 : 0, &t.s.challenge);
    }
    const qm31 c = t.s.challenge;
    if (lane <= nv) {
        if (lane < nv) t.s.ood[lane] = t.s.assign[lane];
        t.s.prefix[lane] = t.s.prefix_next[lane];
    }
    const qm31 last = qmul(t.s.prefix_next[nv], one_minus(c));
    if (lane == 0) { t.s.ood[nv] = c; t.s.prefix[nv + 1] = last; }
    // claims: two columns of up to sixteen oracles
    const int k = lane & 15, col = lane >> 4;
    const bool live = k < K && !(col == 1 && kind(k) == ZKB_GKR_GRAND_PRODUCT);
    qm31 a = qm31_zero(), b = qm31_zero();
    if (live) {
        const bool one_col = kind(k) == ZKB_GKR_GRAND_PRODUCT;
        if (col == 1 || one_col) { a = ldq_r(den(k), 0); b = ldq_r(den(k), 1); }
        else if (kind(k) == ZKB_GKR_LOGUP_GENERIC) { a = ldq_r(num(k), 0); b = ldq_r(num(k), 1); }
        else a = b = qm31_one();
    }
    const qm31 v = qm31_add(qmul(c, qm31_sub(b, a)), a);
    if (live) {
        t.s.claims[L.inst[k]][col] = v;
        t.s.n_claims[L.inst[k]] = kind(k) == ZKB_GKR_GRAND_PRODUCT ? 1u : 2u;
    }
    __syncwarp();
}

// Sum over a pass's terms by every thread of the CTA, each thread's share in s0 / s2.
template <int KIND, bool FOLD>
__device__ __forceinline__ void chain_pass(const void* num, const void* den, void* num_out, void* den_out, uint32_t nt, qm31 r, qm31 lambda, const void* eq,
                                           qm31& s0, qm31& s2) {
    for (uint32_t i = (threadIdx.x - 64u) & (RES_THREADS - 1); i < nt; i += RES_THREADS) {
        qm31 t0, t2;
        pass_term<KIND, FOLD, false>(num, den, num_out, den_out, nt, i, r, lambda, t0, t2);
        const qm31 e = ldq_r(eq, i);
        s0 = qm31_add(s0, qm31_mul(e, t0));
        s2 = qm31_add(s2, qm31_mul(e, t2));
    }
}

// A pass of few terms is the latency of one thread's 16 multiplications: it is taken in two steps instead, one multiplication per
// thread for the fold (an entry each), then a unit of work per warp: 32 terms at one node (t = 0 or t = 2), and of a term one of
// the two products it is the sum of, (n0 + lambda d0) d1 or n1 d0, times eq.
constexpr uint32_t CHAIN_SMALL = 256;
__device__ __forceinline__ qm31 small_unit(int kind, const void* num, const void* den, uint32_t nt, uint32_t i, int node, int part, qm31 lambda, const void* eq) {
    qm31 s = qm31_zero();
    if (i < nt) {
        auto at = [&](const void* p, uint32_t b) {
            const qm31 v0 = ldq_r(p, 2 * i + b);
            return node ? at_two(v0, ldq_r(p, 2 * (nt + i) + b)) : v0;
        };
        qm31 n = kind == ZKB_GKR_GRAND_PRODUCT ? qm31_zero() : qm31_one();  // numerator `part`; LogUpSingles has ones
        if (kind == ZKB_GKR_LOGUP_GENERIC) {
            n = at(num, part);
        } else if (kind == ZKB_GKR_LOGUP_MULTIPLICITIES) {
            const uint32_t* m = static_cast<const uint32_t*>(num);
            const uint32_t v0 = m[2 * i + part];
            n = qm31_from_m31(node ? m31_sub(m31_dbl(m[2 * (nt + i) + part]), v0) : v0);
        }
        const qm31 d0 = at(den, 0);
        if (part == 0) s = qm31_mul(qm31_add(n, kind == ZKB_GKR_GRAND_PRODUCT ? d0 : qm31_mul(lambda, d0)), at(den, 1));
        else s = qm31_mul(n, d0);
        s = qm31_mul(ldq_r(eq, i), s);
    }
    return warp_sum_q(s);
}
// The same for one oracle, whose numerators have been changed for m = n + (lambda / 2) d: products m0 d1 and m1 d0 (a grand product: d0 d1).
__device__ __forceinline__ qm31 small_unit_m(bool product, const void* m, const void* den, uint32_t nt, uint32_t i, int node, int part, const void* eq) {
    qm31 s = qm31_zero();
    if (i < nt && !(product && part)) {
        auto at = [&](const void* p, uint32_t b) {
            const qm31 v0 = ldq_r(p, 2 * i + b);
            return node ? at_two(v0, ldq_r(p, 2 * (nt + i) + b)) : v0;
        };
        s = qm31_mul(ldq_r(eq, i), qm31_mul(at(product ? den : m, part), at(den, 1 - part)));
    }
    if (nt >= 16) return warp_sum_q(s);
    for (uint32_t off = nt >> 1; off; off >>= 1) s = qm31_add(s, shfl_q(s, (threadIdx.x & 31) + off));  // lane 0 has the sum
    return s;
}

// ---- the small rounds of one oracle, a round ahead of the transcript
//
// A layer fixed at r is linear in r and a term is a product of two of its entries, so the next round's sums are quadratic in this round's
// challenge: S(r) = C0 + C1 r + C2 r^2, and with the correction, linear in r, and the claim, this round's cubic at r, the coefficients of the
// next polynomial are cubics in r. Their coefficients are worked out while the first warp hashes this round's polynomial; when it
// has the challenge it has the next polynomial two products later and hashes on. The layer itself is fixed under the next hash. What was on a
// round's path and no longer is: the fold, the sums and three levels of products, with the barriers between them.
//
// A round:
//   warp 0          next polynomial from `ahead`, its hash, the challenge
//   LOOK_WARPS      the layer fixed at the last challenge; then six sums, two warps each (the second for passes of more than 32 terms): two
//                   nodes (t = 0, 2) x the term at r = 0, at r = 1 and its leading coefficient
//   the last one    correction at the last challenge besides; `ahead` from the sums and the polynomial being hashed
// Warp 0 has its scheduler to itself: what other warps issue there is taken from its turns (three compressions 3,930 -> 4,600 cycles).
constexpr int LOOK_WARPS = 12;
constexpr uint32_t LOOK_TERMS = 256;  // passes of more terms take longer this way than the hash they would hide under
static_assert(RES_WARPS == 16, "twelve warps are not on warp 0's scheduler");
// The barriers: a polynomial is there (warp 0 to the helper), the layer is fixed (the twelve), the sums are there (the twelve to the helper), so is the last
// round's basis (solo_last_basis to the helper). Warp 0 and the twelve meet when a challenge is there: what is due by then (`ahead`, the mask) is.
__device__ __forceinline__ void look_poly_set() { asm volatile("bar.arrive 3, 64;" ::: "memory"); }
__device__ __forceinline__ void look_poly_wait() { asm volatile("bar.sync 3, 64;" ::: "memory"); }
__device__ __forceinline__ void look_fixed() { asm volatile("bar.sync 4, %0;" ::"n"(32 * LOOK_WARPS) : "memory"); }
__device__ __forceinline__ void look_sums_set() { asm volatile("bar.arrive 5, %0;" ::"n"(32 * LOOK_WARPS) : "memory"); }
__device__ __forceinline__ void look_sums_wait() { asm volatile("bar.sync 5, %0;" ::"n"(32 * LOOK_WARPS) : "memory"); }
__device__ __forceinline__ void look_basis_set() { asm volatile("bar.arrive 7, 64;" ::: "memory"); }
__device__ __forceinline__ void look_basis_wait() { asm volatile("bar.sync 7, 64;" ::: "memory"); }
__device__ __forceinline__ void look_challenge() { asm volatile("bar.sync 6, %0;" ::"n"(32 * (LOOK_WARPS + 1)) : "memory"); }

// A layer that is taken whole this way.
__device__ __forceinline__ bool is_solo(const ChainLayer& L) {
    return L.flags == (CHAIN_BEGIN | CHAIN_ROUNDS | CHAIN_END) && L.n_oracles == 1 && L.nv > 0 && (1u << (L.nv - 1)) <= LOOK_TERMS;
}
// The work areas of two such layers, of at most 4 LOOK_TERMS entries a column: while one ends the next is fetched.
constexpr uint32_t SOLO_BYTES = 64 * LOOK_TERMS;
constexpr int SOLO_BASIS_WARPS = 5;
static_assert(4 * SOLO_BYTES <= CHAIN_WORK_BYTES, "two layers of two columns");
__device__ __forceinline__ void solo_done() { asm volatile("bar.sync 9, %0;" ::"n"(RES_THREADS) : "memory"); }

// Where one_lead starts and ends.
enum : int { LEAD_BEGIN = 1, LEAD_ROUNDS = 2, LEAD_SUMS = 4 };

// Warp 0, for a layer with one oracle. LEAD_BEGIN: its claims into the channel, lambda (gkr_prover.rs:669-735). LEAD_ROUNDS: rounds round0 ... nv - 1, from the sums of round0's units in red (LEAD_SUMS) or, with the begin, from `ahead` at lambda; the
// mask into the channel, the next layer's last coordinate and claims (gkr_prover.rs:745-800). The mask's hash is the loop's last turn, so that the
// code of the hash is there once. With both it goes on to the layers after this one while they are taken whole; returns the layer it stopped at.
__device__ __noinline__ int one_lead(TrSm& t, const ChainLayer* bufs, int d, int n_layers, int what, int round0, const qm31* red, uint32_t units, const unsigned char* num,
                                     const unsigned char* den) {
    const int lane = threadIdx.x & 31;
    const QuadWords words(t.ch.msg, t.ch.sched);
    const QuadConst qc;
    for (;;) {
        const ChainLayer& L = bufs[d & 1];
        const int nv = L.nv, inst = L.inst[0];
        const bool product = L.kind[0] == ZKB_GKR_GRAND_PRODUCT;
        const uint32_t area = what & LEAD_SUMS ? 0u : (d & 1) * SOLO_BYTES;
        qm31 r = qm31_zero(), mask = r;
        uint32_t c = 0u;  // lane = 4 k + coordinate (and 16 more): coefficient k of the round's polynomial
        if (what & LEAD_SUMS) {
            const qm31 v = (uint32_t)lane < units ? red[lane] : qm31_zero();
            const qm31 s0 = warp_sum_q((lane & 1) ? qm31_zero() : v), s2 = warp_sum_q((lane & 1) ? v : qm31_zero());
            const qm31 p = qmul((lane & 4) ? s2 : s0, t.A[lane & 7]);
            const qm31 q = qm31_add(qm31_add(p, shfl_q(p, (lane + 4) & 31)), t.base[lane & 3]);  // coefficient `lane` in lanes 0-3
            const qm31 mine = shfl_q(q, (lane >> 2) & 3);
            c = (lane & 3) == 0 ? mine.c[0] : (lane & 3) == 1 ? mine.c[1] : (lane & 3) == 2 ? mine.c[2] : mine.c[3];
        }
        for (int round = what & LEAD_BEGIN ? -1 : round0;; round++) {
            unsigned nonzero = 0xffffu;  // the words mixed in
            if (round >= 0 && round < nv) {
                if (!(round == round0 && (what & LEAD_SUMS))) {
                    // (d3 r + d2) r^2 + (d1 r + d0): the low half in lanes 0-15, the high one in 16-31
                    const int at = (lane & 12) + (lane >> 4) * 2;
                    const qm31 d1 = ldq_r(t.ahead, at + 1);
                    const uint32_t d0 = t.ahead[at].c[lane & 3];
                    const slice_by by(r);
                    const uint32_t m = by.mul_add(d1, d0), r2 = by.mul_add(r, 0u);
                    c = slice_by(gather_q(r2, 0)).mul_add(gather_q(m, 16 + (lane & 12)), m);
                }
                if (lane < 16) t.ch.msg[8 + lane] = c;
                nonzero = __ballot_sync(0xffffffffu, lane < 16 && c != 0u);
                if (!(nonzero & 0xff00u)) {  // two coefficients or fewer
                    __syncwarp();
                    chan_copy_digest(t.ch);
                    if (lane < 8) t.ch.msg[24 + lane] = c;
                }
            } else if (round < 0) {
                const int n = 4 * (int)t.s.n_claims[inst];
                nonzero = (1u << n) - 1u;
                chan_copy_digest(t.ch);
                if (lane < n) t.ch.msg[24 + lane] = reinterpret_cast<const uint32_t*>(t.s.claims[inst])[lane];
            } else {
                // two entries a column (num0, num1, den0, den1; a grand product has the denominators only)
                const void* const col = (product || (lane & 2) ? den : num) + area;
                mask = fold_q(r, ldq_r(col, lane & 1), ldq_r(col, (lane & 1) + 2));
                if (product) {
                    nonzero = 0xffu;
                    chan_copy_digest(t.ch);
                }
                if (lane < (product ? 2 : 4)) stq_r(t.ch.msg + (product ? 24 : 8), lane, mask);
            }
            __syncwarp();
            const uint32_t v = chan_round(
                t.ch, words, qc, (nonzero & 0xff00u) != 0u, round < 0 ? 1u : 0u,  // (alpha, the first draw of a begin, is the power of nothing here)
                [&] { return 32u + 16u * (uint32_t)((35 - __clz(nonzero)) >> 2); },    // whole coefficients, up to the last that is not zero
                [&] {
                    if (round >= 0 && round < nv) {
                        if (lane < 16) t.look_coef[round & 1][lane >> 2].c[lane & 3] = c;
                        __syncwarp();
                        if (nv - round >= 2) look_poly_set();
                    } else if (round == nv && lane < 4) {
                        stq_r(L.masks, lane, lane < (product ? 2 : 4) ? mask : qm31_zero());
                    }
                });
            if (round < nv && lane < 4) t.look_r[round & 1].c[lane] = v;
            r = gather_q(v, 0);
            __syncwarp();
            if (round == nv) break;
            if (round < 0) {
                if (lane == 0) {
                    t.s.lambda = r;
                    t.s.prefix_next[0] = t.pcur = t.s.apow[0] = t.s.corr[0] = qm31_one();
                }
                __syncwarp();
                if (!(what & LEAD_ROUNDS)) {  // the claim, for rounds that are not worked out ahead
                    const qm31 sc = qm31_add(qmul(product ? qm31_zero() : t.s.claims[inst][1], r), t.s.claims[inst][0]);
                    if (lane == 0) t.s.sc[0] = sc;
                    __syncwarp();
                    return d;
                }
            }
            look_challenge();
        }
        const qm31 claim = fold_q(r, shfl_q(mask, 2 * (lane & 1)), shfl_q(mask, 2 * (lane & 1) + 1));
        if (lane < (product ? 1 : 2)) stq_r(t.s.claims[inst], lane, claim);
        if (lane == 0) {
            t.s.n_claims[inst] = product ? 1u : 2u;
            t.s.challenge = t.s.ood[nv] = r;
        }
        __syncwarp();
        if (what & LEAD_SUMS) return d;
        solo_done();
        if (++d == n_layers || !is_solo(bufs[d & 1])) return d;
    }
}

// A layer's entries into the work area, numerators as they are.
__device__ __forceinline__ void solo_fetch(const ChainLayer& L, unsigned char* num, unsigned char* den, uint32_t thread, uint32_t n_threads) {
    const int kind = L.kind[0];
    for (uint32_t e = thread; e < (2u << L.nv); e += n_threads) {
        stq_r(den, e, ldq_r(L.den[0], e));
        if (kind != ZKB_GKR_GRAND_PRODUCT)
            stq_r(num, e, kind == ZKB_GKR_LOGUP_GENERIC ? ldq_r(L.num[0], e) : qm31_from_m31(kind == ZKB_GKR_LOGUP_MULTIPLICITIES ? L.num[0][e] : 1u));
    }
}

// The twelve: rounds round0 ... nv - 1. num, den: the layer, 2^(nv - round0 + 1) entries, numerators as small_unit_m has them; `begins`: numerators
// as they are, lambda is the first challenge. next (or null), then: the layer after this one, whose description goes to next_buf. If it is taken whole, its
// arrays (to next_num, next_den) and all of its basis but for the last round are made ready while the mask is hashed.
__device__ __forceinline__ void look_work(TrSm& t, qm31* basis, qm31* inv, int nv, int round0, bool begins, bool product, unsigned char* num, unsigned char* den, const void* eq,
                                          uint32_t* polys, const ChainLayer* next, ChainLayer* next_buf, unsigned char* next_num, unsigned char* next_den) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t w = (uint32_t)((warp >> 2) * 3 + (warp & 3) - 1), sum = w % 6, node = sum & 1, at_r = sum >> 1, half = w / 6;
    const bool helper = w == LOOK_WARPS - 1, keeper = w == LOOK_WARPS - 2;  // (the keeper: the point and its prefix products, the polynomials into the proof)
    // the helper: lane = 16 node + 4 c + k has that node's share of the coefficient of r^k in coefficient c of the next polynomial
    const int hn = lane >> 4, c = (lane >> 2) & 3, k = lane & 3;
    qm31 corr = begins ? qm31_one() : t.s.corr[0], a0 = qm31_zero(), a1 = a0, l1 = a0, half_lambda = begins ? a0 : qm31_mul_m31(t.s.lambda, 1u << 30);
    for (int round = round0; round <= nv; round++) {
        const uint32_t n_rem = (uint32_t)(nv - round), n_out = 2u << n_rem;
        if (helper && n_rem >= 2) {  // what does not depend on the challenge; the next correction is corr (w0 + w1 r)
            if (n_rem == 2 && begins) look_basis_wait();
            const qm31 *B = basis + BASIS_Q * round, *N = B + BASIS_Q;
            const qm31 w0 = ldq_r(B, 15), g = qm31_mul(ldq_r(N, 12 + hn), ldq_r(N, 8 * hn + c));
            a0 = qm31_mul(g, w0);
            a1 = qm31_mul(g, qm31_sub(ldq_r(B, 14), w0));
            l1 = ldq_r(N, 4 + c);
        }
        if (round > round0) {
            look_challenge();
            const qm31 r = ldq_r(t.look_r, (round & 1) ^ 1);
            if (n_rem) {
                for (uint32_t i = 32 * w + lane; i < (product ? n_out : 2 * n_out); i += 32 * LOOK_WARPS) {
                    unsigned char* const p = i < n_out ? den : num;
                    const uint32_t e = i & (n_out - 1);
                    stq_r(p, e, fold_q(r, ldq_r(p, e), ldq_r(p, e + n_out)));
                }
                look_fixed();
            }
            if (helper && n_rem >= 2) {  // eq(r, y) in two parts
                const qm31* L = basis + BASIS_Q * (round - 1);
                const qm31 m = qm31_mul((lane & 1) ? one_minus(r) : r, ldq_r(L, 14 + (lane & 1)));
                corr = qm31_mul(corr, qm31_add(m, shfl_q(m, lane ^ 1)));
            }
            if (keeper) {
                const qm31 p = qmul(ldq_r(t.s.prefix_next, round - 1), one_minus(r));
                __syncwarp();
                if (lane == 0) { stq_r(t.s.prefix_next, round, p); stq_r(t.s.assign, round - 1, r); }
                const qm31 v = ldq_r(t.look_coef[(round & 1) ^ 1], lane & 3);
                const int len = 32 - __clz(__ballot_sync(0xffffffffu, lane < 4 && !qm31_is_zero(v)));
                uint32_t* const poly = polys + (size_t)POLY_WORDS * (round - 1);
                if (lane < 4) stq_r(poly, lane, v);
                if (lane == 0) poly[16] = (uint32_t)len;
                __syncwarp();
            }
            if (n_rem == 0) {
                look_fixed();  // behind the keeper
                if (keeper && lane <= nv) {
                    if (lane < nv) t.s.ood[lane] = t.s.assign[lane];
                    t.s.prefix[lane] = t.s.prefix_next[lane];
                }
                if (!next || !is_solo(*next_buf)) break;
                if (w < SOLO_BASIS_WARPS) {
                    basis_inverses(t.s.assign, t.s.prefix_next, inv, 0, nv, 32 * w + lane, 32 * SOLO_BASIS_WARPS);
                    asm volatile("bar.sync 1, %0;" ::"n"(32 * SOLO_BASIS_WARPS) : "memory");
                    basis_rounds(t.s.assign, inv, basis, 0, nv, 32 * w + lane, 32 * SOLO_BASIS_WARPS);
                } else {
                    solo_fetch(*next_buf, next_num, next_den, 32 * (w - SOLO_BASIS_WARPS) + lane, 32 * (LOOK_WARPS - SOLO_BASIS_WARPS));
                }
                break;
            }
        } else if (begins) {
            look_challenge();
            half_lambda = qm31_mul_m31(ldq_r(t.look_r, 1), 1u << 30);
            if (n_rem >= 2 && !product) {
                for (uint32_t e = 32 * w + lane; e < n_out; e += 32 * LOOK_WARPS) stq_r(num, e, qm31_mul_add(half_lambda, ldq_r(den, e), ldq_r(num, e)));
                look_fixed();
            }
        }
        if (keeper && begins && next && round == round0)  // the next layer's description: read after the next challenge
            for (int i = lane; i < (int)(sizeof(ChainLayer) / 16); i += 32) reinterpret_cast<uint4*>(next_buf)[i] = __ldg(reinterpret_cast<const uint4*>(next) + i);
        if (n_rem < 2) {  // what is left is folded to the mask by warp 0: numerators as they are again
            if (!helper) continue;
            if (lane < 4 && !product && !(begins && nv == 1)) stq_r(num, lane, qm31_sub(ldq_r(num, lane), qm31_mul(half_lambda, ldq_r(den, lane))));
            continue;
        }
        const uint32_t nt = n_out >> 3;
        qm31 s = qm31_zero();
        for (uint32_t i = 32 * half + lane; i < nt; i += 64) {
            auto fixed = [&](const void* p, uint32_t b, uint32_t h) {  // the half that stays at r = h
                const uint32_t o = h * 4 * nt + 2 * i + b;
                const qm31 v0 = ldq_r(p, o);
                return node ? at_two(v0, ldq_r(p, o + 2 * nt)) : v0;
            };
            auto at = [&](const void* p, uint32_t b) {
                const qm31 v = fixed(p, b, at_r ? 1u : 0u);
                return at_r == 2 ? qm31_sub(v, fixed(p, b, 0u)) : v;
            };
            const qm31 d0 = at(den, 0), d1 = at(den, 1);
            s = qm31_add(s, qm31_mul(ldq_r(eq, i), product ? qm31_mul(d0, d1) : qm31_dot2(at(num, 0), d1, at(num, 1), d0)));
        }
        if (nt >= 16) s = warp_sum_q(s);
        else for (uint32_t off = nt >> 1; off; off >>= 1) s = qm31_add(s, shfl_q(s, lane + off));
        if (lane == 0) stq_r(t.look_sums, w, s);
        __syncwarp();
        if (!helper) {
            look_sums_set();
            continue;
        }
        const qm31 b0 = qm31_mul(corr, a0), b1 = qm31_mul(corr, a1);
        look_poly_wait();
        const qm31 q = hn ? qm31_zero() : qm31_mul(ldq_r(t.look_coef[round & 1], k), l1);  // this round's polynomial at r is the next claim
        look_sums_wait();
        auto sums = [&](int at) { return qm31_add(ldq_r(t.look_sums, hn + 2 * at), ldq_r(t.look_sums, hn + 2 * at + 6)); };
        const qm31 s0 = sums(0), s2 = sums(2), mid = qm31_sub(sums(1), qm31_add(s0, s2));
        const qm31 lo = k == 0 ? s0 : k == 1 ? mid : k == 2 ? s2 : qm31_zero(), hi = k == 0 ? qm31_zero() : k == 1 ? s0 : k == 2 ? mid : s2;
        const qm31 v = qm31_add(qm31_dot2(b0, lo, b1, hi), q), o = qm31_add(v, shfl_q(v, lane ^ 16));
        if (lane < 16) stq_r(t.ahead, lane, o);
    }
}

// The basis of a layer's last round, whose variable is the challenge that the layer before ended with: by a warp of its own, under the begin.
__device__ __forceinline__ void solo_last_basis(TrSm& t, qm31* basis, qm31* inv, int nv) {
    const int lane = threadIdx.x & 31;
    basis_inverses(t.s.ood, t.s.prefix, inv, nv - 1, nv, lane, 32);
    __syncwarp();
    basis_rounds(t.s.ood, inv, basis, nv - 1, nv, lane, 32);
    __syncwarp();
    look_basis_set();
}

// The begin of a small layer by the twelve, while warp 0 hashes the claims and draws lambda: the layer into the work area (unless it is there, and its basis
// with it), eq(., point), and the first round's sums, linear in lambda: `ahead` has the first polynomial at lambda. lo, hi: 32 entries each.
static_assert(2 * (LOOK_TERMS / 32) * 2 <= 32, "first_sums");
__device__ __forceinline__ void solo_begin(TrSm& t, const ChainLayer& L, qm31* basis, qm31* inv, unsigned char* num, unsigned char* den, void* eq, qm31* lo, qm31* hi,
                                           bool ready) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, w = (warp >> 2) * 3 + (warp & 3) - 1, nv = L.nv, ny = nv - 1;
    const bool product = L.kind[0] == ZKB_GKR_GRAND_PRODUCT;
    const uint32_t nt = 1u << ny, blocks = (nt + 31) >> 5;
    if (w >= LOOK_WARPS - 2) {
        // eq = lo[low five bits] hi[the rest]; the first variable's share is 1 - y
        const bool high = w == LOOK_WARPS - 1;
        const int lo_bits = ny < 5 ? ny : 5, bits = high ? ny - lo_bits : lo_bits, first = high ? lo_bits : 0;
        auto f = [&](int b) {
            const qm31 y = ldq_r(t.s.ood, b < bits ? ny - first - b : 0);
            return b >= bits ? qm31_one() : (lane >> b) & 1 ? y : one_minus(y);
        };
        const qm31 v = qm31_mul(qm31_mul(f(0), f(1)), qm31_mul(f(2), f(3)));
        stq_r(high ? hi : lo, lane, qm31_mul(v, high ? one_minus(ldq_r(t.s.ood, 0)) : f(4)));
    } else if (!ready) {
        if (w < SOLO_BASIS_WARPS) {
            basis_inverses(t.s.ood, t.s.prefix, inv, 0, nv - 1, 32 * w + lane, 32 * SOLO_BASIS_WARPS);
            asm volatile("bar.sync 1, %0;" ::"n"(32 * SOLO_BASIS_WARPS) : "memory");
            basis_rounds(t.s.ood, inv, basis, 0, nv - 1, 32 * w + lane, 32 * SOLO_BASIS_WARPS);
        } else {
            solo_fetch(L, num, den, 32 * (w - SOLO_BASIS_WARPS) + lane, 32 * (LOOK_WARPS - 2 - SOLO_BASIS_WARPS));
        }
    }
    look_fixed();
    // 32 terms at one node a turn, its share without lambda (n0 d1 + n1 d0) or with it (d0 d1)
    for (uint32_t job = w; job < 4 * blocks; job += LOOK_WARPS) {
        const bool with = job & 1, node = job & 2;
        const uint32_t i = 32 * (job >> 2) + lane;
        qm31_sum x = qm31_sum_zero();
        if (i < nt && !(with && product)) {
            const qm31 e = qm31_mul(ldq_r(lo, i & 31), ldq_r(hi, i >> 5));
            if (!with && !node) stq_r(eq, i, e);
            auto at = [&](const void* p, uint32_t b) {
                const qm31 v0 = ldq_r(p, 2 * i + b);
                return node ? at_two(v0, ldq_r(p, 2 * (nt + i) + b)) : v0;
            };
            const qm31 d0 = at(den, 0), d1 = at(den, 1), e0 = qm31_mul(e, d0);
            x.add_product(e0, with || product ? d1 : at(num, 1));
            if (!with && !product) x.add_product(qm31_mul(e, d1), at(num, 0));
        }
        const qm31 s = warp_sum_q(x.value());
        if (lane == 0) stq_r(t.first_sums, job, s);
    }
    __syncwarp();
    if (w < LOOK_WARPS - 1) {
        look_sums_set();
        return;
    }
    // look_work's helper; lanes as there
    if (nv == 1) look_basis_wait();
    const int hn = lane >> 4, c = (lane >> 2) & 3, k = lane & 3;
    const qm31 a = qm31_mul(ldq_r(basis, 12 + hn), ldq_r(basis, 8 * hn + c)), l1 = ldq_r(basis, 4 + c);
    const qm31 claim = k < (product ? 1 : 2) && !hn ? ldq_r(t.s.claims[L.inst[0]], k) : qm31_zero();
    look_sums_wait();
    qm31 s = qm31_zero();
    for (uint32_t p = 0; p < blocks; p++) s = qm31_add(s, ldq_r(t.first_sums, 4 * p + 2 * hn + (k & 1)));
    const qm31 v = qm31_dot2(k < 2 ? s : qm31_zero(), a, claim, l1), o = qm31_add(v, shfl_q(v, lane ^ 16));
    if (lane < 16) stq_r(t.ahead, lane, o);
}

struct ResInit { uint32_t digest[8], n_draws; int use; };  // use: the proof's first launch starts from this channel, not from *st
__global__ void __launch_bounds__(RES_THREADS, 1) res_chain_kernel(ResState* st, const ChainLayer* __restrict__ layers, int n_layers, ResInit init) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ struct alignas(16) { TrSm tr; qm31 basis[(RES_MAX_VARS + 2) * BASIS_Q]; } sm;
    TrSm& tr = sm.tr;
    qm31* const basis = sm.basis;
    __shared__ ChainLayer layer_buf[2];  // the layer at hand and the next one
    __shared__ alignas(16) qm31 inv[RES_MAX_VARS * 5];
    __shared__ alignas(16) qm31 red[RES_MAX_INST][32];  // per oracle: a warp's two sums (warps x 2), or the units of a small pass
    void* const eq = dyn;
    unsigned char* const work = dyn + CHAIN_EQ_BYTES;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (init.use) {
        for (int i = tid; i < (int)(sizeof(ResState) / 4); i += RES_THREADS) {
            uint32_t v = i == 8 ? init.n_draws : 0u;
#pragma unroll
            for (int k = 0; k < 8; k++) v = i == k ? init.digest[k] : v;
            reinterpret_cast<uint32_t*>(&tr.s)[i] = v;
        }
        chan_make_schedule(tr.ch, tid, RES_THREADS);
        __syncthreads();
        // the round kernels keep their bases behind TrSm too: the table travels with the state
        step_tables(tr, (uint32_t)((const char*)basis - (const char*)&tr), tid, RES_THREADS);
    } else {
        tr_load(tr, st, tid, RES_THREADS);
    }
    if (tid == 32) tr.zero = qm31_zero();
    __syncthreads();
    if (warp == 0) tr_open_channel(tr, lane);
    for (int d = 0; d < n_layers; d++) {
        ChainLayer& L = layer_buf[d & 1];
        if (d == 0)
            for (int i = tid; i < (int)(sizeof(ChainLayer) / 16); i += RES_THREADS) reinterpret_cast<uint4*>(&L)[i] = __ldg(reinterpret_cast<const uint4*>(layers) + i);
        __syncthreads();
        const int K = L.n_oracles, nv = L.nv, ny = nv - 1;
        if (tid == 0 && L.round_start) tr.pcur = tr.s.prefix_next[L.round_start];
        if (tid < K) tr.n_vars[tid] = L.n_vars[tid];
        const bool one = K == 1 && nv > 0;  // the first layer, of no variables, has the instances that start
        if (is_solo(L)) {
            unsigned char *const den = work, *const num = work + 2 * SOLO_BYTES;
            if (warp == 0) {
                d = one_lead(tr, layer_buf, d, n_layers, LEAD_BEGIN | LEAD_ROUNDS, 0, nullptr, 0, num, den);
            } else {
                bool ready = false;
                do {
                    const ChainLayer& S = layer_buf[d & 1];
                    const uint32_t here = (d & 1) * SOLO_BYTES, there = SOLO_BYTES - here;
                    if (warp & 3) {
                        solo_begin(tr, S, basis, inv, num + here, den + here, eq, red[0], red[1], ready);
                        look_work(tr, basis, inv, S.nv, 0, true, S.kind[0] == ZKB_GKR_GRAND_PRODUCT, num + here, den + here, eq, S.polys, d + 1 < n_layers ? layers + d + 1 : nullptr,
                                  &layer_buf[(d + 1) & 1], num + there, den + there);
                    } else if (warp == 4) {
                        solo_last_basis(tr, basis, inv, S.nv);
                    }
                    solo_done();
                    ready = true;
                } while (++d < n_layers && is_solo(layer_buf[d & 1]));
            }
            d--;
            continue;
        }
        if (warp == 0) {
            if (L.flags & CHAIN_BEGIN) {
                if (one) one_lead(tr, layer_buf, d, n_layers, LEAD_BEGIN, 0, nullptr, 0, nullptr, nullptr);
                else tr_begin(tr, L);
            }
        } else if (tid < 32 + BASIS_THREADS) {
            const int th = tid - 32;
            if (L.flags & CHAIN_BEGIN) {
                basis_inverses(tr.s.ood, tr.s.prefix, inv, 0, nv, th, BASIS_THREADS);
                basis_bar();
                basis_rounds(tr.s.ood, inv, basis, 0, nv, th, BASIS_THREADS);
                basis_bar();
                if (!(L.flags & CHAIN_ROUNDS))  // the rounds on launches of their own come next and read it from memory
                    for (int i = th; i < BASIS_Q * nv; i += BASIS_THREADS) L.basis[i] = basis[i];
            } else if (L.flags & CHAIN_ROUNDS) {
                for (int i = th; i < BASIS_Q * nv; i += BASIS_THREADS) basis[i] = L.basis[i];
            }
        } else if ((L.flags & CHAIN_ROUNDS) && nv > 0) {
            // the passes have at most 2^bits terms: index bits above are zero, a factor 1 - y each
            const int bits = nv - L.round_start - 1;
            if (bits >= 0) eq_build(eq, tr.s.ood, ny, 0, bits, tr.s.prefix[ny - bits + 1]);
        } else if ((L.flags & CHAIN_BEGIN) && !(L.flags & CHAIN_ROUNDS)) {
            const int th = tid - (RES_THREADS - EQ_THREADS);
            eq_build(eq, tr.s.ood, ny, 0, EQ_LOW, qm31_one());
            for (uint32_t i = th; i < (1u << EQ_LOW); i += EQ_THREADS) stq_r(L.eq_low, i, ldq_r(eq, i));
            eq_build(work, tr.s.ood, ny, EQ_LOW, L.table_bits, tr.s.prefix[1]);
            for (uint32_t i = th; i < (1u << L.table_bits); i += EQ_THREADS) stq_r(L.eq_high, i, ldq_r(work, i));
        }
        __syncthreads();
        if (warp == RES_WARPS - 1 && d + 1 < n_layers)  // under the rounds
            for (int i = lane; i < (int)(sizeof(ChainLayer) / 16); i += 32) reinterpret_cast<uint4*>(&layer_buf[(d + 1) & 1])[i] = __ldg(reinterpret_cast<const uint4*>(layers + d + 1) + i);
        // oracle k's arrays: the caller's until the first fold of this launch, then the work area's
        auto den_work = [&](int k) { return L.work_global ? reinterpret_cast<void*>(L.den_work[k]) : static_cast<void*>(work + L.den_work[k]); };
        auto num_work = [&](int k) { return L.work_global ? reinterpret_cast<void*>(L.num_work[k]) : static_cast<void*>(work + L.num_work[k]); };
        if (L.flags & CHAIN_ROUNDS) {
            // one oracle: where its layer is
            struct { const void *num, *den; int kind; } at = {L.num[0], L.den[0], L.kind[0]};
            const bool one_product = L.kind[0] == ZKB_GKR_GRAND_PRODUCT;
            for (int round = L.round_start; round <= nv; round++) {
                // Pass of this round: the oracles that were active before are fixed at the last challenge; those and the ones that
                // enter now give their sums (none after the last round). The second warp brings claims and corrections up to date
                // and prepares this round meanwhile.
                const uint32_t n_rem = (uint32_t)(nv - round);
                const qm31 r = tr.s.challenge, lambda = tr.s.lambda;
                const bool sums = round < nv;
                const uint32_t nt = sums ? 1u << (n_rem - 1) : 0u;
                const bool small = nt <= (K == 1 ? LOOK_TERMS : CHAIN_SMALL);
                if (warp == 1) {
                    if (round > L.round_start) tr_update(tr, basis + BASIS_Q * (round - 1), 16u * BASIS_Q * (round - 1), K, n_rem + 1, round - 1, true);
                    else if (sums) tr_prepare(tr, basis + BASIS_Q * round, 16u * BASIS_Q * round, K, n_rem);
                }
                if (K == 1 && small && sums) {
                    // The layer goes to the work area, fixed at the last challenge if it has had one, with n changed for m = n + (lambda / 2) d: a
                    // term is then m0 d1 + m1 d0.
                    const bool fold = round > 0;
                    const qm31 half_lambda = qm31_mul_m31(lambda, 1u << 30);
                    unsigned char* const num_to = work + L.num_work[0];
                    if (warp >= 2) {
                        const uint32_t n_out = 2u << n_rem;
                        for (uint32_t e = tid - 64u; e < n_out; e += RES_THREADS - 64u) {
                            qm31 d = ldq_r(at.den, e), n = qm31_one();
                            if (fold) d = fold_q(r, d, ldq_r(at.den, e + n_out));
                            if (at.kind == ZKB_GKR_LOGUP_MULTIPLICITIES) {
                                const uint32_t* m = static_cast<const uint32_t*>(at.num);
                                n = fold ? fold_m(r, m[e], m[e + n_out]) : qm31_from_m31(m[e]);
                            } else if (at.kind == ZKB_GKR_LOGUP_GENERIC) {
                                n = ldq_r(at.num, e);
                                if (fold) n = fold_q(r, n, ldq_r(at.num, e + n_out));
                            }
                            stq_r(work, e, d);
                            if (!one_product) stq_r(num_to, e, qm31_add(n, qm31_mul(half_lambda, d)));
                        }
                    }
                    __syncthreads();
                    // by the warps after the first two, whose instruction caches hold the transcript
                    const uint32_t units = 4 * ((nt + 31) / 32);
                    for (uint32_t w = (warp + RES_WARPS - 2) & (RES_WARPS - 1); w < units; w += RES_WARPS) {
                        const qm31 v = small_unit_m(one_product, num_to, work, nt, 32 * (w >> 2) + lane, w & 1, (w >> 1) & 1, eq);
                        if (lane == 0) red[0][w] = v;
                    }
                    __syncthreads();
                    if (warp == 0) one_lead(tr, layer_buf, d, n_layers, LEAD_ROUNDS | LEAD_SUMS, round, red[0], units, num_to, work);
                    else if (warp & 3) look_work(tr, basis, inv, nv, round, false, one_product, num_to, work, eq, L.polys, nullptr, nullptr, nullptr, nullptr);
                    break;
                }
                for (int k = small && warp < 2 ? K : 0; k < K; k++) {
                    const uint32_t vars = tr.n_vars[k];
                    const bool fold = vars > n_rem, fresh = round == L.round_start || vars == n_rem + 1;  // fresh: nothing folded here yet
                    if (!fold && (vars < n_rem || small)) continue;
                    const int kind = fresh || L.kind[k] != ZKB_GKR_LOGUP_MULTIPLICITIES ? L.kind[k] : (int)ZKB_GKR_LOGUP_GENERIC;
                    const void* den = fresh || !fold ? static_cast<const void*>(L.den[k]) : den_work(k);
                    const void* num = fresh || !fold ? static_cast<const void*>(L.num[k]) : num_work(k);
                    void *den_w = den_work(k), *num_w = num_work(k);
                    if (small) {
                        const uint32_t e_out = 2u << n_rem;  // entries of the fixed layer
                        const bool has_num = kind == ZKB_GKR_LOGUP_GENERIC || kind == ZKB_GKR_LOGUP_MULTIPLICITIES;
                        for (uint32_t i = tid - 64u; i < (has_num ? 2 : 1) * e_out; i += RES_THREADS - 64u) {  // not by the first two warps
                            const uint32_t e = i & (e_out - 1);
                            if (i >= e_out && kind == ZKB_GKR_LOGUP_MULTIPLICITIES) {
                                const uint32_t* m = static_cast<const uint32_t*>(num);
                                stq_r(num_w, e, fold_m(r, m[e], m[e + e_out]));
                            } else {
                                const void* p = i < e_out ? den : num;
                                stq_r(i < e_out ? den_w : num_w, e, fold_q(r, ldq_r(p, e), ldq_r(p, e + e_out)));
                            }
                        }
                        continue;
                    }
                    qm31 s0 = qm31_zero(), s2 = qm31_zero();
                    switch (kind + (fold ? 4 : 0)) {
                        case 0: chain_pass<0, false>(num, den, num_w, den_w, nt, r, lambda, eq, s0, s2); break;
                        case 1: chain_pass<1, false>(num, den, num_w, den_w, nt, r, lambda, eq, s0, s2); break;
                        case 2: chain_pass<2, false>(num, den, num_w, den_w, nt, r, lambda, eq, s0, s2); break;
                        case 3: chain_pass<3, false>(num, den, num_w, den_w, nt, r, lambda, eq, s0, s2); break;
                        case 4: chain_pass<0, true>(num, den, num_w, den_w, nt, r, lambda, eq, s0, s2); break;
                        case 5: chain_pass<1, true>(num, den, num_w, den_w, nt, r, lambda, eq, s0, s2); break;
                        case 6: chain_pass<2, true>(num, den, num_w, den_w, nt, r, lambda, eq, s0, s2); break;
                        default: chain_pass<3, true>(num, den, num_w, den_w, nt, r, lambda, eq, s0, s2); break;
                    }
                    s0 = warp_sum_q(s0);
                    s2 = warp_sum_q(s2);
                    if (lane == 0) { red[k][2 * warp] = s0; red[k][2 * warp + 1] = s2; }
                    if (K == 1 && fold) {
                        at.den = den_w;
                        at.num = num_w;
                        if (kind == ZKB_GKR_LOGUP_MULTIPLICITIES) at.kind = ZKB_GKR_LOGUP_GENERIC;
                    }
                }
                __syncthreads();
                if (!sums) break;
                uint32_t units = 2 * RES_WARPS;
                if (small) {
                    // by the warps after the first two, whose instruction caches hold the transcript
                    units = 4 * ((nt + 31) / 32);
                    for (uint32_t u = (warp + RES_WARPS - 2) & (RES_WARPS - 1); u < units * K; u += RES_WARPS) {
                        const int k = u / units, w = u % units;
                        if (tr.n_vars[k] < n_rem) continue;
                        const bool folded = tr.n_vars[k] > n_rem;
                        const void* den = folded ? den_work(k) : static_cast<const void*>(L.den[k]);
                        const void* num = folded ? num_work(k) : static_cast<const void*>(L.num[k]);
                        const int kind = folded && L.kind[k] == ZKB_GKR_LOGUP_MULTIPLICITIES ? (int)ZKB_GKR_LOGUP_GENERIC : L.kind[k];
                        const qm31 v = small_unit(kind, num, den, nt, 32 * (w >> 2) + lane, w & 1, (w >> 1) & 1, lambda, eq);
                        if (lane == 0) red[k][w] = v;
                    }
                    __syncthreads();
                }
                if (warp == 0) {
                    for (int k = 0; k < K; k++) {
                        if (tr.n_vars[k] < n_rem) continue;
                        const qm31 v = (uint32_t)lane < units ? red[k][lane] : qm31_zero();
                        const qm31 s0 = warp_sum_q((lane & 1) ? qm31_zero() : v), s2 = warp_sum_q((lane & 1) ? v : qm31_zero());
                        if (lane == 0) { stq_r(tr.s.sums[k], 0, s0); stq_r(tr.s.sums[k], 1, s2); }
                    }
                    __syncwarp();
                }
                if (warp == 0) tr_round(tr, basis + BASIS_Q * round, K, n_rem, round, L.polys + (size_t)POLY_WORDS * round);
                __syncthreads();
            }
        }
        if ((L.flags & CHAIN_END) && warp == 0 && !one) {
            tr_end(tr, L, [&](int k) { return L.n_vars[k] && L.kind[k] == ZKB_GKR_LOGUP_MULTIPLICITIES ? (int)ZKB_GKR_LOGUP_GENERIC : L.kind[k]; },
                   [&](int k) { return L.n_vars[k] ? num_work(k) : static_cast<const void*>(L.num[k]); },
                   [&](int k) { return L.n_vars[k] ? den_work(k) : static_cast<const void*>(L.den[k]); });
        }
    }
    __syncthreads();
    if (warp == 0) tr_close_channel(tr, lane);
    __syncthreads();
    tr_store(tr, st, tid, RES_THREADS);
}

}  // namespace zk

using namespace zk;
using b200::BaseColumn;
using b200::Device;
using b200::Layer;

namespace b200 {

bool gkr_resident_supported(int n_inst, const uint64_t* ns) {
    if (n_inst < 1 || n_inst > RES_MAX_INST) return false;
    for (int i = 0; i < n_inst; i++)
        if (ns[i] < 2 || ns[i] > ((uint64_t)1 << (EQ_LOW + EQ_HIGH_MAX + 2))) return false;
    return true;
}

namespace {

// One instance's layers: level 0 is the caller's input, level j has 2^(log - j) entries.
struct Tower {
    int kind, log;
    const uint32_t *num, *den;
    std::vector<uint32_t*> num_l, den_l;  // levels 1 ... log at [level]
    int kind_at(int level) const { return level == 0 || kind == ZKB_GKR_GRAND_PRODUCT ? kind : (int)ZKB_GKR_LOGUP_GENERIC; }
    const uint32_t* num_at(int level) const { return level == 0 ? num : num_l[level]; }
    const uint32_t* den_at(int level) const { return level == 0 ? den : den_l[level]; }
};

// Launches of one proof: all but the first are programmatic dependents of the one before (every kernel here waits for its
// predecessor before it reads anything), except under the per-kernel timeline, whose events sit between the launches.
struct Launcher {
    zkb_ctx* ctx;
    bool chained = false;
    cudaError_t err = cudaSuccess;
    template <class... P, class... A>
    void run(const char* name, void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem, A... args) {
        if (err != cudaSuccess) return;
        ProfScope prof(ctx, name);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = ctx->stream;
        cfg.attrs = attr;
        cfg.numAttrs = chained && !ctx->prof_on ? 1 : 0;
        err = cudaLaunchKernelEx(&cfg, kernel, P(args)...);
        chained = true;
    }
};

}  // namespace

int gkr_prove_resident(zkb_ctx* ctx, std::vector<Layer> input_layers, uint32_t digest[8], uint32_t* n_draws,
                       std::vector<uint32_t>& o) {
    Device d(ctx);
    DeviceGuard guard(ctx);
    const int n_inst = (int)input_layers.size();
    std::vector<Tower> towers(n_inst);
    int n_layers = 0;
    for (int i = 0; i < n_inst; i++) {
        const Layer& l = input_layers[i];
        towers[i].kind = l.kind;
        towers[i].log = (int)l.n_variables();
        towers[i].num = l.kind == ZKB_GKR_LOGUP_MULTIPLICITIES ? l.num_base.ptr() : l.num_ptr();
        towers[i].den = l.den.words.ptr();
        n_layers = std::max(n_layers, towers[i].log);
    }
    // ---- one allocation: the proof (state, round polynomials, masks: what the copy at the end brings back), the towers, the
    // folded copies of the input layers, the basis and eq tables of the layers whose rounds are launches
    const size_t n_polys = (size_t)n_layers * (n_layers - 1) / 2;
    size_t words = 0;
    auto reserve = [&](size_t n) { size_t at = words; words += (n + 63) & ~(size_t)63; return at; };
    const size_t at_state = reserve(sizeof(ResState) / 4), at_polys = reserve(n_polys * POLY_WORDS);
    std::vector<size_t> at_masks(n_layers);
    std::vector<std::vector<int>> oracle_inst(n_layers);
    for (int layer = 0; layer < n_layers; layer++) {
        for (int i = 0; i < n_inst; i++)
            if (towers[i].log >= n_layers - layer) oracle_inst[layer].push_back(i);
        at_masks[layer] = reserve(MASK_WORDS * oracle_inst[layer].size());
    }
    const size_t copy_words = words;
    std::vector<std::vector<std::pair<size_t, size_t>>> at_tower(n_inst);
    std::vector<std::pair<size_t, size_t>> at_fold(n_inst);
    for (int i = 0; i < n_inst; i++) {
        at_tower[i].resize(towers[i].log + 1);
        const bool nums = towers[i].kind != ZKB_GKR_GRAND_PRODUCT;
        for (int lv = 1; lv <= towers[i].log; lv++) {
            at_tower[i][lv].second = reserve((size_t)4 << (towers[i].log - lv));
            at_tower[i][lv].first = nums ? reserve((size_t)4 << (towers[i].log - lv)) : 0;
        }
        const bool fold_nums = towers[i].kind == ZKB_GKR_LOGUP_GENERIC || towers[i].kind == ZKB_GKR_LOGUP_MULTIPLICITIES;
        at_fold[i].second = reserve((size_t)2 << towers[i].log);
        at_fold[i].first = fold_nums ? reserve((size_t)2 << towers[i].log) : 0;
    }
    const size_t at_basis = reserve(4 * BASIS_Q * RES_MAX_VARS), at_low = reserve((size_t)4 << EQ_LOW), at_high = reserve((size_t)4 << EQ_HIGH_MAX);
    BaseColumn buf(d, words);
    uint32_t* const base = buf.ptr();
    ResState* const st = reinterpret_cast<ResState*>(base + at_state);
    for (int i = 0; i < n_inst; i++) {
        towers[i].num_l.assign(towers[i].log + 1, nullptr);
        towers[i].den_l.assign(towers[i].log + 1, nullptr);
        for (int lv = 1; lv <= towers[i].log; lv++) {
            towers[i].den_l[lv] = base + at_tower[i][lv].second;
            if (towers[i].kind != ZKB_GKR_GRAND_PRODUCT) towers[i].num_l[lv] = base + at_tower[i][lv].first;
        }
    }
    // ---- the plan: chain layers, and the launched rounds that go between two of them
    struct Step { int chain_first, chain_count; std::vector<std::pair<int, RoundArgs>> rounds; };  // (kind + 4 if it folds, arguments)
    std::vector<ChainLayer> chain;
    std::vector<Step> steps(1, Step{0, 0, {}});
    int poly_base = 0;
    for (int layer = 0; layer < n_layers; layer++) {
        const int nv = layer, K = (int)oracle_inst[layer].size();
        ChainLayer L;
        memset(&L, 0, sizeof(L));
        L.nv = nv;
        L.n_inst = n_inst;
        L.n_oracles = K;
        L.polys = base + at_polys + (size_t)POLY_WORDS * poly_base;
        L.masks = base + at_masks[layer];
        L.basis = reinterpret_cast<qm31*>(base + at_basis);
        L.eq_low = base + at_low;
        L.eq_high = base + at_high;
        for (int i = 0; i < n_inst; i++) {
            const Tower& t = towers[i];
            L.start_kind[i] = -1;
            L.active[i] = t.log >= n_layers - layer;
            if (L.active[i]) L.last_active = i;
            if (t.log == n_layers - layer) { L.start_kind[i] = t.kind_at(t.log); L.out_num[i] = t.num_at(t.log); L.out_den[i] = t.den_at(t.log); }
        }
        std::vector<int> level(K);
        size_t smem = 0;
        for (int k = 0; k < K; k++) {
            const int i = oracle_inst[layer][k];
            const Tower& t = towers[i];
            const int log_entries = 1 + layer - (n_layers - t.log);
            level[k] = t.log - log_entries;
            L.inst[k] = i;
            L.n_vars[k] = (uint32_t)(log_entries - 1);
            L.kind[k] = t.kind_at(level[k]);
            L.num[k] = t.num_at(level[k]);
            L.den[k] = t.den_at(level[k]);
            if (L.kind[k] == ZKB_GKR_LOGUP_MULTIPLICITIES && L.n_vars[k] == 0)
                return set_error(ctx, ZKB_EINVAL, "gkr: a multiplicities layer cannot be a mask");
            const size_t bytes = (size_t)16 << std::min<uint32_t>(L.n_vars[k], CHAIN_LOG - 1);
            L.den_work[k] = smem; smem += bytes;
            if (L.kind[k] != ZKB_GKR_GRAND_PRODUCT) { L.num_work[k] = smem; smem += bytes; }
        }
        if (K == 1 && L.kind[0] != ZKB_GKR_GRAND_PRODUCT) L.num_work[0] = CHAIN_WORK_BYTES / 2;  // (a small layer goes there whole)
        L.work_global = smem > CHAIN_WORK_BYTES ? 1 : 0;
        if (L.work_global)  // several tall oracles at once: in place for the towers' layers, the folded copies for the inputs
            for (int k = 0; k < K; k++) {
                const Tower& t = towers[L.inst[k]];
                L.den_work[k] = (uint64_t)(level[k] ? t.den_l[level[k]] : base + at_fold[L.inst[k]].second);
                L.num_work[k] = (uint64_t)(level[k] ? t.num_l[level[k]] : base + at_fold[L.inst[k]].first);
            }
        // Rounds whose pass reads more than 2^CHAIN_LOG entries are launches of their own (the first pass of a layer reads
        // 2^(nv + 1), a fold with k variables left after it 2^(k + 2)).
        const int round_start = nv + 1 > CHAIN_LOG ? nv - (CHAIN_LOG - 2) : 0;
        if (round_start > 0) {
            ChainLayer B = L;
            B.flags = CHAIN_BEGIN;
            B.table_bits = nv - 1 - EQ_LOW;
            chain.push_back(B);
            steps.back().chain_count++;
            std::vector<int> kind(L.kind, L.kind + K);
            for (int round = 0; round < round_start; round++) {
                const uint32_t n_rem = (uint32_t)(nv - round);
                size_t last = 0;
                for (int k = 0; k < K; k++) {
                    if (L.n_vars[k] < n_rem) continue;
                    RoundArgs a;
                    memset(&a, 0, sizeof(a));
                    const bool fold = L.n_vars[k] > n_rem;
                    const Tower& t = towers[L.inst[k]];
                    a.num = L.num[k];
                    a.den = L.den[k];
                    const int in_kind = kind[k];
                    if (fold) {
                        a.den_out = level[k] ? t.den_l[level[k]] : base + at_fold[L.inst[k]].second;
                        a.num_out = level[k] ? t.num_l[level[k]] : base + at_fold[L.inst[k]].first;
                        L.den[k] = a.den_out;
                        if (in_kind == ZKB_GKR_LOGUP_GENERIC || in_kind == ZKB_GKR_LOGUP_MULTIPLICITIES) { L.num[k] = a.num_out; kind[k] = ZKB_GKR_LOGUP_GENERIC; }
                    }
                    a.eq_low = L.eq_low;
                    a.eq_high = L.eq_high;
                    a.nt = (size_t)1 << (n_rem - 1);
                    // chunks: as long as possible (a factor of the high table is taken once per chunk) while there are enough for every SM
                    a.chunk_log = EQ_LOW;
                    while (a.chunk_log > 8 && (a.nt >> a.chunk_log) < 148 * 2) a.chunk_log--;
                    a.partials = ctx->scratch;
                    a.ticket = ctx->ticket;
                    a.st = st;
                    a.basis = L.basis + BASIS_Q * round;
                    a.poly = L.polys + (size_t)POLY_WORDS * round;
                    a.oracle = k;
                    a.n_oracles = K;
                    a.n_rem = (int)n_rem;
                    a.round = round;
                    for (int q = 0; q < K; q++) a.n_vars[q] = L.n_vars[q];
                    steps.back().rounds.push_back({in_kind + (fold ? 4 : 0), a});
                    last = steps.back().rounds.size() - 1;
                }
                steps.back().rounds[last].second.transcript = 1;
            }
            for (int k = 0; k < K; k++) L.kind[k] = kind[k];
            L.flags = CHAIN_ROUNDS | CHAIN_END;
            L.round_start = round_start;
            steps.push_back(Step{(int)chain.size(), 0, {}});
        } else {
            L.flags = CHAIN_BEGIN | CHAIN_ROUNDS | CHAIN_END;
        }
        chain.push_back(L);
        steps.back().chain_count++;
        poly_base += nv;
    }
    // ---- enqueue
    void* d_chain = nullptr;
    if (int rc = stage_blob(ctx, chain.data(), chain.size() * sizeof(ChainLayer), &d_chain)) return rc;
    if (!ctx->res_ready) {
        ZKB_CUDA(ctx, cudaFuncSetAttribute(res_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CHAIN_SMEM));
        ctx->res_ready = true;
    }
    Launcher launch{ctx};
    for (int i = 0; i < n_inst; i++) {
        const Tower& t = towers[i];
        for (int level = 0; level < t.log;) {
            TowerArgs a;
            memset(&a, 0, sizeof(a));
            a.num = t.num_at(level);
            a.den = t.den_at(level);
            a.cta_log = std::min(TOWER_LEVELS, t.log - level);
            a.levels = a.cta_log;
            for (int l = 0; l < a.levels; l++) { a.num_out[l] = t.num_l[level + 1 + l]; a.den_out[l] = t.den_l[level + 1 + l]; }
            const unsigned grid = 1u << (t.log - level - a.cta_log);
            switch (t.kind_at(level)) {
                case ZKB_GKR_GRAND_PRODUCT: launch.run("tower_kernel", tower_kernel<0>, grid, TOWER_THREADS, 0, a); break;
                case ZKB_GKR_LOGUP_GENERIC: launch.run("tower_kernel", tower_kernel<1>, grid, TOWER_THREADS, 0, a); break;
                case ZKB_GKR_LOGUP_MULTIPLICITIES: launch.run("tower_kernel", tower_kernel<2>, grid, TOWER_THREADS, 0, a); break;
                default: launch.run("tower_kernel", tower_kernel<3>, grid, TOWER_THREADS, 0, a); break;
            }
            level += a.levels;
        }
    }
    ResInit init;
    memcpy(init.digest, digest, 32);
    init.n_draws = *n_draws;
    init.use = 1;
    for (auto& s : steps) {
        launch.run("res_chain_kernel", res_chain_kernel, 1u, RES_THREADS, CHAIN_SMEM, st, (const ChainLayer*)d_chain + s.chain_first, s.chain_count, init);
        init.use = 0;
        for (auto& r : s.rounds) {
            const unsigned grid = (unsigned)std::min<size_t>(r.second.nt >> r.second.chunk_log, ROUND_MAX_CTAS);
            switch (r.first) {
                case 0: launch.run("res_round_kernel(sums)", res_round_kernel<0, false>, grid, ROUND_THREADS, 0, r.second); break;
                case 1: launch.run("res_round_kernel(sums)", res_round_kernel<1, false>, grid, ROUND_THREADS, 0, r.second); break;
                case 2: launch.run("res_round_kernel(sums)", res_round_kernel<2, false>, grid, ROUND_THREADS, 0, r.second); break;
                case 3: launch.run("res_round_kernel(sums)", res_round_kernel<3, false>, grid, ROUND_THREADS, 0, r.second); break;
                case 4: launch.run("res_round_kernel(fold)", res_round_kernel<0, true>, grid, ROUND_THREADS, 0, r.second); break;
                case 5: launch.run("res_round_kernel(fold)", res_round_kernel<1, true>, grid, ROUND_THREADS, 0, r.second); break;
                case 6: launch.run("res_round_kernel(fold)", res_round_kernel<2, true>, grid, ROUND_THREADS, 0, r.second); break;
                default: launch.run("res_round_kernel(fold)", res_round_kernel<3, true>, grid, ROUND_THREADS, 0, r.second); break;
            }
        }
    }
    if (launch.err != cudaSuccess) return set_error(ctx, ZKB_ECUDA, "gkr: %s", cudaGetErrorString(launch.err));
    // ---- one copy, one synchronisation
    if (copy_words > (size_t)SMALL_WORDS) return set_error(ctx, ZKB_EINVAL, "gkr: the proof exceeds the landing buffer");
    ZKB_CUDA(ctx, cudaMemcpyAsync(ctx->h_small, base, copy_words * 4, cudaMemcpyDeviceToHost, ctx->stream));
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const uint32_t* h = ctx->h_small;
    const ResState* hs = reinterpret_cast<const ResState*>(h + at_state);
    memcpy(digest, hs->digest, 32);
    *n_draws = hs->n_draws;
    auto put = [&](const uint32_t* q) { o.insert(o.end(), q, q + 4); };
    o.reserve(o.size() + copy_words);
    o.push_back((uint32_t)n_layers);
    const uint32_t* poly = h + at_polys;
    for (int layer = 0; layer < n_layers; layer++) {
        o.push_back((uint32_t)layer);
        for (int r = 0; r < layer; r++, poly += POLY_WORDS) {
            o.push_back(poly[16]);
            for (uint32_t j = 0; j < poly[16]; j++) put(poly + 4 * j);
        }
    }
    for (int i = 0; i < n_inst; i++) {
        o.push_back((uint32_t)towers[i].log);  // one mask per layer the instance is in
        for (int layer = n_layers - towers[i].log; layer < n_layers; layer++) {
            const size_t k = std::find(oracle_inst[layer].begin(), oracle_inst[layer].end(), i) - oracle_inst[layer].begin();
            const uint32_t* m = h + at_masks[layer] + MASK_WORDS * k;
            const uint32_t cols = towers[i].kind == ZKB_GKR_GRAND_PRODUCT ? 1u : 2u;
            o.push_back(cols);
            for (uint32_t c = 0; c < 2 * cols; c++) put(m + 4 * c);
        }
    }
    for (int i = 0; i < n_inst; i++) {
        o.push_back(hs->n_out_claims[i]);
        for (uint32_t c = 0; c < hs->n_out_claims[i]; c++) put(hs->out_claims[i][c].c);
    }
    o.push_back((uint32_t)n_layers);
    for (int j = 0; j < n_layers; j++) put(hs->ood[j].c);
    for (int i = 0; i < n_inst; i++) {
        o.push_back(hs->n_claims[i]);
        for (uint32_t c = 0; c < hs->n_claims[i]; c++) put(hs->claims[i][c].c);
    }
    return ZKB_OK;
}

}  // namespace b200
