// GKR batches of many instances (the prover's reductions hold hundreds: one instance per component and
// power-of-two share of its lookups, prover/src/gkr_key_tile.rs:34-55). prove_batch
// (nitroo/crates/stwo/src/prover/lookups/gkr_prover.rs:657-882) runs ONE sum-check per layer over all
// instances, so what every instance needs in a round is known together: a table of work items (one per
// instance) says what to do with which arrays.
//
// A whole layer's sum-check is one launch (gkr_batch_layer_begin): its CTAs take the rounds' tables one after the other, CTA 0 runs the
// transcript step between them (the batch's round polynomial, the channel, the challenge, the claims). Where the transcript of the
// rounds stays on the host, a round is a launch and a read-back (gkr_batch_round): a flat grid of CTAs is split over the items in
// proportion to their size, and every item's eight result words (and, at the end of a layer, its two-entry mask) land in one array.
//
//   mode 0  sum_as_poly_in_first_variable sums of the item's layer (first round of a layer's sum-check)
//   mode 1  fix_first_variable with the round's challenge on every column, and the sums of the fixed layer
//   mode 2  fix_first_variable of a 4-entry layer; the 2 fixed entries are also copied to the results (the mask)
//
// Arithmetic as in gkr.cu / gkr_fused.cu (cpu/lookups/gkr.rs:17-263, cpu/lookups/mle.rs:13-46).
#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "channel.cuh"
#include "common.cuh"
#include "gkr_batch.hpp"
#include "gkr_tower.cuh"

namespace zk {

namespace {

// (no __restrict__: the kernel of the small rounds reads in one round what it wrote in the round before)
__device__ __forceinline__ qm31 ldqb(const uint32_t* p, size_t i) {
    uint4 v = reinterpret_cast<const uint4*>(p)[i];
    return {{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ void stqb(uint32_t* p, size_t i, qm31 v) {
    reinterpret_cast<uint4*>(p)[i] = make_uint4(v.c[0], v.c[1], v.c[2], v.c[3]);
}
__device__ __forceinline__ qm31 foldb(qm31 r, qm31 a, qm31 b) { return qm31_mul_add(r, qm31_sub(b, a), a); }
__device__ __forceinline__ qm31 fold_m31(qm31 r, uint32_t a, uint32_t b) {
    qm31 v = qm31_mul_m31(r, m31_sub(b, a));
    v.c[0] = m31_add(v.c[0], a);
    return v;
}
// The item a CTA of the flat grid works for: the last item whose first CTA is not after this one.
__device__ __forceinline__ int find_item(const GkrBatchItem* __restrict__ items, int n_items, uint32_t block) {
    int lo = 0, hi = n_items - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (items[mid].first_block <= block) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// One term of the round sums from the four denominators (and numerators) at (0, i, {0,1}) and (1, i, {0,1}).
template <int KIND>
__device__ __forceinline__ void term(const qm31 d[4], const qm31 nu[4], qm31 lambda, qm31& t0, qm31& t2) {
    qm31 d20 = qm31_sub(qm31_dbl(d[2]), d[0]), d21 = qm31_sub(qm31_dbl(d[3]), d[1]);
    if (KIND == ZKB_GKR_GRAND_PRODUCT) {
        t0 = qm31_mul(d[0], d[1]);
        t2 = qm31_mul(d20, d21);
        return;
    }
    qm31 n0, n2;
    if (KIND == ZKB_GKR_LOGUP_SINGLES) {
        n0 = qm31_add(d[0], d[1]);
        n2 = qm31_add(d20, d21);
    } else {
        qm31 n20 = qm31_sub(qm31_dbl(nu[2]), nu[0]), n21 = qm31_sub(qm31_dbl(nu[3]), nu[1]);
        // n0 d1 + n1 d0 + lambda d0 d1 as (n0 + lambda d0) d1 + n1 d0
        t0 = qm31_dot2(qm31_mul_add(lambda, d[0], nu[0]), d[1], nu[1], d[0]);
        t2 = qm31_dot2(qm31_mul_add(lambda, d20, n20), d21, n21, d20);
        return;
    }
    t0 = qm31_mul_add(lambda, qm31_mul(d[0], d[1]), n0);
    t2 = qm31_mul_add(lambda, qm31_mul(d20, d21), n2);
}

template <int KIND>
__device__ __forceinline__ void item_sums(const GkrBatchItem& it, size_t first, size_t stride, qm31 r, const uint32_t* __restrict__ eq, qm31 lambda,
                                          qm31& s0, qm31& s2) {
    qm31_sum a0 = qm31_sum_zero(), a2 = qm31_sum_zero();
    if (it.mode == 0) {
        const size_t nt = it.n / 4;  // entries (0, i, b) at 2i + b, (1, i, b) at 2(nt + i) + b
        for (size_t i = first; i < nt; i += stride) {
            const size_t o[4] = {2 * i, 2 * i + 1, 2 * (nt + i), 2 * (nt + i) + 1};
            qm31 d[4], nu[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                d[q] = ldqb(it.den, o[q]);
                if (KIND == ZKB_GKR_LOGUP_GENERIC) nu[q] = ldqb(it.num, o[q]);
                else if (KIND == ZKB_GKR_LOGUP_MULTIPLICITIES) nu[q] = qm31_from_m31(it.num[o[q]]);
            }
            qm31 t0, t2;
            term<KIND>(d, nu, lambda, t0, t2);
            qm31 e = ldqb(eq, i);
            a0.add_product(e, t0);
            a2.add_product(e, t2);
        }
    } else {
        const size_t half = it.n / 2, nt = half / 4;
        for (size_t i = first; i < nt; i += stride) {
            const size_t o[4] = {2 * i, 2 * i + 1, 2 * (nt + i), 2 * (nt + i) + 1};
            qm31 d[4], nu[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                d[q] = foldb(r, ldqb(it.den, o[q]), ldqb(it.den, o[q] + half));
                stqb(it.den_out, o[q], d[q]);
                if (KIND == ZKB_GKR_LOGUP_GENERIC) {
                    nu[q] = foldb(r, ldqb(it.num, o[q]), ldqb(it.num, o[q] + half));
                    stqb(it.num_out, o[q], nu[q]);
                } else if (KIND == ZKB_GKR_LOGUP_MULTIPLICITIES) {
                    nu[q] = fold_m31(r, it.num[o[q]], it.num[o[q] + half]);
                    stqb(it.num_out, o[q], nu[q]);
                }
            }
            qm31 t0, t2;
            term<KIND>(d, nu, lambda, t0, t2);
            qm31 e = ldqb(eq, i);
            a0.add_product(e, t0);
            a2.add_product(e, t2);
        }
    }
    s0 = qm31_add(s0, a0.value());
    s2 = qm31_add(s2, a2.value());
}

// ---- the transcript step of a round, for a layer enqueued at once
//
// The batch's round polynomial is sum_k alpha^k (r0_k L0 + r1_k L1 + r2_k L2) over the active oracles plus the constants of those
// that wait, with r0_k = sum0_k corr_k e0a, r2_k = sum2_k corr_k e2a, r1_k = claim_k - r0_k (correct_sum, gkr_prover.rs:884-923).
// None of it needs an oracle's own record on the device:
//   * corr_k = eq(challenges since the oracle entered, point) is the same for all that entered in the same round: one per group.
//     So the sums of a group's oracles, each times alpha^k, are only needed added up, and a CTA adds its share to the group's
//     accumulator itself (8 reductions in L2; the terms are below 2^31, so 64-bit integers add up without a fold).
//   * sum_k alpha^k claim_k over the active oracles is, after a round, that round's polynomial (without the waiting constants) at
//     its challenge, plus what the oracles entering next bring; the constants are worked out on the host.
// The step is then one warp's work whatever the number of instances: two products, three compressions (channel.cuh), four products.
// (The form it replaces kept a record per oracle, passed over all of them twice per round and hashed on one thread: 5.5 us of
// hashing alone, a launch with its step 27-40 us.)
// The combination keeps the length of its longest term, each trimmed on its own (lookups/utils.rs:165-170 under sumcheck.rs:139-149). The
// step trims the sum instead, which is the same unless the longest terms' leading coefficients, times powers of alpha, cancel. Alpha is
// drawn after everything that fixes them, so they do with a chance of some K / 2^124 a round, and the proof is a valid one even then. A
// batch of constant layers (padding instances, products of ones) so takes no longer than any other.
constexpr int GKR_GROUPS = 32;  // rounds of a layer at most, so groups of oracles that enter together

struct GkrStepConst {        // of a round; host-made
    qm31 A[4], B[4], L1[4];  // e0a (L0 - L1), e2a L2 and L1, coefficients low first
    qm31 y;                  // the coordinate of the layer's point the round fixes
    qm31 waiting;            // sum of alpha^k claim_k / 2^(round + 1) over the oracles that wait
    qm31 entering;           // sum of alpha^k claim_k over those that enter in the NEXT round
    uint32_t round, pad[3];
};
static_assert(sizeof(GkrStepConst) == 256, "GkrStepConst layout");

struct alignas(16) GkrStepState {
    uint32_t digest[8], n_draws, pad[3];
    qm31 challenge, claim;                            // claim: sum of alpha^k claim_k over the active oracles
    qm31 corr[GKR_GROUPS];
};
static_assert(sizeof(GkrStepState) % 16 == 0, "GkrStepState layout");

// What of a layer's description depends on the transcript, in words: the channel (digest, n_draws), the first claim, the rounds' constants, the powers of
// alpha. It is known last, so the launch carries it as a parameter where it fits (a copy before the launch is 3 us of host time, and
// the launch behind it starts later: 34 instances of 2^10 ... 2^13 983 -> 950 us a proof); for many instances it is staged and copied.
constexpr size_t OPEN_CLAIM = 12, OPEN_CONSTS = 16, OPEN_WORDS = 2000;
struct alignas(16) GkrLayerOpen {
    uint32_t words[OPEN_WORDS];
};
__host__ __device__ inline size_t open_alpha(int n_rounds) { return OPEN_CONSTS + 64 * (size_t)n_rounds; }
// Word i of the state that a layer begins with.
__device__ __forceinline__ uint32_t open_state_word(const uint32_t* open, int i) {
    constexpr int claim = offsetof(GkrStepState, claim) / 4, corr = offsetof(GkrStepState, corr) / 4;
    return i < 9 ? open[i] : i >= claim && i < claim + 4 ? open[OPEN_CLAIM + i - claim] : i >= corr && !((i - corr) & 3) ? 1u : 0u;
}

// The groups' sums of the round at hand, and zeros for the next: [2][groups][24] 64-bit words. Of a round whose challenge is known its two sums (t =
// 0, t = 2); of one that is worked out ahead (look_pass) three pairs.
constexpr int ACC_WORDS = 24;
struct GkrAcc {
    unsigned long long* words;
    int groups;
    __device__ __forceinline__ unsigned long long* at(int round, int group) const { return words + (size_t)ACC_WORDS * ((round & 1) * groups + group); }
};

struct alignas(16) GkrStepSm {
    ChanSm ch;
    qm31 coef[4], r;
    // rounds worked out ahead: the next polynomial (but for what the waiting oracles add) as cubics in the challenge, low first; the groups' sums with
    // their corrections, of two nodes at three points; the sums of the oracles that enter next; of this round and the last the polynomial,
    // with and without the waiting, and the challenge
    qm31 ahead[16], look_sums[6], look_enter[2], look_coef[2][4], look_sent[2][4], look_r[2];
};

__device__ __noinline__ qm31 qmul(qm31 a, qm31 b) { return qm31_mul(a, b); }
struct qm31_pair { qm31 a, b; };
__device__ __noinline__ qm31_pair product_pair(qm31 a0, qm31 a1, qm31 b0, qm31 b1) { return {qm31_mul(a0, a1), qm31_mul(b0, b1)}; }
__device__ __noinline__ void chan_step_b(ChanSm& s, int n, int draws, qm31* felts) { chan_step(s, n, draws, reinterpret_cast<uint32_t*>(felts)); }
__device__ __forceinline__ qm31 shflb(qm31 v, int src) {
    qm31 r;
#pragma unroll
    for (int c = 0; c < 4; c++) r.c[c] = __shfl_sync(0xffffffffu, v.c[c], src);
    return r;
}
__device__ __forceinline__ qm31 warp_sum_m(qm31 v) {
    qm31 r;
#pragma unroll
    for (int c = 0; c < 4; c++) r.c[c] = warp_sum_m31(v.c[c]);
    return r;
}

// Coefficient (lane & 3) of the round's polynomial but for what the waiting oracles add. By one warp; s0, s2: lane g's group's sums.
__device__ __forceinline__ qm31 batch_coefficients(const GkrStepState& st, const GkrStepConst& rc, qm31 corr, qm31 s0, qm31 s2) {
    const int lane = threadIdx.x & 31, c4 = lane & 3;
    const qm31_pair w = product_pair(s0, corr, s2, corr);
    const qm31 S0 = warp_sum_m(w.a), S2 = warp_sum_m(w.b);
    // coefficient c4: lanes 0-3 of the first sum, 4-7 of the second, 8-11 of the claim
    const int q = lane >> 2;
    const qm31 p = qmul(q == 0 ? S0 : q == 1 ? S2 : st.claim, q == 0 ? rc.A[c4] : q == 1 ? rc.B[c4] : rc.L1[c4]);
    return qm31_add(qm31_add(p, shflb(p, (lane + 4) & 31)), shflb(p, (lane + 8) & 31));
}
// By one warp; sm.ch's schedule is made and its message holds the digest. st: the state, wherever it is; s0, s2: lane g's group's sums; out: the
// round's record. drawn() is called as soon as the challenge is in sm.r, before what the next step needs of it is worked out.
template <class Drawn>
__device__ __forceinline__ void batch_step(GkrStepSm& sm, GkrStepState& st, const GkrStepConst& rc, qm31 s0, qm31 s2, uint32_t* out, Drawn drawn) {
    const int lane = threadIdx.x & 31;
    const qm31 corr = st.corr[lane], act = batch_coefficients(st, rc, corr, s0, s2);
    const qm31 c = lane == 0 ? qm31_add(act, rc.waiting) : act;
    const int len = 32 - __clz(__ballot_sync(0xffffffffu, lane < 4 && !qm31_is_zero(c)));
    if (lane < 4) {
        sm.coef[lane] = act;
        stqb(sm.ch.msg + 8, lane, c);
    }
    chan_step_b(sm.ch, 4 * len, 1, &sm.r);
    const qm31 r = sm.r, y = rc.y, one = qm31_one();
    drawn();
    if (lane < 4) stqb(out, lane, c);
    if (lane == 0) out[16] = (uint32_t)len;
    // (c3 r + c2) r^2 + (c1 r + c0), eq(r, y)
    qm31 x = r, z = r;
    if (lane == 0) x = sm.coef[3];
    if (lane == 1) x = sm.coef[1];
    if (lane == 3) z = y;
    if (lane == 4) { x = qm31_sub(one, r); z = qm31_sub(one, y); }
    qm31 m = qmul(x, z);
    if (lane < 2) m = qm31_add(m, sm.coef[lane == 0 ? 2 : 0]);
    const qm31 hi = shflb(m, 0), lo = shflb(m, 1), r2 = shflb(m, 2), step = qm31_add(shflb(m, 3), shflb(m, 4));
    // lane 31: the claim; the others: their group's correction (a group that enters next starts at one)
    const qm31 v = qmul(lane == 31 ? hi : corr, lane == 31 ? r2 : step);
    __syncwarp();
    if (lane == 31) st.claim = qm31_add(qm31_add(v, lo), rc.entering);
    else if (lane <= (int)rc.round) st.corr[lane] = v;
    if (lane == 0) st.challenge = r;
    if (lane < 4) out[20 + lane] = r.c[lane];
    __syncwarp();
}
__device__ __forceinline__ void batch_step_open(GkrStepSm& sm, const GkrStepState& st, int lane) {
    chan_make_schedule(sm.ch, lane, 32);
    sm.ch.msg[lane] = lane < 8 ? st.digest[lane] : 0u;
    if (lane == 0) sm.ch.n_draws = st.n_draws;
    __syncwarp();
}
// The channel's state (digest, n_draws) to where the next launch, or the host, finds it.
__device__ __forceinline__ void batch_step_close(const GkrStepSm& sm, uint32_t* channel, int lane) {
    const uint32_t w = lane < 8 ? sm.ch.msg[lane] : lane == 8 ? sm.ch.n_draws : 0u;
    if (lane < 12) channel[lane] = w;
}

// What a layer brings back is written by its last launch into page-locked host memory (the masks by the threads that fix them; the
// rounds' records and the channel, which the launches before keep on the device, by `threads` threads at the end), then the layer's
// number: the host has it a PCIe write after the last round, without a copy and a stream synchronisation of its own.
struct GkrLayerOut {
    uint32_t *records, *channel, *masks;  // host
    volatile unsigned int* flag;
    unsigned int id;
};
__device__ __forceinline__ void layer_out_words(const GkrLayerOut& o, const uint32_t* records, int n_rounds, int i, int threads) {
    for (int k = i; k < 6 * n_rounds; k += threads) reinterpret_cast<uint4*>(o.records)[k] = reinterpret_cast<const uint4*>(records)[k];
}
__device__ __forceinline__ qm31 acc_value(const unsigned long long* a) { return {{m31_reduce64(a[0]), m31_reduce64(a[1]), m31_reduce64(a[2]), m31_reduce64(a[3])}}; }

// Fixes a 4-entry layer, one thread per entry: the mask, also in the oracle's record.
__device__ __forceinline__ void fix_mask(const GkrBatchItem& it, int e, qm31 r, uint32_t* res) {
    const qm31 dv = foldb(r, ldqb(it.den, e), ldqb(it.den, e + 2));
    stqb(it.den_out, e, dv);
    stqb(res, e, dv);
    if (it.kind == ZKB_GKR_LOGUP_GENERIC || it.kind == ZKB_GKR_LOGUP_MULTIPLICITIES) {
        const qm31 nv = it.kind == ZKB_GKR_LOGUP_GENERIC ? foldb(r, ldqb(it.num, e), ldqb(it.num, e + 2)) : fold_m31(r, it.num[e], it.num[e + 2]);
        stqb(it.num_out, e, nv);
        stqb(res + 8, e, nv);
    }
}
__device__ __forceinline__ void item_sums_of(const GkrBatchItem& it, size_t first, size_t stride, qm31 r, const uint32_t* __restrict__ eq, qm31 lambda, qm31& s0, qm31& s2) {
    switch (it.kind) {
        case ZKB_GKR_GRAND_PRODUCT: item_sums<ZKB_GKR_GRAND_PRODUCT>(it, first, stride, r, eq, lambda, s0, s2); break;
        case ZKB_GKR_LOGUP_GENERIC: item_sums<ZKB_GKR_LOGUP_GENERIC>(it, first, stride, r, eq, lambda, s0, s2); break;
        case ZKB_GKR_LOGUP_MULTIPLICITIES: item_sums<ZKB_GKR_LOGUP_MULTIPLICITIES>(it, first, stride, r, eq, lambda, s0, s2); break;
        default: item_sums<ZKB_GKR_LOGUP_SINGLES>(it, first, stride, r, eq, lambda, s0, s2); break;
    }
}

// The terms of `g` neighbouring lanes (a power of two up to 32) are one item's: they are added up, taken times the item's power of
// alpha and added to its group's sums in shared memory, as 16-bit halves (32-bit adds, no carries to fold; 2^16 additions
// fit: a piece makes 16 to a counter for items of 32 terms and more, and the largest layer that 180 GB hold, 2^31 terms, is some 3,600 pieces for
// each of 148 CTAs; smaller items, of which a launch has at most 2^13, are two pieces). By whole warps; adds: the lane belongs to an item.
__device__ __forceinline__ void add_to_group(uint32_t (*acc)[2 * ACC_WORDS], int g, bool adds, uint32_t oracle, uint32_t group, const uint32_t* __restrict__ alpha_pow, qm31 s0, qm31 s2) {
    const int lane = threadIdx.x & 31, sub = lane & (g - 1);
    const qm31 a = adds ? ldqb(alpha_pow, oracle) : qm31_zero();
    for (int off = g >> 1; off > 0; off >>= 1) {
        s0 = qm31_add(s0, shflb(s0, (lane & ~(g - 1)) | ((sub + off) & (g - 1))));
        s2 = qm31_add(s2, shflb(s2, (lane & ~(g - 1)) | ((sub + off) & (g - 1))));
    }
    adds = adds && sub == 0;
    const unsigned who = __ballot_sync(0xffffffffu, adds);
    if (!who) return;
    const qm31 v0 = qmul(s0, a), v2 = qmul(s2, a);
    const uint32_t g0 = __shfl_sync(0xffffffffu, group, __ffs(who) - 1);
    if (__all_sync(0xffffffffu, !adds || group == g0)) {  // one group in the warp: add up before going to memory
        const qm31 a0 = warp_sum_m(adds ? v0 : qm31_zero()), a2 = warp_sum_m(adds ? v2 : qm31_zero());
        uint32_t w = 0;
#pragma unroll
        for (int c = 0; c < 4; c++) { w = (lane >> 1) == c ? a0.c[c] : w; w = (lane >> 1) == 4 + c ? a2.c[c] : w; }
        if (lane < 16) atomicAdd(&acc[g0][lane], (lane & 1) ? w >> 16 : w & 0xffffu);
    } else if (adds) {
#pragma unroll
        for (int c = 0; c < 4; c++) {
            atomicAdd(&acc[group][2 * c], v0.c[c] & 0xffffu);
            atomicAdd(&acc[group][2 * c + 1], v0.c[c] >> 16);
            atomicAdd(&acc[group][8 + 2 * c], v2.c[c] & 0xffffu);
            atomicAdd(&acc[group][8 + 2 * c + 1], v2.c[c] >> 16);
        }
    }
}

// ---- a layer in one launch
//
// A cooperative launch of up to a CTA an SM runs all tables of a layer. Measured with a launch per round: of the 26,500 cycles (14 us)
// that every round of a small batch took, whatever its size, half were the fetching of code that the SM at hand had not run
// yet (the pass 14,500 cycles cold and 6,300 warm, the transcript step 12,000 and 8,000) and the rest of the gap the launch
// itself; a round in one CTA took 9.3 us warm. Here the code stays warm in every SM, CTA 0 keeps the transcript in shared memory and
// what goes round in a round is a count of arrivals and a challenge.
//
// A pass has two forms. With many terms a thread takes whole terms (bound by their 18 products). With few, what counts is the length of
// the chain: four lanes take a term, one for each of its four entries, and every product is half of a pair (product_pair): a
// sixth of the instructions and six products one after the other.
//
// The waits end: every CTA is resident (the launch is refused otherwise), a CTA waits only for what the others do before they wait
// themselves, and after SPIN_LIMIT polls (about a second) it gives up and leaves; the host then sees no layer number and reports it.
constexpr int GKR_THREADS = 1 << GKR_THREADS_LOG;
constexpr int LOOK_MIN_LOG = 7;                  // the fewest threads (log2) that a CTA is given work for
constexpr uint32_t SPIN_LIMIT = 1u << 21;

constexpr int EQ_TABLES = GKR_EQ_BITS / 5;       // of five bits of a term's index each

struct alignas(16) GkrTable {
    uint32_t first, n_items;  // its items
    int terms_log;            // log2 of the terms an item has
    int form;                 // 0: a thread per term, 1: four lanes per term, 2: masks, two threads an item; 3: a pass of a round ahead, 4: the last of them
    int run_log;              // form 0, items of 2^GKR_THREADS_LOG terms and more: a chunk is 2^run_log terms a thread; the other forms: a chunk is 2^run_log threads
    uint32_t chunks, ctas;    // pieces of work, CTAs that take them in turn
    uint32_t later;           // the most CTAs a later table has
};
static_assert(sizeof(GkrTable) == 32, "GkrTable layout");

struct alignas(16) GkrSync {  // zero at launch
    uint32_t count[GKR_LAYER_MAX_ROUNDS + 1];   // CTAs done with the table
    uint32_t slot[GKR_LAYER_MAX_ROUNDS + 1][4];  // the challenge the table folds with; the top bit of a word: it is there
    uint32_t look_count[GKR_LAYER_MAX_ROUNDS + 1];  // CTAs done with a pass of a round ahead
};
static_assert(sizeof(GkrSync) % 16 == 0, "GkrSync layout");


// The sums of `v` over the warp's lanes with even and odd `which` go to the group's accumulator; lanes that do not add hold `adds` false.
__device__ __forceinline__ void add_quad_terms(uint32_t (*acc)[2 * ACC_WORDS], bool adds, int which, uint32_t group, qm31 v) {
    const int lane = threadIdx.x & 31;
    const unsigned who = __ballot_sync(0xffffffffu, adds);
    if (!who) return;
    const uint32_t g0 = __shfl_sync(0xffffffffu, group, __ffs(who) - 1);
    if (__all_sync(0xffffffffu, !adds || group == g0)) {
        uint32_t w = 0;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint32_t e = warp_sum_m31(adds && which == 0 ? v.c[c] : 0u), o = warp_sum_m31(adds && which == 1 ? v.c[c] : 0u);
            w = (lane >> 1) == c ? e : w;
            w = (lane >> 1) == 4 + c ? o : w;
        }
        if (lane < 16) atomicAdd(&acc[g0][lane], (lane & 1) ? w >> 16 : w & 0xffffu);
    } else if (adds) {
#pragma unroll
        for (int c = 0; c < 4; c++) {
            atomicAdd(&acc[group][8 * which + 2 * c], v.c[c] & 0xffffu);
            atomicAdd(&acc[group][8 * which + 2 * c + 1], v.c[c] >> 16);
        }
    }
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// ---- the small rounds, a round ahead of the transcript
//
// A round is a chain: the challenge goes out, the CTAs fold and sum, their sums come back (together some 9,000 cycles however small the round), the
// transcript's three compressions follow (4,400). A layer fixed at r is linear in r and a term is a product of two entries, so a group's sums of the next
// round are quadratic in this round's challenge, and its correction is linear. From round look_from on, then, the CTAs work on the round after the one that is being
// hashed: they fold with the challenge before, and bring back the next round's sums at r = 0, at r = 1 and their leading coefficient; warps of CTA 0 make
// of those the next polynomial as cubics in the challenge to come. When the challenge is there the next polynomial is two products away. The two chains
// run beside each other: 16,000 cycles a round before, 9,500 after (34 instances of 2^13). The CTAs' chain is the longer one (hash and challenge 5,000), so what can
// stand beside it does: the fence before the next challenge, and the loads of the next pass's entries, which are there some 2,000 cycles before the
// challenge they are fixed at (34 instances 904 -> 868 us a proof, micro segment 14.56 -> 14.37 ms). The sums' words counting the CTAs themselves, instead of a
// count behind a fence, gained nothing more (857 of 895 us).
//
// CTA 0 keeps the transcript and takes no pieces: warp 0 hashes, six warps take a node and point each, one makes the polynomial of them, one sends the challenge. Those are on other
// schedulers than warp 0, and the CTA has its SM to itself (a CTA an SM: with two of half the size the hash beside a worker took 5,700 cycles instead of 4,200).
constexpr int LOOK_SUM_WARPS = 6, LOOK_LAST_WARP = 9, LOOK_SEND_WARP = 10;
static_assert(GKR_THREADS / 32 > LOOK_SEND_WARP, "the warps of CTA 0");
__device__ __forceinline__ int look_value(int warp) {  // 1-3, 5-7
    return warp == LOOK_LAST_WARP || warp == LOOK_SEND_WARP ? LOOK_SUM_WARPS : warp < 8 && (warp & 3) ? warp - 1 - (warp >> 2) : -1;
}

// What a pass does for an item: the layer is there / fix it at the challenge first / it enters in the next round (nothing but its sums then).
enum : uint32_t { LOOK_AS_IS = 0, LOOK_FIX = 1, LOOK_ENTERS = 2 };

__device__ __forceinline__ bool wait_count(const uint32_t* count, uint32_t want) {
    uint32_t n = ld_acquire(count);
    for (uint32_t spin = 0; n != want && spin < SPIN_LIMIT; spin++) n = ld_acquire(count);
    return n == want;
}

// One entry of a layer: its denominator and numerator (one where the kind has none, zero for a grand product).
struct entry { qm31 d, n; };
__device__ __forceinline__ entry load_entry(const GkrBatchItem& it, size_t e) {
    entry v{ldqb(it.den, e), qm31_zero()};
    if (it.kind == ZKB_GKR_LOGUP_SINGLES) v.n = qm31_one();
    if (it.kind == ZKB_GKR_LOGUP_GENERIC) v.n = ldqb(it.num, e);
    if (it.kind == ZKB_GKR_LOGUP_MULTIPLICITIES) v.n = qm31_from_m31(it.num[e]);
    return v;
}
// The entry fixed at r, also where the folded layer goes: v0, v1 are entries e and e + half of the layer, half the entries of the folded one.
__device__ __forceinline__ entry fix_entry(const GkrBatchItem& it, size_t e, entry v0, entry v1, qm31 r) {
    const qm31_pair p = product_pair(r, qm31_sub(v1.d, v0.d), r, qm31_sub(v1.n, v0.n));
    const entry v{qm31_add(v0.d, p.a), qm31_add(v0.n, p.b)};
    stqb(it.den_out, e, v.d);
    if (it.kind == ZKB_GKR_LOGUP_GENERIC || it.kind == ZKB_GKR_LOGUP_MULTIPLICITIES) stqb(it.num_out, e, v.n);
    return v;
}

// Eight lanes a term of the next round, one for each of its entries: bit 2 the variable this round fixes, bit 1 the next round's, bit 0 the pair. A term is
// n0 d1 + n1 d0 + lambda d0 d1 = m0 d1 + m1 d0 with m = n + k d, k = lambda / 2 (a grand product's d0 d1 with n = 0, k = 1 / 2). Lanes 0 and 2 end with the term at r
// = 0, 4 and 6 with it at r = 1, 5 and 7 with its leading coefficient. ea: eq times the oracle's power of alpha. The sums are 16-bit halves as in
// add_to_group: at most 64 additions a piece to a counter, and gkr_look_from allows few pieces.
__device__ __forceinline__ size_t look_entry(uint32_t term, int terms_log) {  // this lane's
    const int q = threadIdx.x & 7;
    const size_t nt = (size_t)1 << terms_log;
    return (size_t)(q >> 2) * 4 * nt + (size_t)((q >> 1) & 1) * 2 * nt + 2 * (size_t)term + (q & 1);
}
__device__ __forceinline__ bool look_live(const GkrBatchItem& it) { return !(it.mode == LOOK_ENTERS && (threadIdx.x & 4)); }
// v0: the lane's entry, v1: the one it is fixed with, where there is one
__device__ __forceinline__ void look_term(uint32_t (*acc)[2 * ACC_WORDS], const GkrBatchItem& it, bool live, uint32_t term, int terms_log, entry v0, entry v1, qm31 r,
                                          qm31 half_lambda, qm31 ea) {
    const int lane = threadIdx.x & 31, q = lane & 7;
    live = live && look_live(it);
    entry v{qm31_zero(), qm31_zero()};
    if (live) v = it.mode == LOOK_FIX ? fix_entry(it, look_entry(term, terms_log), v0, v1, r) : v0;
    qm31 x = v.d, m = qm31_add(v.n, qmul(it.kind == ZKB_GKR_GRAND_PRODUCT ? qm31_from_m31(1u << 30) : half_lambda, x));
    const qm31 x0 = shflb(x, lane & ~2), m0 = shflb(m, lane & ~2);
    if (q & 2) { x = qm31_sub(qm31_dbl(x), x0); m = qm31_sub(qm31_dbl(m), m0); }
    const qm31 xp = shflb(x, lane ^ 1);
    const qm31 xp0 = shflb(xp, lane & ~4), mm0 = shflb(m, lane & ~4);
    const qm31_pair p = product_pair(m, xp, qm31_sub(m, mm0), qm31_sub(xp, xp0));
    const qm31 a = qm31_add(p.a, shflb(p.a, lane ^ 1)), b = qm31_add(p.b, shflb(p.b, lane ^ 1));
    const bool adds = live && (it.mode == LOOK_ENTERS ? !(q & 1) : q != 1 && q != 3);
    qm31 t = qmul((q & 1) ? b : a, ea);
    // value 2 point + node
    const uint32_t value = 2 * ((q >> 2) + (q & 1)) + ((q >> 1) & 1), group = (uint32_t)(it.slot >> 32);
    const unsigned who = __ballot_sync(0xffffffffu, adds);
    if (!who) return;
    const uint32_t g0 = __shfl_sync(0xffffffffu, group, __ffs(who) - 1);
    bool mine = adds;
    if (__all_sync(0xffffffffu, !adds || group == g0)) {  // one group in the warp: the same value's lanes first
        if (!adds) t = qm31_zero();
        t = qm31_add(t, shflb(t, lane ^ 8));
        t = qm31_add(t, shflb(t, lane ^ 16));
        mine = lane < 8 && (who & (0x01010101u << lane)) != 0u;
    }
    if (mine) {
        uint32_t* const at = &acc[adds ? group : g0][8 * value];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            atomicAdd(at + 2 * c, t.c[c] & 0xffffu);
            atomicAdd(at + 2 * c + 1, t.c[c] >> 16);
        }
    }
}

// Warp 0 of CTA 0: the rounds from `from` on. act0: coefficient (lane & 3) of the first one's polynomial. `met` is the meeting with the other warps
// once a round: the challenge is there, and so is `ahead`.
__device__ __forceinline__ void look_met() { asm volatile("bar.sync 1, %0;" ::"n"(32 * (LOOK_SUM_WARPS + 3)) : "memory"); }
__device__ __noinline__ void look_lead(GkrStepSm& sm, const GkrStepConst* consts, int from, int n_rounds, qm31 act0) {
    const int lane = threadIdx.x & 31, c4 = lane & 3;
    const QuadWords words(sm.ch.msg, sm.ch.sched);
    const QuadConst qc;
    const qm31 mine = shflb(act0, (lane >> 2) & 3);
    uint32_t act = c4 == 0 ? mine.c[0] : c4 == 1 ? mine.c[1] : c4 == 2 ? mine.c[2] : mine.c[3];  // lane = 4 k + coordinate: coefficient k
    qm31 r = qm31_zero();
    for (int round = from;; round++) {
        if (round > from) {
            // (d3 r + d2) r^2 + (d1 r + d0): the low half in lanes 0-15, the high one in 16-31
            const int at = (lane & 12) + (lane >> 4) * 2;
            const qm31 d1 = ldqb(reinterpret_cast<const uint32_t*>(sm.ahead), at + 1);
            const uint32_t d0 = sm.ahead[at].c[c4];
            const slice_by by(r);
            const uint32_t m = by.mul_add(d1, d0), r2 = by.mul_add(r, 0u);
            act = slice_by(gather_q(r2, 0)).mul_add(gather_q(m, 16 + (lane & 12)), m);
        }
        const uint32_t c = lane < 4 ? m31_add(act, consts[round].waiting.c[lane]) : act;
        if (lane < 16) sm.ch.msg[8 + lane] = c;
        const unsigned nonzero = __ballot_sync(0xffffffffu, lane < 16 && c != 0u);
        if (!(nonzero & 0xff00u)) {  // two coefficients or fewer
            __syncwarp();
            chan_copy_digest(sm.ch);
            if (lane < 8) sm.ch.msg[24 + lane] = c;
        }
        __syncwarp();
        const uint32_t v = chan_round(
            sm.ch, words, qc, (nonzero & 0xff00u) != 0u, 0u, [&] { return 32u + 16u * (uint32_t)((35 - __clz(nonzero)) >> 2); },
            [&] {
                if (lane < 16) {
                    sm.look_coef[round & 1][lane >> 2].c[c4] = act;
                    sm.look_sent[round & 1][lane >> 2].c[c4] = c;
                }
                __syncwarp();
                if (round + 1 < n_rounds) asm volatile("bar.arrive 3, 64;" ::: "memory");
            });
        if (lane < 4) sm.look_r[round & 1].c[lane] = v;
        r = gather_q(v, 0);
        __syncwarp();
        look_met();
        if (round + 1 == n_rounds) return;
    }
}
// The warps of CTA 0 with a look_value. Returns whether a wait has run out.
__device__ __forceinline__ bool look_helpers(GkrStepSm& sm, const GkrStepConst* consts, const GkrTable* looks, const GkrStepState& s, const GkrAcc acc, GkrSync* sync, int from,
                                             int n_rounds, uint32_t* records) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = (lane >> 2) & 3, k = lane & 3, hn = lane >> 4;
    const bool last_warp = warp == LOOK_LAST_WARP, sends = warp == LOOK_SEND_WARP;
    const int value = look_value(warp), node = value & 1;
    qm31 corr = s.corr[lane];  // group `lane`'s
    bool gave_up = false;
    auto record = [&](int round) {  // by warp 2
        const uint32_t* const sent = sm.look_sent[round & 1][0].c;
        uint32_t* const out = records + GKR_LAYER_OUT_WORDS * (size_t)round;
        const uint32_t w = lane < 16 ? sent[lane] : 0u;
        const unsigned nonzero = __ballot_sync(0xffffffffu, w != 0u);
        if (lane < 16) out[lane] = w;
        if (lane == 16) out[16] = (uint32_t)((35 - __clz(nonzero)) >> 2);
        if (lane >= 20 && lane < 24) out[lane] = sm.look_r[round & 1].c[lane - 20];
    };
    for (int round = from; round < n_rounds; round++) {
        const bool next = round + 1 < n_rounds;
        const GkrStepConst &rc = consts[round], &rn = consts[next ? round + 1 : round];
        const GkrTable& tb = looks[round];
        const qm31 w0 = qm31_sub(qm31_one(), rc.y), w1 = qm31_sub(rc.y, w0);  // the next correction is corr (w0 + w1 r)
        if (sends) {
            // What the CTAs have folded, and the zeros of the round before, have to be there before the challenge that follows: the fence, some 700 cycles,
            // stands beside the sums' way to the next polynomial.
            if (!gave_up && tb.ctas && !wait_count(&sync->look_count[round], tb.ctas)) gave_up = true;
            gave_up = __any_sync(0xffffffffu, gave_up);
            __threadfence();
        } else if (!last_warp) {
            if (round > from) {
                const qm31 r = sm.look_r[(round & 1) ^ 1], y = consts[round - 1].y, omy = qm31_sub(qm31_one(), y);
                const qm31_pair p = product_pair(r, y, qm31_sub(qm31_one(), r), omy);
                const qm31 up = qmul(corr, qm31_add(p.a, p.b));
                if (lane < round) corr = up;
                if (warp == 2) record(round - 1);
            }
            if (!gave_up && tb.ctas && !wait_count(&sync->look_count[round], tb.ctas)) gave_up = true;
            gave_up = __any_sync(0xffffffffu, gave_up);
            if (next) {
                unsigned long long* const a = acc.at(round + 1, lane) + 4 * value;
                const bool mine = lane < acc.groups && !gave_up;
                ulonglong2 lo = make_ulonglong2(0ull, 0ull), hi = lo;
                if (mine) { lo = __ldcg(reinterpret_cast<const ulonglong2*>(a)); hi = __ldcg(reinterpret_cast<const ulonglong2*>(a) + 1); }
                const qm31 v{{m31_reduce64(lo.x), m31_reduce64(lo.y), m31_reduce64(hi.x), m31_reduce64(hi.y)}};
                const qm31 sum = warp_sum_m(lane <= round ? qmul(v, corr) : qm31_zero());
                if (lane == round + 1 && value < 2) sm.look_enter[node] = v;
                if (lane == 0) sm.look_sums[value] = sum;
                __syncwarp();
                asm volatile("bar.arrive 2, %0;" ::"n"(32 * (LOOK_SUM_WARPS + 1)) : "memory");
                if (mine) reinterpret_cast<ulonglong2*>(a)[0] = reinterpret_cast<ulonglong2*>(a)[1] = make_ulonglong2(0ull, 0ull);  // for the round after the next
            }
        } else if (next) {
            // lane = 16 node + 4 c + k: that node's share of the coefficient of r^k in coefficient c
            const qm31 a = hn ? rn.B[c] : rn.A[c], a0 = qmul(a, w0), a1 = k == 0 ? a : qmul(a, w1), l1 = rn.L1[c];
            asm volatile("bar.sync 3, 64;" ::: "memory");  // this round's polynomial: its value at r, and what enters, is the next claim
            const qm31 claim = hn ? qm31_zero() : k == 0 ? qm31_add(sm.look_coef[round & 1][0], rc.entering) : sm.look_coef[round & 1][k];
            const qm31 q = qmul(claim, l1);
            asm volatile("bar.sync 2, %0;" ::"n"(32 * (LOOK_SUM_WARPS + 1)) : "memory");
            const qm31 s0 = sm.look_sums[hn], s1 = sm.look_sums[2 + hn], s2 = sm.look_sums[4 + hn], mid = qm31_sub(s1, qm31_add(s0, s2));
            const qm31 lo = k == 0 ? s0 : k == 1 ? mid : k == 2 ? s2 : qm31_zero(), hi = k == 0 ? sm.look_enter[hn] : k == 1 ? s0 : k == 2 ? mid : s2;
            const qm31_pair p = product_pair(a0, lo, a1, hi);
            qm31 v = qm31_add(qm31_add(p.a, p.b), q);
            v = qm31_add(v, shflb(v, lane ^ 16));
            if (lane < 16) sm.ahead[lane] = v;
        }
        look_met();
        if (sends && next && lane < 4 && !gave_up) *reinterpret_cast<volatile uint32_t*>(&sync->slot[round + 1][lane]) = sm.look_r[round & 1].c[lane] | 0x80000000u;
    }
    if (warp == 2) record(n_rounds - 1);
    return gave_up;
}

// Tables [first, end) of the layer; then, where look_from >= 0, the rounds from that on ahead of the transcript (the tables behind the n_rounds + 1 of the others) and
// the masks; end is look_from + 1. keeps_transcript: zero where the transcript's steps are launches of their own (gkr_batch_step_kernel); no CTA then
// keeps it, and the challenge is in its slot before the launch. copied: what the launch does not carry (GkrLayerOpen), or null.
__global__ void __launch_bounds__(GKR_THREADS, 1) gkr_batch_layer_kernel(const GkrBatchItem* __restrict__ items_base, const GkrTable* __restrict__ tables, int first, int end,
                                                                         const uint32_t* __restrict__ eq, qm31 lambda, const __grid_constant__ GkrLayerOpen carried,
                                                                         const uint32_t* copied, GkrStepState* st, GkrAcc acc, GkrSync* sync, int keeps_transcript,
                                                                         int look_from, uint32_t* records, int n_rounds, GkrLayerOut host) {
    __shared__ uint32_t sums[GKR_GROUPS][2 * ACC_WORDS];  // of the pass at hand; zero before it
    __shared__ GkrTable tabs[2 * GKR_LAYER_MAX_ROUNDS + 1];
    __shared__ qm31 r_sh, eq_tab[EQ_TABLES][32];
    __shared__ bool gave_up;
    // CTA 0 only: the transcript
    __shared__ GkrStepSm sm;
    __shared__ GkrStepState s;
    __shared__ GkrStepConst consts[GKR_LAYER_MAX_ROUNDS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool lead = blockIdx.x == 0 && keeps_transcript;
    const uint32_t* const open = copied ? copied : carried.words;
    const GkrStepConst* const rc = reinterpret_cast<const GkrStepConst*>(open + OPEN_CONSTS);
    const uint32_t* const alpha_pow = open + open_alpha(n_rounds);
    for (int i = tid; i < 2 * (look_from >= 0 ? 2 * n_rounds + 1 : end); i += GKR_THREADS) reinterpret_cast<uint4*>(tabs)[i] = reinterpret_cast<const uint4*>(tables)[i];
    for (int i = tid; i < GKR_GROUPS * 2 * ACC_WORDS; i += GKR_THREADS) (&sums[0][0])[i] = 0u;
    if (tid == 0) gave_up = false;
    if (lead) {
        for (int i = tid; i < 16 * n_rounds; i += GKR_THREADS) reinterpret_cast<uint4*>(consts)[i] = reinterpret_cast<const uint4*>(rc)[i];
        for (int i = tid; i < (int)(sizeof(s) / 4); i += GKR_THREADS) reinterpret_cast<uint32_t*>(&s)[i] = open_state_word(open, i);
    }
    // eq(., point) of a term's index: from a table, or, where there is none, as a product over the index's bits, five to a table of a warp's making
    // (bit k goes with coordinate n_rounds - 1 - k; the first coordinate's share is 1 - y)
    if (!eq && warp < EQ_TABLES) {
        auto factor = [&](int b) {
            const int bit = 5 * warp + b;
            const qm31 y = bit < n_rounds - 1 ? rc[n_rounds - 1 - bit].y : qm31_zero();
            return (lane >> b) & 1 ? y : qm31_sub(qm31_one(), y);
        };
        qm31 v = factor(4);
        if (warp == 0) v = qmul(v, qm31_sub(qm31_one(), rc[0].y));
        const qm31_pair p = product_pair(factor(0), factor(1), factor(2), factor(3));
        eq_tab[warp][lane] = qmul(v, qmul(p.a, p.b));
    }
    __syncthreads();
    auto eq_at = [&](uint32_t i) {
        if (eq) return ldqb(eq, i);
        const qm31 low = qmul(eq_tab[0][i & 31], eq_tab[1][(i >> 5) & 31]);
        return qmul(low, eq_tab[2][i >> 10]);
    };
    if (lead && warp == 0) batch_step_open(sm, s, lane);
    for (int t = first; t < end; t++) {
        const GkrTable tb = tabs[t];
        if (blockIdx.x >= tb.ctas) {
            if (blockIdx.x >= tb.later) return;
            continue;
        }
        const GkrBatchItem* const items = items_base + tb.first;
        const bool step = t < n_rounds;
        // what does not depend on the challenge: the first piece's item, in the small form its factor of the sums
        // CTA 0 has the last piece, its first warp the end of it: often there is nothing there, and that warp comes late (below).
        uint32_t chunk = tb.form == 0 ? blockIdx.x : tb.ctas - 1u - blockIdx.x;
        GkrBatchItem it{};
        uint32_t term = 0;
        bool live = false;
        qm31 ea = qm31_zero();
        auto look_up = [&]() {  // forms 1 and 2
            const uint32_t mine = (tid + GKR_THREADS - 32) & (GKR_THREADS - 1), flat = (chunk << tb.run_log) + mine;
            const uint32_t at = tb.form == 1 ? flat >> 2 : flat;
            term = at & ((1u << tb.terms_log) - 1);
            live = (at >> tb.terms_log) < tb.n_items && !(mine >> tb.run_log);
            if (live) it = items[at >> tb.terms_log];
            if (tb.form == 1 && live) ea = qmul(eq_at(term), ldqb(alpha_pow, (uint32_t)it.slot));
        };
        if (tb.form != 0) look_up();
        if (!lead && t > 0) {
            if (tid < 4) {
                uint32_t w = ld_acquire(&sync->slot[t][tid]);
                for (uint32_t spin = 0; !(w >> 31) && spin < SPIN_LIMIT; spin++) w = ld_acquire(&sync->slot[t][tid]);
                if (!(w >> 31)) gave_up = true;
                r_sh.c[tid] = w & 0x7fffffffu;
            }
            __syncthreads();
            if (gave_up) return;
        }
        const qm31 r = lead ? sm.r : r_sh;
        if (tb.form == 1) {
            for (;;) {
                const int q = lane & 3;
                const uint32_t group = (uint32_t)(it.slot >> 32);
                const size_t nt = (size_t)1 << tb.terms_log, o = 2 * ((size_t)(q >> 1) * nt + term) + (q & 1);
                const bool nums = it.kind == ZKB_GKR_LOGUP_GENERIC || it.kind == ZKB_GKR_LOGUP_MULTIPLICITIES, base = it.kind == ZKB_GKR_LOGUP_MULTIPLICITIES;
                qm31 x = qm31_zero(), u = qm31_one();  // the entry's denominator and numerator
                if (live) {
                    x = ldqb(it.den, o);
                    if (nums) u = base ? qm31_from_m31(it.num[o]) : ldqb(it.num, o);
                    if (it.mode == 1) {
                        const qm31 x1 = ldqb(it.den, o + 4 * nt);
                        const qm31 u1 = !nums ? u : base ? qm31_from_m31(it.num[o + 4 * nt]) : ldqb(it.num, o + 4 * nt);
                        const qm31_pair p = product_pair(r, qm31_sub(x1, x), r, qm31_sub(u1, u));
                        x = qm31_add(x, p.a);
                        u = qm31_add(u, p.b);
                        stqb(it.den_out, o, x);
                        if (nums) stqb(it.num_out, o, u);
                    }
                }
                // lanes 2 and 3 go on with the entries' values at two
                const qm31 x0 = shflb(x, lane & ~2), u0 = shflb(u, lane & ~2);
                if (q & 2) { x = qm31_sub(qm31_dbl(x), x0); u = qm31_sub(qm31_dbl(u), u0); }
                const qm31 xp = shflb(x, lane ^ 1);
                const qm31_pair p = product_pair(xp, u, x, xp);  // half of the numerator; the denominator
                qm31 n = qm31_add(p.a, shflb(p.a, lane ^ 1));
                const qm31 d = qmul(lambda, p.b);
                const qm31 v = qmul(it.kind == ZKB_GKR_GRAND_PRODUCT ? p.b : qm31_add(n, d), ea);
                add_quad_terms(sums, live && !(q & 1), q >> 1, group, v);
                chunk += tb.ctas;
                if (chunk >= tb.chunks) break;
                look_up();
            }
        } else if (tb.form == 0) {
            for (; chunk < tb.chunks; chunk += tb.ctas) {
                qm31 s0 = qm31_zero(), s2 = qm31_zero();
                const int whole = tb.terms_log - GKR_THREADS_LOG - tb.run_log;  // log2 of an item's chunks
                const uint32_t flat = chunk * GKR_THREADS + tid;
                const uint32_t idx = tb.terms_log < GKR_THREADS_LOG ? flat >> tb.terms_log : chunk >> whole;
                live = idx < tb.n_items;
                if (live) {
                    it = items[idx];
                    if (tb.terms_log < GKR_THREADS_LOG) item_sums_of(it, flat & ((1u << tb.terms_log) - 1), (size_t)1 << tb.terms_log, r, eq, lambda, s0, s2);
                    else item_sums_of(it, (size_t)(chunk & ((1u << whole) - 1)) * GKR_THREADS + tid, (size_t)GKR_THREADS << whole, r, eq, lambda, s0, s2);
                }
                add_to_group(sums, tb.terms_log < 5 ? 1 << tb.terms_log : 32, live, (uint32_t)it.slot, (uint32_t)(it.slot >> 32), alpha_pow, s0, s2);
            }
        } else {
            for (;;) {
                if (live) fix_mask(it, (int)term, r, host.masks + 16 * (size_t)(uint32_t)it.slot);
                chunk += tb.ctas;
                if (chunk >= tb.chunks) break;
                look_up();
            }
        }
        __syncthreads();
        if (!lead) {
            if (step && tid < 8 * GKR_GROUPS) {
                uint32_t* const h = &sums[tid >> 3][2 * (tid & 7)];
                const unsigned long long v = (unsigned long long)h[0] + ((unsigned long long)h[1] << 16);
                h[0] = h[1] = 0u;
                if (v) atomicAdd(acc.at(t, tid >> 3) + (tid & 7), v);
                __threadfence();
            }
            if (!step) __threadfence_system();
            __syncthreads();
            if (tid == 0) { __threadfence(); atomicAdd(&sync->count[t], 1u); }
            continue;
        }
        // CTA 0 from here on; its own sums stay where they are
        const bool ahead = t == look_from;  // (its own part of the layer is then read by others before there is a challenge)
        if (ahead && tid == 0) { __threadfence(); atomicAdd(&sync->count[t], 1u); }
        if (tb.ctas > 1) {
            if (tid == 0 && !wait_count(&sync->count[t], tb.ctas - (ahead ? 0u : 1u))) gave_up = true;
            __syncthreads();
            if (gave_up) return;
        }
        if (!step) break;
        auto challenge_drawn = [] { asm volatile("bar.sync 1, %0;" ::"n"(GKR_THREADS) : "memory"); };
        if (ahead && warp) {
            if (look_value(warp) >= 0 && look_helpers(sm, consts, tabs + n_rounds + 1, s, acc, sync, look_from, n_rounds, records)) gave_up = true;
            break;
        }
        if (warp == 0) {
            unsigned long long a[8];
            const bool theirs = tb.ctas > 1 && lane < acc.groups;
#pragma unroll
            for (int c = 0; c < 8; c++) a[c] = theirs ? __ldcg(acc.at(t, lane) + c) : 0ull;
#pragma unroll
            for (int c = 0; c < 8; c++) {
                a[c] += (unsigned long long)sums[lane][2 * c] + ((unsigned long long)sums[lane][2 * c + 1] << 16);
                sums[lane][2 * c] = sums[lane][2 * c + 1] = 0u;
            }
            if (ahead) {
                if (theirs) {
#pragma unroll
                    for (int c = 0; c < 8; c++) acc.at(t, lane)[c] = 0ull;
                    __threadfence();
                }
                look_lead(sm, consts, look_from, n_rounds, batch_coefficients(s, consts[t], s.corr[lane], acc_value(a), acc_value(a + 4)));
                break;
            }
            batch_step(sm, s, consts[t], acc_value(a), acc_value(a + 4), records + GKR_LAYER_OUT_WORDS * (size_t)t, challenge_drawn);
            if (theirs) {
#pragma unroll
                for (int c = 0; c < 8; c++) acc.at(t, lane)[c] = 0ull;  // for the round after the next: seen with the next challenge
            }
        } else {
            // Warp 1 sends the challenge. Its fence stands behind the barrier that put everybody's folded layers behind this point,
            // and takes as long as a third of a compression: warp 0 hashes meanwhile, and the CTA goes on with the next table
            // while it works out what the step after that needs.
            if (warp == 1 && tb.later > 1) __threadfence();
            challenge_drawn();
            if (warp == 1 && lane < 4 && tb.later > 1) *reinterpret_cast<volatile uint32_t*>(&sync->slot[t + 1][lane]) = sm.r.c[lane] | 0x80000000u;
        }
    }
    if (look_from >= 0 && !lead) {
        const GkrTable* const looks = tabs + n_rounds + 1;
        const qm31 half_lambda = qm31_mul_m31(lambda, 1u << 30);
        const uint32_t block = blockIdx.x - 1;
        for (int t = look_from; t < n_rounds; t++) {
            const GkrTable tb = looks[t];
            if (block >= tb.ctas) {
                if (block >= tb.later) return;
                continue;
            }
            const GkrBatchItem* const items = items_base + tb.first;
            const int lanes_log = tb.form == 3 ? 3 : 2;  // lanes a term (form 3), an item (4)
            uint32_t chunk = block, term = 0;
            GkrBatchItem it{};
            bool live = false;
            qm31 ea = qm31_zero();
            auto look_up = [&]() {
                const uint32_t at = ((chunk << tb.run_log) + tid) >> lanes_log, item = at >> tb.terms_log;
                term = at & ((1u << tb.terms_log) - 1);
                live = item < tb.n_items && !(tid >> tb.run_log);
                if (live) it = items[item];
                if (tb.form == 3 && live) ea = qmul(eq_at(term), ldqb(alpha_pow, (uint32_t)it.slot));
            };
            look_up();
            entry v0{qm31_zero(), qm31_zero()}, v1 = v0;
            auto load = [&] {
                if (!live || !look_live(it)) return;
                const size_t e = look_entry(term, tb.terms_log);
                v0 = load_entry(it, e);
                if (it.mode == LOOK_FIX) v1 = load_entry(it, e + ((size_t)8 << tb.terms_log));
            };
            // The layer is whole when the pass before is counted, some 2,000 cycles before the challenge: the first piece's entries are on their way then.
            const bool early = tb.form == 3 && t > look_from;
            if (early) {
                if (tid == 0 && !wait_count(&sync->look_count[t - 1], looks[t - 1].ctas)) gave_up = true;
                __syncthreads();
                load();
            }
            if (t > look_from) {
                if (tid < 4) {
                    uint32_t w = ld_acquire(&sync->slot[t][tid]);
                    for (uint32_t spin = 0; !(w >> 31) && spin < SPIN_LIMIT; spin++) w = ld_acquire(&sync->slot[t][tid]);
                    if (!(w >> 31)) gave_up = true;
                    r_sh.c[tid] = w & 0x7fffffffu;
                }
            } else if (t > 0 && tid == 0 && !wait_count(&sync->count[t], tabs[t].ctas)) {  // the layer as the table before left it
                gave_up = true;
            }
            __syncthreads();
            if (gave_up) return;
            const qm31 r = r_sh;
            for (;;) {
                if (tid >> tb.run_log) {  // (whole warps)
                } else if (tb.form == 3) {
                    if (!early || chunk != block) load();
                    look_term(sums, it, live, term, tb.terms_log, v0, v1, r, half_lambda, ea);
                } else if (live) fix_entry(it, tid & 3, load_entry(it, tid & 3), load_entry(it, (tid & 3) + 4), r);
                chunk += tb.ctas;
                if (chunk >= tb.chunks) break;
                look_up();
            }
            __syncthreads();
            if (tb.form == 3)
                for (int i = tid; i < ACC_WORDS * acc.groups; i += GKR_THREADS) {
                    uint32_t* const h = &sums[0][0] + 2 * i;
                    const unsigned long long v = (unsigned long long)h[0] + ((unsigned long long)h[1] << 16);
                    h[0] = h[1] = 0u;
                    if (v) atomicAdd(acc.at(t + 1, 0) + i, v);
                }
            __syncthreads();
            if (tid == 0) { __threadfence(); atomicAdd(&sync->look_count[t], 1u); }
        }
        return;
    }
    if (!lead) return;
    __syncthreads();
    if (gave_up) return;
    // What the rounds ahead leave, four entries an oracle, is fixed here: the challenge is, and it goes to the host with the rest. (As one more pass of the
    // CTAs, each with its fence for the host, the masks took 9,700 cycles of a layer, and the channel by way of memory 1,400.)
    if (look_from >= 0) {
        const GkrTable& tb = tabs[n_rounds];
        const qm31 r = sm.look_r[(n_rounds - 1) & 1];
        for (uint32_t i = tid; i < 2 * tb.n_items; i += GKR_THREADS) {
            const GkrBatchItem it = items_base[tb.first + (i >> 1)];
            fix_mask(it, (int)(i & 1), r, host.masks + 16 * (size_t)(uint32_t)it.slot);
        }
    }
    if (warp == 0) batch_step_close(sm, host.channel, lane);
    layer_out_words(host, records, n_rounds, tid, GKR_THREADS);
    __threadfence_system();
    __syncthreads();
    if (tid == 0) *host.flag = host.id;
}

// The step after table t < n_rounds by itself, one warp; after the last table, what goes to the host.
__global__ void __launch_bounds__(32) gkr_batch_step_kernel(GkrStepState* st, GkrAcc acc, GkrSync* sync, const uint32_t* __restrict__ open, uint32_t* records, int t, int n_rounds,
                                                            GkrLayerOut host) {
    __shared__ GkrStepSm sm;
    const int lane = threadIdx.x;
    const GkrStepConst* const rc = reinterpret_cast<const GkrStepConst*>(open + OPEN_CONSTS);
    if (t == 0) {
        for (int i = lane; i < (int)(sizeof(*st) / 4); i += 32) reinterpret_cast<uint32_t*>(st)[i] = open_state_word(open, i);
        __syncwarp();
    }
    if (t == n_rounds) {
        layer_out_words(host, records, n_rounds, lane, 32);
        if (lane < 12) host.channel[lane] = reinterpret_cast<const uint32_t*>(st)[lane];
        __threadfence_system();
        __syncwarp();
        if (lane == 0) *host.flag = host.id;
        return;
    }
    unsigned long long a[8];
#pragma unroll
    for (int c = 0; c < 8; c++) {
        a[c] = lane < acc.groups ? acc.at(t, lane)[c] : 0ull;
        if (lane < acc.groups) acc.at(t, lane)[c] = 0ull;
    }
    batch_step_open(sm, *st, lane);
    batch_step(sm, *st, rc[t], acc_value(a), acc_value(a + 4), records + GKR_LAYER_OUT_WORDS * (size_t)t, [] {});
    if (lane < 4) sync->slot[t + 1][lane] = sm.r.c[lane] | 0x80000000u;
    batch_step_close(sm, reinterpret_cast<uint32_t*>(st), lane);
}

// ---- a single round with its results to the host
//
// The CTA that completes an item reports it. When every item of the launch has reported, the
// round's sequence number is written after the results. `results` and `flag` are then page-locked host memory the device
// writes directly, so the host sees a round's results a PCIe write after the last CTA ends, without a copy and a stream
// synchronisation of its own (a round of a small batch is a 5-10 us kernel; the copy and the wake-up cost as much again).
__device__ __forceinline__ void item_done(unsigned int* done, int n_items, volatile unsigned int* flag, unsigned int round_id) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence_system();
        if (atomicAdd(done, 1u) == (unsigned int)n_items - 1u) {
            *done = 0u;  // every item has counted: ready for the next launch
            __threadfence_system();
            *flag = round_id;
        }
    }
}

__global__ void __launch_bounds__(256) gkr_batch_round_kernel(const GkrBatchItem* __restrict__ items, int n_items, qm31 r,
                                                              const uint32_t* __restrict__ eq, qm31 lambda, uint32_t* __restrict__ partials,
                                                              unsigned int* __restrict__ tickets, uint32_t* __restrict__ results,
                                                              unsigned int* __restrict__ done, volatile unsigned int* flag, unsigned int round_id) {
    const int idx = find_item(items, n_items, blockIdx.x);
    const GkrBatchItem it = items[idx];
    const uint32_t bx = blockIdx.x - it.first_block;
    uint32_t* res = results + (size_t)GKR_BATCH_RESULT_WORDS * (size_t)idx;
    if (it.mode == 2) {
        if (threadIdx.x < 2) fix_mask(it, threadIdx.x, r, res + 8);  // four entries -> two; one thread per entry
        item_done(done, n_items, flag, round_id);
        return;
    }
    qm31 s0 = qm31_zero(), s2 = qm31_zero();
    item_sums_of(it, (size_t)bx * blockDim.x + threadIdx.x, (size_t)it.blocks * blockDim.x, r, eq, lambda, s0, s2);
    __shared__ uint32_t sh[8][8];
    __shared__ bool is_last;
    s0 = warp_sum_m(s0);
    s2 = warp_sum_m(s2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { stqb(sh[warp], 0, s0); stqb(sh[warp], 1, s2); }
    __syncthreads();
    uint32_t* part = partials + 8 * (size_t)it.first_block;
    if (threadIdx.x < 8) {
        uint32_t acc = 0;
        for (int w = 0; w < 8; w++) acc = m31_add(acc, sh[w][threadIdx.x]);
        if (it.blocks == 1) res[threadIdx.x] = acc;
        else { part[8 * bx + threadIdx.x] = acc; __threadfence(); }
    }
    if (it.blocks == 1) {
        item_done(done, n_items, flag, round_id);
        return;
    }
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(tickets + idx, 1u) == it.blocks - 1;
    __syncthreads();
    if (is_last) {
        __threadfence();
        if (threadIdx.x < 8) {
            uint32_t acc = 0;
            for (uint32_t b = 0; b < it.blocks; b++) acc = m31_add(acc, __ldcg(&part[8 * b + threadIdx.x]));
            res[threadIdx.x] = acc;
        }
        if (threadIdx.x == 0) tickets[idx] = 0u;
        item_done(done, n_items, flag, round_id);
    }
}

// The towers of all instances, ten levels a launch (gkr_tower.cuh); an item's layers lie one after the other from num_out / den_out
// on. A launch per level and its table cost some 15 us of host time each, for levels of a microsecond or two: 582 instances of up
// to 2^19 entries took 19 launches, now two.
__global__ void __launch_bounds__(TOWER_THREADS) gkr_batch_tower_kernel(const GkrBatchItem* __restrict__ items, int n_items, int level0, uint32_t* __restrict__ tops) {
    __shared__ uint4 sd[512], sn[512];
    const GkrBatchItem it = items[find_item(items, n_items, blockIdx.x)];
    const int log = 63 - __clzll(it.n), left = log - level0, cta_log = left < TOWER_LEVELS ? left : TOWER_LEVELS;
    auto words_before = [&](int level) { return 4 * (it.n - (it.n >> (level - 1))); };
    auto outs = [&](int l, uint32_t*& num, uint32_t*& den) {
        const size_t at = words_before(level0 + l + 1);
        num = it.num_out + at;
        den = it.den_out + at;
    };
    uint32_t* const top = left == cta_log ? tops + GKR_TOP_WORDS * it.slot : nullptr;
    const uint32_t bx = blockIdx.x - it.first_block;
    const uint32_t *num = it.num, *den = it.den;
    if (level0) {
        num = it.num_out + words_before(level0);
        den = it.den_out + words_before(level0);
    }
    switch (level0 == 0 || it.kind == ZKB_GKR_GRAND_PRODUCT ? it.kind : ZKB_GKR_LOGUP_GENERIC) {
        case ZKB_GKR_GRAND_PRODUCT: tower_cta<ZKB_GKR_GRAND_PRODUCT>(num, den, bx, cta_log, cta_log, sd, sn, outs, top); break;
        case ZKB_GKR_LOGUP_GENERIC: tower_cta<ZKB_GKR_LOGUP_GENERIC>(num, den, bx, cta_log, cta_log, sd, sn, outs, top); break;
        case ZKB_GKR_LOGUP_MULTIPLICITIES: tower_cta<ZKB_GKR_LOGUP_MULTIPLICITIES>(num, den, bx, cta_log, cta_log, sd, sn, outs, top); break;
        default: tower_cta<ZKB_GKR_LOGUP_SINGLES>(num, den, bx, cta_log, cta_log, sd, sn, outs, top); break;
    }
}

// Splits the flat grid over the items (first_block, blocks) by the work each has; returns the number of CTAs.
uint32_t plan_blocks(GkrBatchItem* items, int n_items) {
    uint32_t total = 0;
    for (int k = 0; k < n_items; k++) {
        GkrBatchItem& it = items[k];
        const size_t units = it.mode == 0 ? it.n / 4 : it.mode == 1 ? it.n / 8 : 1;
        const size_t blocks = std::min<size_t>(std::max<size_t>((units + 255) / 256, 1), 148u * 4u);
        it.first_block = total;
        it.blocks = (uint32_t)blocks;
        total += it.blocks;
    }
    return total;
}

int stage_items(zkb_ctx* ctx, const GkrBatchItem* items, int n_items, const GkrBatchItem** d_items) {
    static_assert(sizeof(GkrBatchItem) % sizeof(void*) == 0, "items are staged through the pointer ring");
    void** d = nullptr;
    int rc = stage_ptrs(ctx, reinterpret_cast<const void* const*>(items), (int)(n_items * (sizeof(GkrBatchItem) / sizeof(void*))), &d);
    if (rc) return rc;
    *d_items = reinterpret_cast<const GkrBatchItem*>(d);
    return ZKB_OK;
}

}  // namespace

// Page-locked words: the per-item results of a round, then the sequence number of the last completed round. (A layer enqueued at once
// lands its records there: never more words, with at most a mask per oracle and 24 words a round.)
constexpr size_t H_BATCH_FLAG = GKR_BATCH_RESULT_WORDS * GKR_BATCH_MAX_ITEMS + 4096;
constexpr size_t H_BATCH_WORDS = H_BATCH_FLAG + 4;

// The description of a layer is built in a buffer the calling thread keeps (a batch of hundreds of instances describes 100-500 KB a layer).
static std::vector<uint32_t>& ctx_blob() {
    thread_local std::vector<uint32_t> blob;
    return blob;
}

static int batch_buffers(zkb_ctx* ctx) {
    if (ctx->batch_tickets) return ZKB_OK;
    // tickets per item, then the launch's count of completed items
    ZKB_CUDA(ctx, cudaMalloc(&ctx->batch_tickets, (GKR_BATCH_MAX_ITEMS + 1) * sizeof(unsigned int)));
    ZKB_CUDA(ctx, cudaMemsetAsync(ctx->batch_tickets, 0, (GKR_BATCH_MAX_ITEMS + 1) * sizeof(unsigned int), ctx->stream));
    int sms = 0, per_sm = 0;
    ZKB_CUDA(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
    ZKB_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gkr_batch_layer_kernel, GKR_THREADS, 0));
    ctx->batch_grid = sms * std::min(per_sm, 1);
    ZKB_CUDA(ctx, cudaMallocHost(&ctx->h_batch, H_BATCH_WORDS * 4));
    ctx->h_batch[H_BATCH_FLAG] = 0;
    ctx->batch_round = 0;
    return ZKB_OK;
}

// Waits for a launch to report `id`: a bounded spin on the host (2 10^7 polls, a second at most), then the stream.
static cudaError_t batch_wait(zkb_ctx* ctx, unsigned int id) {
    volatile unsigned int* flag = reinterpret_cast<volatile unsigned int*>(ctx->h_batch + H_BATCH_FLAG);
    if (!ctx->prof_on)
        for (long spin = 0; spin < 20000000L && *flag != id; spin++) {
#if defined(__x86_64__)
            __builtin_ia32_pause();
#endif
        }
    cudaError_t e = cudaSuccess;
    if (*flag != id) e = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess && *flag != id) e = cudaErrorUnknown;  // the launch ended without completing every item
    std::atomic_thread_fence(std::memory_order_acquire);
    return e;
}

int gkr_batch_towers(zkb_ctx* ctx, GkrBatchItem* items, int n_items, uint32_t* h_tops) {
    if (n_items <= 0) return ZKB_OK;
    if ((size_t)n_items > GKR_BATCH_MAX_ITEMS) return set_error(ctx, ZKB_EINVAL, "gkr batch: more than %d instances", (int)GKR_BATCH_MAX_ITEMS);
    DeviceGuard g(ctx);
    if (int rc = batch_buffers(ctx)) return rc;
    uint32_t* d_tops = nullptr;
    if (int rc = zkb_malloc(ctx, GKR_TOP_WORDS * 4 * (size_t)n_items, (void**)&d_tops)) return rc;
    for (int k = 0; k < n_items; k++) items[k].slot = (unsigned long long)k;
    cudaError_t e = cudaSuccess;
    int rc = ZKB_OK;
    std::vector<GkrBatchItem> live;
    for (int level0 = 0; rc == ZKB_OK && e == cudaSuccess; level0 += TOWER_LEVELS) {
        live.clear();
        uint32_t total = 0;
        for (int k = 0; k < n_items; k++) {
            if ((items[k].n >> level0) < 2) continue;
            live.push_back(items[k]);
            live.back().first_block = total;
            total += (uint32_t)std::max<unsigned long long>(items[k].n >> (level0 + TOWER_LEVELS), 1);
        }
        if (live.empty()) break;
        const GkrBatchItem* d_items;
        rc = stage_items(ctx, live.data(), (int)live.size(), &d_items);
        if (rc) break;
        ProfScope prof(ctx, "gkr_batch_tower_kernel");
        gkr_batch_tower_kernel<<<total, TOWER_THREADS, 0, ctx->stream>>>(d_items, (int)live.size(), level0, d_tops);
        e = cudaGetLastError();
    }
    const size_t bytes = GKR_TOP_WORDS * 4 * (size_t)n_items;
    if (rc == ZKB_OK && e == cudaSuccess) e = cudaMemcpyAsync(ctx->h_batch, d_tops, bytes, cudaMemcpyDeviceToHost, ctx->stream);
    if (rc == ZKB_OK && e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    zkb_free(ctx, d_tops);
    if (rc) return rc;
    if (e != cudaSuccess) return set_error(ctx, ZKB_ECUDA, "gkr batch towers: %s", cudaGetErrorString(e));
    memcpy(h_tops, ctx->h_batch, bytes);
    return ZKB_OK;
}

int gkr_batch_round(zkb_ctx* ctx, GkrBatchItem* items, int n_items, const uint32_t h_r[4], const uint32_t* eq_evals, const uint32_t h_lambda[4],
                    uint32_t* h_results) {
    if (n_items <= 0) return ZKB_OK;
    if ((size_t)n_items > GKR_BATCH_MAX_ITEMS) return set_error(ctx, ZKB_EINVAL, "gkr batch: more than %d instances", (int)GKR_BATCH_MAX_ITEMS);
    DeviceGuard g(ctx);
    uint32_t total = plan_blocks(items, n_items);
    if (int rc = batch_buffers(ctx)) return rc;
    // The device writes the results straight into the page-locked host buffer (unified addressing: the host pointer is valid
    // on the device). scratch: [(unused) | partials]
    uint32_t* results = ctx->h_batch;
    unsigned int* tickets = ctx->batch_tickets;
    uint32_t* partials = ctx->scratch + (size_t)(GKR_BATCH_RESULT_WORDS + 1) * GKR_BATCH_MAX_ITEMS;
    if ((size_t)(GKR_BATCH_RESULT_WORDS + 1) * GKR_BATCH_MAX_ITEMS + 8 * (size_t)total > ctx->scratch_words)
        return set_error(ctx, ZKB_EINVAL, "gkr batch: %u CTAs exceed the scratch buffer", total);
    const GkrBatchItem* d_items;
    int rc = stage_items(ctx, items, n_items, &d_items);
    if (rc) return rc;
    volatile unsigned int* flag = reinterpret_cast<volatile unsigned int*>(ctx->h_batch + H_BATCH_FLAG);
    const unsigned int round_id = ++ctx->batch_round;
    qm31 r{{h_r[0], h_r[1], h_r[2], h_r[3]}}, lam{{h_lambda[0], h_lambda[1], h_lambda[2], h_lambda[3]}};
    {
        ProfScope prof(ctx, "gkr_batch_round_kernel");
        gkr_batch_round_kernel<<<total, 256, 0, ctx->stream>>>(d_items, n_items, r, eq_evals, lam, partials, tickets, results,
                                                               ctx->batch_tickets + GKR_BATCH_MAX_ITEMS, flag, round_id);
    }
    const size_t bytes = (size_t)n_items * GKR_BATCH_RESULT_WORDS * 4;
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = batch_wait(ctx, round_id);
    if (e != cudaSuccess) {
        // a launch that did not run to its end may have left tickets counted up
        cudaMemsetAsync(ctx->batch_tickets, 0, (GKR_BATCH_MAX_ITEMS + 1) * sizeof(unsigned int), ctx->stream);
        return set_error(ctx, ZKB_ECUDA, "gkr batch round: %s", cudaGetErrorString(e));
    }
    memcpy(h_results, ctx->h_batch, bytes);
    return ZKB_OK;
}

// What is staged with a layer's items, in words: room for the transcript's state, the CTAs' meeting place (zero), the tables, room for the rounds' records (every
// part a multiple of four words).
struct LayerBlob { size_t acc, sync, tables, records, words; };
static LayerBlob layer_blob(const GkrLayerPlan& plan) {
    LayerBlob o;
    o.acc = sizeof(GkrStepState) / 4;
    o.sync = o.acc + 2 * 2 * ACC_WORDS * (size_t)plan.n_rounds;
    o.tables = o.sync + sizeof(GkrSync) / 4;
    o.records = o.tables + plan.tables.size();
    o.words = o.records + GKR_LAYER_OUT_WORDS * (size_t)plan.n_rounds;
    return o;
}
static size_t open_words(const GkrLayerPlan& plan) { return open_alpha(plan.n_rounds) + 4 * plan.n_vars.size(); }

// The rounds that are taken ahead of the transcript (gkr_look_from). Their tables go behind the others, and the items that are used into look_items.
static GkrTable* tables_of(GkrLayerPlan& plan) { return reinterpret_cast<GkrTable*>(plan.tables.data()); }
static void plan_look(GkrLayerPlan& plan, uint32_t grid) {
    const int n = plan.n_rounds;
    size_t terms[GKR_LAYER_MAX_ROUNDS];
    for (int j = 0; j < n; j++) terms[j] = (size_t)tables_of(plan)[j].n_items << tables_of(plan)[j].terms_log;
    const int from = plan.look_from = plan.launches ? -1 : gkr_look_from(terms, n, grid);
    if (from < 0) return;
    plan.tables.resize((sizeof(GkrTable) / 4) * (2 * (size_t)n + 1), 0u);
    GkrTable* const tables = tables_of(plan);
    std::vector<GkrBatchItem>& out = plan.look_items;
    auto table = [&](int j) { return std::make_pair(plan.items.begin() + plan.table_at[j], plan.items.begin() + plan.table_at[j + 1]); };
    out.assign(plan.items.begin(), table(from).second);
    auto add = [&](const GkrBatchItem& it, uint32_t mode) {
        out.push_back(it);
        out.back().mode = mode;
    };
    for (int j = from; j <= n; j++) {
        GkrTable& tb = tables[j < n ? n + 1 + j : n];
        tb.first = (uint32_t)out.size();
        for (auto it = table(j).first; it != table(j).second; ++it) {
            if (j == n) { add(*it, it->mode); continue; }
            if (j == n - 1) {  // eight entries to four; those that enter now are folded with the last challenge
                if (it->mode == 1) add(*it, LOOK_FIX);
                continue;
            }
            if (it->mode == 1 && j > from) { add(*it, LOOK_FIX); continue; }
            add(*it, LOOK_AS_IS);
            GkrBatchItem& as_is = out.back();
            if (it->mode == 1) {  // as table `from` has left it
                as_is.den = as_is.den_out;
                as_is.num = as_is.num_out;
                if (as_is.kind == ZKB_GKR_LOGUP_MULTIPLICITIES) as_is.kind = ZKB_GKR_LOGUP_GENERIC;
            }
        }
        if (j < n - 1)
            for (auto it = table(j + 1).first; it != table(j + 1).second; ++it)
                if (it->mode == 0) add(*it, LOOK_ENTERS);
        tb.n_items = (uint32_t)(out.size() - tb.first);
        tb.terms_log = j == n ? 1 : j == n - 1 ? 0 : n - j - 2;
        tb.form = j == n ? 2 : j == n - 1 ? 4 : 3;
        const size_t lanes = ((size_t)tb.n_items << tb.terms_log) << (tb.form == 3 ? 3 : tb.form == 4 ? 2 : 0);
        // as few warps a CTA as there are CTAs for: a pass of a warp a scheduler takes 2,300 cycles, of four 5,100
        tb.run_log = LOOK_MIN_LOG;
        while (tb.run_log < GKR_THREADS_LOG && ((lanes + (1u << tb.run_log) - 1) >> tb.run_log) > grid - 1) tb.run_log++;
        tb.chunks = (uint32_t)((lanes + (1u << tb.run_log) - 1) >> tb.run_log);
        tb.ctas = j == n ? 0u : std::min(tb.chunks, grid - 1);  // (CTA 0 has the masks)
    }
    uint32_t later = 0;
    for (int j = n; j >= from; j--) {
        GkrTable& tb = tables[j < n ? n + 1 + j : n];
        tb.later = later;
        later = std::max(later, tb.ctas);
    }
    later++;  // CTA 0 takes none of them
    for (int j = from; j >= 0; j--) {
        tables[j].later = later;
        later = std::max(later, tables[j].ctas);
    }
}

int gkr_batch_plan(zkb_ctx* ctx, GkrLayerPlan& plan) {
    const int n_rounds = plan.n_rounds;
    if (plan.n_vars.size() > GKR_BATCH_MAX_ITEMS) return set_error(ctx, ZKB_EINVAL, "gkr batch: more than %d instances", (int)GKR_BATCH_MAX_ITEMS);
    if (n_rounds > GKR_LAYER_MAX_ROUNDS) return set_error(ctx, ZKB_EINVAL, "gkr batch: %d rounds in a layer", n_rounds);
    DeviceGuard g(ctx);
    if (int rc = batch_buffers(ctx)) return rc;
    const uint32_t grid = (uint32_t)ctx->batch_grid;
    plan.tables.assign((sizeof(GkrTable) / 4) * ((size_t)n_rounds + 1), 0u);
    GkrTable* const tables = reinterpret_cast<GkrTable*>(plan.tables.data());
    uint32_t later = 0;
    for (int j = n_rounds; j >= 0; j--) {
        GkrBatchItem* const t = plan.items.data() + plan.table_at[j];
        const int nt = (int)(plan.table_at[j + 1] - plan.table_at[j]);
        if (!nt) return set_error(ctx, ZKB_EINVAL, "gkr batch: round %d of the layer has no work", j);
        for (int q = 0; q < nt; q++)
            t[q].slot = (t[q].slot & 0xffffffffull) | (unsigned long long)(n_rounds - (int)plan.n_vars[t[q].slot & 0xffffffffull]) << 32;
        GkrTable& tb = tables[j];
        tb.first = (uint32_t)plan.table_at[j];
        tb.n_items = (uint32_t)nt;
        // n_rounds - j variables are left: 2^(that - 1) terms an item; at the end two entries of a mask each
        tb.terms_log = j < n_rounds ? n_rounds - j - 1 : 1;
        const size_t terms = (size_t)nt << tb.terms_log;
        tb.form = j == n_rounds ? 2 : gkr_four_lanes(terms, grid) ? 1 : 0;
        // Whole items of 2^GKR_THREADS_LOG terms and more: a thread takes up to eight terms for one reduction, as long as four pieces per CTA remain.
        tb.run_log = 0;
        if (tb.form == 0)
            while (tb.run_log < 3 && tb.terms_log - GKR_THREADS_LOG > tb.run_log && (terms >> (GKR_THREADS_LOG + tb.run_log + 1)) >= 4 * (size_t)grid) tb.run_log++;
        if (tb.form) {
            const size_t lanes = tb.form == 1 ? 4 * terms : terms;
            for (tb.run_log = LOOK_MIN_LOG; tb.run_log < GKR_THREADS_LOG && ((lanes + (1u << tb.run_log) - 1) >> tb.run_log) > grid;) tb.run_log++;
        }
        const size_t chunks = tb.form == 0 && tb.terms_log >= GKR_THREADS_LOG ? terms >> (GKR_THREADS_LOG + tb.run_log) : tb.form == 0 ? (terms + GKR_THREADS - 1) / GKR_THREADS : ((tb.form == 1 ? 4 * terms : terms) + (1u << tb.run_log) - 1) >> tb.run_log;
        tb.chunks = (uint32_t)chunks;
        // (sending the sums and the challenge round costs less than a second piece in CTA 0: 6,400 cycles against 8,500)
        tb.ctas = (uint32_t)std::min<size_t>(chunks, grid);
        tb.later = later;
        later = std::max(later, tb.ctas);
    }
    plan_look(plan, grid);
    // Rounds that take four and eight lanes a term can work eq out: a term a thread would take two products more for each of its six.
    plan.needs_eq = plan.look_from != 0 || tables_of(plan)[0].terms_log > GKR_EQ_BITS;
    const std::vector<GkrBatchItem>& items = plan.look_from >= 0 ? plan.look_items : plan.items;
    // What the launch stages later must not come to lie over this: room for both.
    const size_t item_words = items.size() * (sizeof(GkrBatchItem) / 4);
    const LayerBlob at = layer_blob(plan);
    if (int rc = stage_reserve(ctx, blob_slots(4 * (item_words + at.words)) + blob_slots(4 * open_words(plan)))) return rc;
    std::vector<uint32_t>& blob = ctx_blob();
    blob.assign(item_words + at.words, 0u);
    memcpy(blob.data(), items.data(), 4 * item_words);
    memcpy(&blob[item_words + at.tables], plan.tables.data(), 4 * plan.tables.size());
    void* d = nullptr;
    if (int rc = stage_blob(ctx, blob.data(), 4 * blob.size(), &d)) return rc;
    plan.d_items = static_cast<const GkrBatchItem*>(d);
    plan.d_blob = static_cast<uint32_t*>(d) + item_words;
    return ZKB_OK;
}

int gkr_batch_layer_begin(zkb_ctx* ctx, GkrLayerPlan& plan, const uint32_t* alpha_pow, const uint32_t* claims, const GkrRoundConst* rounds,
                          const uint32_t* eq_evals, const uint32_t h_lambda[4], const uint32_t chan[9]) {
    ZKB_CHECK_ARG(ctx, eq_evals || !plan.needs_eq);
    DeviceGuard g(ctx);
    if (int rc = batch_buffers(ctx)) return rc;
    const size_t K = plan.n_vars.size();
    const int n_rounds = plan.n_rounds;
    const LayerBlob at = layer_blob(plan);
    const bool carries = !plan.launches && open_words(plan) <= OPEN_WORDS;
    GkrLayerOpen carried;
    std::vector<uint32_t>& blob = ctx_blob();
    if (!carries) blob.assign(open_words(plan), 0u);
    uint32_t* const open = carries ? carried.words : blob.data();
    auto q4 = [](const uint32_t* w) { return qm31{{w[0], w[1], w[2], w[3]}}; };
    // The oracles' claims by the round they enter in (group; those without variables never do), each times alpha^k. The claims come
    // scaled by 2^(rounds they wait), and a waiting oracle's claim halves every round (sumcheck.rs:115-125).
    qm31 entering[GKR_LAYER_MAX_ROUNDS + 1];
    for (auto& v : entering) v = qm31_zero();
    for (size_t k = 0; k < K; k++) {
        qm31& v = entering[n_rounds - (int)plan.n_vars[k]];
        v = qm31_add(v, qm31_mul(q4(alpha_pow + 4 * k), q4(claims + 4 * k)));
    }
    memcpy(open, chan, 36);
    memcpy(open + OPEN_CLAIM, entering[0].c, 16);
    memcpy(open + open_alpha(n_rounds), alpha_pow, 16 * K);
    GkrStepConst* const consts = reinterpret_cast<GkrStepConst*>(open + OPEN_CONSTS);
    qm31 waiting = qm31_zero();
    for (int j = n_rounds; j-- > 0;) {
        waiting = qm31_add(waiting, entering[j + 1]);  // all that enter after round j
        GkrStepConst& c = consts[j];
        const GkrRoundConst& rc = rounds[j];
        const uint32_t half_pow = j + 1 < 31 ? 1u << (31 - (j + 1)) : 1u;  // 2^-(j + 1), as 2^31 = 1
        for (int t = 0; t < 4; t++) {
            c.A[t] = qm31_mul(q4(rc.e0a), qm31_sub(q4(rc.L[0][t]), q4(rc.L[1][t])));
            c.B[t] = qm31_mul(q4(rc.e2a), q4(rc.L[2][t]));
            c.L1[t] = q4(rc.L[1][t]);
        }
        c.y = q4(rc.y);
        c.waiting = qm31_mul_m31(waiting, half_pow);
        c.entering = j + 1 < n_rounds ? qm31_mul_m31(entering[j + 1], half_pow) : qm31_zero();
        c.round = (uint32_t)j;
    }
    uint32_t* const d_blob = plan.d_blob;
    const uint32_t* d_open = nullptr;
    auto copy_open = [&]() -> int {
        void* d = nullptr;
        const int rc = stage_blob(ctx, open, 4 * open_words(plan), &d);
        d_open = static_cast<const uint32_t*>(d);
        return rc;
    };
    if (!carries) if (int rc = copy_open()) return rc;
    GkrStepState* d_state = reinterpret_cast<GkrStepState*>(d_blob);
    const qm31 lam = q4(h_lambda);
    GkrLayerOut host;
    host.records = ctx->h_batch;
    host.channel = host.records + GKR_LAYER_OUT_WORDS * (size_t)n_rounds;
    host.masks = host.channel + 12;
    host.flag = reinterpret_cast<volatile unsigned int*>(ctx->h_batch + H_BATCH_FLAG);
    host.id = ++ctx->batch_round;
    const GkrTable* const h_tables = reinterpret_cast<const GkrTable*>(plan.tables.data());
    const GkrTable* const d_tables = reinterpret_cast<const GkrTable*>(d_blob + at.tables);
    uint32_t* const d_records = d_blob + at.records;
    GkrSync* const d_sync = reinterpret_cast<GkrSync*>(d_blob + at.sync);
    const GkrAcc acc{reinterpret_cast<unsigned long long*>(d_blob + at.acc), n_rounds};
    cudaError_t e = cudaErrorCooperativeLaunchTooLarge;
    if (!plan.launches && !plan.refused) {
        ProfScope prof(ctx, "gkr_batch_layer_kernel");
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;  // every CTA is resident, or the launch fails
        attr[0].val.cooperative = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(std::max(h_tables[0].ctas, h_tables[0].later));
        cfg.blockDim = dim3(GKR_THREADS);
        cfg.stream = ctx->stream;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, gkr_batch_layer_kernel, plan.d_items, d_tables, 0, plan.look_from >= 0 ? plan.look_from + 1 : n_rounds + 1, plan.needs_eq ? eq_evals : nullptr, lam, carried, d_open, d_state, acc,
                               d_sync, 1, plan.look_from, d_records, n_rounds, host);
    }
    // Asked for, or the CTAs are not all resident at once (a share of the GPU's SMs): a launch per table and one per step, where nobody waits.
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        (void)cudaGetLastError();
        if (plan.look_from >= 0) {  // other tables and items then
            plan.launches = true;
            if (int rc = gkr_batch_plan(ctx, plan)) return rc;
            return GKR_BATCH_AGAIN;
        }
        if (!d_open) if (int rc = copy_open()) return rc;
        e = cudaSuccess;
        for (int t = 0; t <= n_rounds && e == cudaSuccess; t++) {
            {
                ProfScope prof(ctx, "gkr_batch_layer_kernel");
                gkr_batch_layer_kernel<<<h_tables[t].ctas, GKR_THREADS, 0, ctx->stream>>>(plan.d_items, d_tables, t, t + 1, eq_evals, lam, carried, d_open, d_state, acc, d_sync, 0,
                                                                                          -1, d_records, n_rounds, host);
            }
            {
                ProfScope prof(ctx, "gkr_batch_step_kernel");
                gkr_batch_step_kernel<<<1, 32, 0, ctx->stream>>>(d_state, acc, d_sync, d_open, d_records, t, n_rounds, host);
            }
            e = cudaGetLastError();
        }
    }
    if (e != cudaSuccess) return set_error(ctx, ZKB_ECUDA, "gkr batch layer: %s", cudaGetErrorString(e));
    return ZKB_OK;
}

int gkr_batch_layer_end(zkb_ctx* ctx, const GkrLayerPlan& plan, GkrLayerResult& res) {
    DeviceGuard g(ctx);
    const cudaError_t e = batch_wait(ctx, ctx->batch_round);
    if (e != cudaSuccess) return set_error(ctx, ZKB_ECUDA, "gkr batch layer: %s", cudaGetErrorString(e));
    res.records = ctx->h_batch;
    res.channel = res.records + GKR_LAYER_OUT_WORDS * (size_t)plan.n_rounds;
    res.masks = res.channel + 12;
    return ZKB_OK;
}

}  // namespace zk
