// A layer's sum-check, or one round of it, for a GKR batch of any number of instances in one launch (gkr_batch.cu); internal to the library.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

struct zkb_ctx;

namespace zk {

// What to do for one instance in a batched launch. kind: ZKB_GKR_* of the INPUT arrays; n: entries of the input layer.
// mode 0: round sums of the layer; 1: fix the first variable into num_out/den_out (n >= 8) and round sums of the result;
// 2: fix the first variable of a 4-entry layer, the result also copied to the result words.
// first_block / blocks are filled by the launcher.
struct GkrBatchItem {
    const uint32_t* num;
    const uint32_t* den;
    uint32_t* num_out;
    uint32_t* den_out;
    unsigned long long n;
    uint32_t kind, mode, first_block, blocks;
    unsigned long long slot;  // gkr_batch_layer: the oracle the item belongs to (its results go to that oracle's record)
};
static_assert(sizeof(GkrBatchItem) == 64, "GkrBatchItem layout");

constexpr size_t GKR_BATCH_MAX_ITEMS = 8192;
// Per item: [0,8) the two sums (t = 0, t = 2); mode 2 only: [8,16) the two fixed denominators, [16,24) the two fixed numerators.
constexpr size_t GKR_BATCH_RESULT_WORDS = 24;

// The layers above every item's input (num, den, n >= 2 entries, kind), one after the other from den_out and (but for a grand
// product) num_out on, n - 1 entries each: level 1 first. h_tops: per item the output's denominator and numerator, then the two
// denominators and the two numerators of the layer below it (numerators of an input without its own: undefined).
constexpr size_t GKR_TOP_WORDS = 24;
int gkr_batch_towers(zkb_ctx* ctx, GkrBatchItem* items, int n_items, uint32_t* h_tops);
// One round for every item with the transcript on the host: one launch that writes n_items * GKR_BATCH_RESULT_WORDS words and
// a completion word into page-locked host memory; returns when the host has seen the completion word (h_results filled).
int gkr_batch_round(zkb_ctx* ctx, GkrBatchItem* items, int n_items, const uint32_t h_r[4], const uint32_t* eq_evals, const uint32_t h_lambda[4],
                    uint32_t* h_results);


// ---- a layer's whole sum-check in one launch (no host round trip per round)
//
// What runs in a round depends on the oracles' sizes only, never on the transcript, so the host describes every round of a
// layer's sum-check up front and the device keeps the transcript. Table j (0 <= j <= rounds) holds the fixes of round j - 1 (mode 1 / 2
// items) and the first sums of the oracles that enter in round j (mode 0 items); between two tables comes the transcript step of round
// j: the batch's round polynomial from all oracles' sums, mixed into the channel, the challenge drawn, every oracle's claim and
// correction updated. The launch leaves the round polynomials, the challenges, the masks and the channel in page-locked
// memory (sumcheck.rs:96-176 inside gkr_prover.rs:669-844).
struct GkrRoundConst {
    // The basis of the round's polynomials (all active oracles have n_rem variables left, so their round polynomials are
    // r0 L0 + r1 L1 + r2 L2 over one basis): e0a = eq(0, y) / prod, e2a = eq(2, y) / prod, L[i] the coefficients (low first)
    // of the basis polynomial of node i; y = the coordinate of the layer's point this round fixes.
    uint32_t e0a[4], e2a[4], L[3][4][4], y[4];
    uint32_t n_rem, pad[3];
};
static_assert(sizeof(GkrRoundConst) == 256, "GkrRoundConst layout");

constexpr int GKR_LAYER_MAX_ROUNDS = 31;
constexpr size_t GKR_LAYER_MASK_WORDS = 16;  // per oracle: the two fixed denominators, the two fixed numerators
constexpr size_t GKR_LAYER_OUT_WORDS = 24;  // per round: [0,16) coefficients, [16] length, [20,24) challenge

// What depends on the oracles' sizes and addresses only: a caller makes and stages it while the layer before runs.
struct GkrLayerPlan {
    int n_rounds = 0;                // the variables of the largest oracle
    std::vector<uint32_t> n_vars;    // per oracle: it is active in the rounds with at most so many variables left
    std::vector<GkrBatchItem> items; // table after table; table j: the fixes of round j - 1, the first sums of those entering in round j (slot = oracle)
    std::vector<size_t> table_at;    // n_rounds + 2
    std::vector<uint32_t> tables;    // filled by gkr_batch_plan: how the kernel takes them
    int look_from = -1;              // and from which round on the rounds are taken ahead of the transcript, with which items (-1: none, and `items`)
    std::vector<GkrBatchItem> look_items;
    bool needs_eq = true;            // whether begin wants the table of eq(., point)
    const GkrBatchItem* d_items = nullptr;  // staged by gkr_batch_plan, and what else does not depend on the transcript
    uint32_t* d_blob = nullptr;
    bool launches = false;           // the layer as a launch per table and one per transcript step
    bool refused = false;            // to be tried: as though the one launch were refused
};
int gkr_batch_plan(zkb_ctx* ctx, GkrLayerPlan& plan);

// How a layer's rounds are taken, by their terms and the CTAs of the launch.
constexpr int GKR_THREADS_LOG = 9;  // of a CTA
constexpr int GKR_EQ_BITS = 15;     // of a term's index, for eq without a table
// Four lanes a term while that is at most two passes of the whole grid: a pass of this form is a third of the other's latency,
// and a third more work.
inline bool gkr_four_lanes(size_t terms, uint32_t grid) { return 4 * terms <= 2 * ((size_t)grid << GKR_THREADS_LOG); }
// The round from which on they are taken ahead of the transcript (gkr_batch.cu), or -1. terms[j]: round j's, of all the oracles that are active by then;
// they fall by half from round to round, and grow where shorter oracles enter. A round ahead takes eight lanes for a term of the round after it: some
// 4,500 cycles and 5,000 for 512 lanes a CTA, 9,500 at least, where an ordinary round takes 16,000 and for a large one less per term than this. So what all rounds
// from a candidate on save has to make up for the large ones among them. One instance of 2^16 above 500 of 2^14: 5.2 ms with no round ahead, 7.3 from the first
// small round on, 5.2 by this rule; of 2^14 above 300 of 2^13: 3.1, 3.3 and 2.8; 34 of 2^10 ... 2^13, whose rounds only fall: 1.10, 0.82 and 0.82. A layer that is ahead from its
// first round on works eq out from the point, and the launch that would write the table is saved: 13 instances of 2^11 ... 2^15 0.921 ms without that in the
// sum, 0.908 with it. No pass has more than 45 times 512 lanes a CTA then: 31 rounds do not save more (look_term's sums rest on it).
inline int gkr_look_from(const size_t* terms, int n_rounds, uint32_t grid) {
    constexpr int64_t ORDINARY = 16000, AHEAD = 9500, AHEAD_BASE = 4500, AHEAD_PIECE = 5000, EQ_TABLE = 10000;
    if (grid < 2) return -1;
    int from = -1;
    int64_t saved = 0, most = 0;
    for (int j = n_rounds - 1; j >= 0; j--) {
        const int64_t lanes = j + 1 < n_rounds ? 8 * (int64_t)terms[j + 1] : 0;
        saved += ORDINARY - std::max(AHEAD, AHEAD_BASE + AHEAD_PIECE * lanes / ((int64_t)(grid - 1) << GKR_THREADS_LOG));
        if (j == 0 && n_rounds - 1 <= GKR_EQ_BITS) saved += EQ_TABLE;
        if (j + 2 > n_rounds || saved <= most || !gkr_four_lanes(terms[j], grid)) continue;
        most = saved;
        from = j;
    }
    return from;
}

// alpha_pow[k] = alpha^k; claims[k]: oracle k's claim before the first round (4 words each). chan: digest (8 words) and n_draws.
// Enqueues the layer; gkr_batch_layer_end waits for it. Only gkr_batch_plan may come between the two. GKR_BATCH_AGAIN: the launch was refused and the plan is
// another one now (launches, which needs the table); call again.
constexpr int GKR_BATCH_AGAIN = -1000;
int gkr_batch_layer_begin(zkb_ctx* ctx, GkrLayerPlan& plan, const uint32_t* alpha_pow, const uint32_t* claims, const GkrRoundConst* rounds,
                          const uint32_t* eq_evals, const uint32_t h_lambda[4], const uint32_t chan[9]);

// In the context's memory, until the next call: n_rounds x GKR_LAYER_OUT_WORDS, the channel as above, n_oracles x GKR_LAYER_MASK_WORDS
// (of every oracle that had a round).
struct GkrLayerResult {
    const uint32_t *records, *channel, *masks;
};
int gkr_batch_layer_end(zkb_ctx* ctx, const GkrLayerPlan& plan, GkrLayerResult& res);

}  // namespace zk
