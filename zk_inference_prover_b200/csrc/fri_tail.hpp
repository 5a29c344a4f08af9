// The last layers of a FRI commitment in one launch (fri_tail.cu); internal to the library.
#pragma once
#include <cstddef>
#include <cstdint>

struct zkb_ctx;

namespace zk {

constexpr int FRI_TAIL_LOG = 10;        // largest layer (log2) the launch takes
constexpr int FRI_TAIL_MAX_LAST = 5;     // largest last layer (log2) it interpolates
constexpr int FRI_TAIL_MAX_BOUND = 2;    // largest log2 of the last layer's coefficients it mixes into the channel

struct FriTailArgs {
    const uint32_t* src[4];              // the first layer's coordinate columns
    int first_log, n_layers;             // its size; committed layers (each half the one before), at least one
    int circle;                          // the first layer lies on the circle domain (first_log >= 3); line domains otherwise
    // Layer k's tree: level j (2^j hashes) at tree[k] + 8 * 2^j. Folded layer k (what layer k becomes): coordinate c at
    // evals[k] + c * fri_tail_stride(log).
    uint32_t* tree[FRI_TAIL_LOG + 1];
    uint32_t* evals[FRI_TAIL_LOG + 1];
    const uint32_t* chan;                // channel state on the device (digest, n_draws), or NULL: the one below
    uint32_t digest[8], n_draws;
    uint32_t* out;                       // fri_tail_out_words(n_layers) words, see below
    // last_bound >= 0: also interpolate the last layer (2^last_log values), mix its 2^last_bound coefficients into the channel and
    // leave the digest a proof of work of pow_bits is searched for, with the search's result slot set to "none found".
    int last_log, last_bound;
    uint32_t pow_bits;
};
// out: [0,8) digest, [8] draws, [9] not zero if the last layer has a higher degree, [10] smallest nonce found (all ones: none),
// [16,24) the digest to search with, [32, 32 + 16) the last layer's coefficients, then a root per layer.
constexpr size_t FRI_TAIL_ROOTS = 48;
inline size_t fri_tail_out_words(int n_layers) { return FRI_TAIL_ROOTS + 8 * (size_t)n_layers; }
inline size_t fri_tail_stride(int log) { return log < 2 ? 4 : (size_t)1 << log; }

int fri_tail(zkb_ctx* ctx, const FriTailArgs& args);

// The layers above those in one launch of many CTAs. Where it runs it also takes the two largest that the other one could (a layer of 2^10 values takes one CTA 16 us,
// sixteen of them 13); for those alone the launch does not pay: a proof of ten columns, domain 2^10: 236 us without it, 241 with; four columns, domain 2^14: 480
// with neither, 437 with it down to 2^11, 425 down to 2^9. Not from larger layers on with more CTAs: 128 from 2^17 on save a STARK proof another 50 us, but a CTA wants its SM
// to itself, and beside other proofs' long kernels (chains of narrow tree layers, a CTA on most SMs for milliseconds) a grid of 128 waits for all of them with
// the SMs it has: eight proofs side by side took 1.85 s a decode step, 1.05 with 32 CTAs and with launches alone.
constexpr int FRI_MID_LOG = 15;        // largest layer (log2) it takes
constexpr int FRI_MID_END = 8;         // what its last layer folds to is no smaller (log2)
constexpr int FRI_MID_CTAS_LOG = 5;    // slices of 2^6 values and more of a first layer, of 2^4 of the last
constexpr int FRI_MID_DONE = 10;       // the word of the channel's sixteen that is one when the first CTA has ended well, zero before
constexpr int FRI_MID_FAILED = 11;     // ... and that is one when a CTA has given up a wait
struct FriMidArgs {
    const uint32_t* src[4];            // the first layer's coordinate columns
    int first_log, n_layers, circle;   // as above; at least one layer, and the last one folds to no less than 2^FRI_MID_END values
    uint32_t* tree[FRI_MID_LOG - FRI_MID_END];   // as above
    uint32_t* evals[FRI_MID_LOG - FRI_MID_END];
    uint32_t *chan, *roots, *sync;     // channel state, in and out; a root per layer; FRI_MID_SYNC_WORDS zeros
    int impatient;                     // filled by fri_mid
};
constexpr size_t FRI_MID_SYNC_WORDS = ((size_t)16 << FRI_MID_CTAS_LOG) + 8;
constexpr int FRI_MID_REFUSED = -1001; // not all CTAs can be resident: nothing was launched
int fri_mid(zkb_ctx* ctx, FriMidArgs args);
// The first nonces (several times 2^pow_bits of them) tested against the digest at prefixed; the smallest that passes goes to *best.
int grind_first(zkb_ctx* ctx, const uint32_t* prefixed, int pow_bits, uint32_t* best);
// zkb_fold_circle_into_line_dalpha (leaves: ..._leaves, or null) into a line that counts as zero: it is neither cleared first nor read.
int fold_circle_fresh(zkb_ctx* ctx, uint32_t* const dst[4], const uint32_t* const src[4], int log_n_src, const uint32_t* d_alpha, uint32_t* leaves);
// A few words to device memory through the staging ring: no synchronisation.
int upload_small(zkb_ctx* ctx, uint32_t* dst, const uint32_t* h, size_t words);
// `words` of device memory to the context's page-locked buffer and a synchronisation; *h is valid until the next such read.
int read_small(zkb_ctx* ctx, const uint32_t* d, size_t words, const uint32_t** h);

}  // namespace zk
