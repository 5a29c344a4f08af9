// Reads of many (column, row) cells in one round trip (ctx.cu); internal to the library.
#pragma once
#include <cstddef>
#include <cstdint>
#include <utility>

struct zkb_ctx;

namespace zk {

// A table of device addresses on the device, where operators that are given the same table soon after find it.
int stage_table(zkb_ctx* ctx, const uint32_t* const* ptrs, int n);
// Several in one copy.
int stage_tables(zkb_ctx* ctx, const std::pair<const uint32_t* const*, size_t>* tables, size_t n_tables);

// out[out_off + i * ncols + c] = cols[c][idx[i]]: the rows idx[0..nidx) of ncols device columns, row-major.
// cols and idx are host arrays (cols holds device pointers).
struct GatherBlock {
    const uint32_t* const* cols;
    int ncols;
    const uint32_t* idx;
    int nidx;
    size_t out_off;
};

// Every cell of every block, every word of word_addrs and every hash (8 words) of hash_addrs, in one round trip: results go to
// h_out as [blocks: total_words][one word per word address][eight words per hash address], which should be page-locked. A
// decommitment's whole read plan (Column::batch_at and batch_at_multi, nitroo/crates/stwo/src/prover/backend/mod.rs:68-89, for all
// the layers of all the trees at once): the addresses and indices travel in one staged block, and one launch reads everything.
int gather_plan(zkb_ctx* ctx, const GatherBlock* blocks, int n_blocks, size_t total_words, const uint32_t* const* word_addrs, size_t n_words,
                const uint32_t* const* hash_addrs, size_t n_hashes, uint32_t* h_out);

}  // namespace zk
