// Protocol drivers over B200Backend: Merkle prover, FRI prover, commitment-scheme prover and the
// GKR batch prover, with the call order of the reference's backend-generic code (cited per
// function; STWO = nitroo/crates/stwo/src). All field and hash work on columns happens on the
// device through the operator ABI; the host runs the Fiat-Shamir channel, the query bookkeeping
// and scalar QM31 arithmetic on a handful of values per round.
#include <algorithm>
#include <iterator>
#include <chrono>
#include <future>
#include <map>
#include <memory>
#include <numeric>
#include <set>
#include <string>
#include <thread>
#include <cstdio>
#include <cstdlib>

#include <cuda_runtime_api.h>

#include "../../../include/zkb200_prover.h"
#include "../air_program.hpp"
#include "b200_backend.hpp"
#include "commit_groups.hpp"
#include "../fft_internal.hpp"
#include "../gkr_resident.hpp"
#include "../gkr_batch.hpp"
#include "../fri_tail.hpp"
#include "../gather_blocks.hpp"
#include "channel.hpp"
#include "../side_stream.hpp"
#include "../quot_lines.hpp"

// Records a message on the context (defined with the context, ctx.cu).
extern "C" int zk_set_error_public(zkb_ctx* ctx, int code, const char* msg);

namespace b200 {

using namespace zk;

// Host-side timing of the protocol code's own steps (the device has per-kernel events; this is for the time the host
// spends between launches). Off unless ZKB_HOST_TIMING is set; totals per label go to stderr when a proof call returns.
struct HostClock {
    static bool on() { static const bool v = getenv("ZKB_HOST_TIMING") != nullptr; return v; }
    static std::map<std::string, std::pair<double, size_t>>& totals() { static std::map<std::string, std::pair<double, size_t>> m; return m; }
    const char* label;
    std::chrono::steady_clock::time_point t0;
    explicit HostClock(const char* l) : label(l) { if (on()) t0 = std::chrono::steady_clock::now(); }
    ~HostClock() {
        if (!on()) return;
        auto& e = totals()[label];
        e.first += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        e.second++;
    }
    static void dump(const char* what) {
        if (!on()) return;
        fprintf(stderr, "[host timing] %s\n", what);
        for (auto& kv : totals()) fprintf(stderr, "  %-34s %10.3f ms %8zu calls\n", kv.first.c_str(), kv.second.first, kv.second.second);
        totals().clear();
    }
};

static inline uint32_t ilog2(size_t n) { return n ? 63u - (uint32_t)__builtin_clzll((unsigned long long)n) : 0u; }
static inline qm31 operator+(qm31 a, qm31 b) { return qm31_add(a, b); }
static inline qm31 operator-(qm31 a, qm31 b) { return qm31_sub(a, b); }
static inline qm31 operator*(qm31 a, qm31 b) { return qm31_mul(a, b); }

static std::vector<size_t> sorted_dedup(std::vector<size_t> v) {
    std::sort(v.begin(), v.end());
    v.erase(std::unique(v.begin(), v.end()), v.end());
    return v;
}
static std::vector<size_t> fold_queries(const std::vector<size_t>& q, uint32_t n_folds) {  // core/queries.rs:55-62
    std::vector<size_t> out;
    for (auto x : q) { size_t y = x >> n_folds; if (out.empty() || out.back() != y) out.push_back(y); }
    return out;
}

// Every address a decommitment will read is known once the query positions are: collect them all,
// read them in one device round trip, then assemble the proof parts from the results.
struct GatherPlan {
    std::vector<const uint32_t*> addrs;        // single words
    std::vector<const uint32_t*> hash_addrs;   // eight words each
    std::vector<uint32_t> words, hash_words;
    size_t add(const uint32_t* p) { addrs.push_back(p); return addrs.size() - 1; }
    size_t add_hash(const uint32_t* p) { hash_addrs.push_back(p); return hash_addrs.size() - 1; }
    // Rows of many columns at once (the queried and witness values of one tree layer): row-major [row][column] in
    // block_words from the returned offset. One pointer per column and one index per row travel, not one address per word.
    struct Block { const std::vector<const uint32_t*>* cols; std::vector<uint32_t> idx; size_t out_off; };  // cols: its owner outlives the plan
    std::vector<Block> blocks;
    // Tens of megabytes for trees of many columns. The buffer is kept per thread between proofs: a fresh allocation of
    // that size comes from mmap, and its first-touch page faults cost as much as the gather itself.
    uint32_t* block_words = nullptr;
    size_t block_total = 0;
    // Page-locked: the device-to-host copy of a wide tree's values then runs at the link's speed instead of through the
    // driver's bounce buffers (50 MB: 4 ms pageable), and a short one does not wait for them.
    struct Arena {
        uint32_t* p = nullptr;
        size_t words = 0;
        bool pinned = false;
        void release() {
            if (!p) return;
            if (pinned) cudaFreeHost(p); else free(p);
            p = nullptr; words = 0;
        }
        // Nothing is released when the thread ends: at process exit the CUDA runtime may already be gone.
    };
    static uint32_t* arena(size_t words) {
        thread_local Arena a;
        if (a.words < words) {
            a.release();
            size_t want = std::max<size_t>(words + words / 4, (size_t)1 << 18);
            void* q = nullptr;
            if (cudaMallocHost(&q, want * 4) == cudaSuccess && q) a.pinned = true;
            else { (void)cudaGetLastError(); q = malloc(want * 4); a.pinned = false; }
            if (!q) throw Error(ZKB_ENOMEM, "gather buffer");
            a.p = (uint32_t*)q;
            a.words = want;
        }
        return a.p;
    }
    size_t add_block(const std::vector<const uint32_t*>& cols, const std::vector<size_t>& rows) {
        Block b;
        b.cols = &cols;
        b.idx.reserve(rows.size());
        for (auto r : rows) b.idx.push_back((uint32_t)r);
        b.out_off = block_total;
        block_total += cols.size() * rows.size();
        blocks.push_back(std::move(b));
        return blocks.back().out_off;
    }
    void execute(const Device& d) {
        const size_t n = addrs.size(), nh = hash_addrs.size();
        uint32_t* out = arena(block_total + n + 8 * nh);
        std::vector<zk::GatherBlock> gb;
        gb.reserve(blocks.size());
        for (auto& b : blocks) gb.push_back({b.cols->data(), (int)b.cols->size(), b.idx.data(), (int)b.idx.size(), b.out_off});
        d.check(zk::gather_plan(d.ctx(), gb.data(), (int)gb.size(), block_total, addrs.data(), n, hash_addrs.data(), nh, out));
        block_words = out;
        words.assign(out + block_total, out + block_total + n);
        hash_words.assign(out + block_total + n, out + block_total + n + 8 * nh);
    }
    Hash hash_at(size_t slot) const { Hash h; for (int k = 0; k < 8; k++) h[k] = hash_words[8 * slot + k]; return h; }
};

// ------------------------------------------------------------------ MerkleProver (STWO/prover/vcs/prover.rs:17-217)
// A word sequence of a proof: its own vector, or runs inside the gather buffer of the plan that read them (the buffer is
// kept per thread until the next proof on that thread, so a proof can be serialised straight out of it: a tree of tens of
// thousands of columns has tens of megabytes of queried values, and every copy of them costs milliseconds).
struct Words {
    std::vector<uint32_t> own;
    std::vector<std::pair<const uint32_t*, size_t>> runs;
    size_t size() const { size_t n = own.size(); for (auto& r : runs) n += r.second; return n; }
    template <class O> void append_to(O& o) const {
        o.insert(o.end(), own.begin(), own.end());
        for (auto& r : runs) o.insert(o.end(), r.first, r.first + r.second);
    }
};
struct MerkleDecommitment { std::vector<Hash> hash_witness; Words column_witness; };
struct PendingMerkle {  // slots of a planned decommitment
    std::vector<size_t> hash_slots;
    struct Run { size_t off, count; bool queried; };  // `count` words of plan.block_words, in proof order
    std::vector<Run> runs;
    std::pair<Words, MerkleDecommitment> finish(const GatherPlan& plan) const {
        std::pair<Words, MerkleDecommitment> r;
        r.second.hash_witness.reserve(hash_slots.size());
        for (auto s : hash_slots) r.second.hash_witness.push_back(plan.hash_at(s));
        for (auto& run : runs) (run.queried ? r.first : r.second.column_witness).runs.push_back({plan.block_words + run.off, run.count});
        return r;
    }
};

// Queries of one layer only.
struct QueriesOf {
    uint32_t log;
    const std::vector<size_t>& positions;
    const std::vector<size_t>& operator()(uint32_t l) const { static const std::vector<size_t> none; return l == log ? positions : none; }
};

struct MerkleProver {
    std::vector<HashColumn> layers;  // layers[log_size]; layers[0] holds the root
    // the committed columns of each layer (device addresses, in commitment order), kept for the decommitment: sorting tens
    // of thousands of columns by size a second time costs milliseconds
    std::vector<std::vector<const uint32_t*>> layer_col_ptrs;

    // `leaves`, when given, is the already hashed largest layer (see zkb_merkle_leaves_partial).
    // `chan_step`, when given, is a FRI layer's channel step (channel state, challenge slot, root copy; device addresses) to run
    // in the launch that builds the root; *chan_done says whether it ran (a tree of one node has no such launch).
    struct ChanStep { uint32_t *chan, *alpha, *root_copy; };
    // The launch that ends a tree takes it from 2^8 hashes on: below, a hash is a quad's (blake2s.cu), and the two levels above cost
    // the launch before it 2 us and this one, with the code for a thread a hash to fetch, 7.
    static constexpr uint32_t TOP_LOG = 8;
    static MerkleProver commit(const Device& d, const std::vector<const BaseColumn*>& columns, HashColumn* leaves = nullptr,
                               const ChanStep* chan_step = nullptr, bool* chan_done = nullptr);  // :39-64
    Hash root(const Device& d) const {
        if (!have_root) {
            const uint32_t* h = nullptr;
            d.check(zk::read_small(d.ctx(), layers[0].ptr(), 8, &h));
            std::copy(h, h + 8, root_cache.begin());
            have_root = true;
        }
        return root_cache;
    }
    mutable Hash root_cache{};
    mutable bool have_root = false;

    // :84-217 — the reference plans the indices of all layers on the host first (its phase 1) and then
    // reads layer by layer; here the reads of all layers join one GatherPlan, over the layers' columns as commit() recorded them.
    // queries(log): the ascending distinct nodes queried of the layer of 2^log (rows of its columns).
    // `hashes_per_layer`, when given, receives the number of witness hashes each layer contributed (largest layer first).
    template <class Queries>
    PendingMerkle plan_decommit(GatherPlan& plan, Queries queries, std::vector<size_t>* hashes_per_layer = nullptr) const {
        PendingMerkle pm;
        static const std::vector<const uint32_t*> no_columns;
        // Sorted vectors walked in step: `last` (the nodes of the layer below) is ascending, so are its halves and the layer's
        // own queries; a FRI proof plans some twenty trees of some twenty layers each.
        std::vector<size_t> last, nodes, order, witness_nodes;
        for (uint32_t log = (uint32_t)layers.size(); log-- > 0;) {
            const bool has_prev = (size_t)log + 1 < layers.size();
            const std::vector<const uint32_t*>& ptrs = log < layer_col_ptrs.size() ? layer_col_ptrs[log] : no_columns;
            const std::vector<size_t>& col_queries = queries(log);
            nodes.clear();
            order.clear();
            witness_nodes.clear();
            size_t p = 0, q = 0, hashes = 0;
            while (p < last.size() || q < col_queries.size()) {
                const size_t node = p == last.size() ? col_queries[q] : q == col_queries.size() ? last[p] / 2 : std::min(last[p] / 2, col_queries[q]);
                bool child[2] = {false, false};
                for (; p < last.size() && last[p] / 2 == node; p++) child[last[p] & 1] = true;
                const bool queried = q < col_queries.size() && col_queries[q] == node;
                if (queried) q++;
                if (has_prev)
                    for (size_t k = 0; k < 2; k++)
                        if (!child[k]) { pm.hash_slots.push_back(plan.add_hash(layers[log + 1].ptr() + 8 * (2 * node + k))); hashes++; }
                nodes.push_back(node);
                (queried ? order : witness_nodes).push_back(node);
            }
            if (hashes_per_layer) hashes_per_layer->push_back(hashes);
            if (!ptrs.empty() && !nodes.empty()) {
                // every node of the layer is read once; the proof lists the queried nodes' values first, then the witnesses'
                const size_t n_queried = order.size();
                order.insert(order.end(), witness_nodes.begin(), witness_nodes.end());
                const size_t off = plan.add_block(ptrs, order);
                if (n_queried) pm.runs.push_back({off, n_queried * ptrs.size(), true});
                if (!witness_nodes.empty()) pm.runs.push_back({off + n_queried * ptrs.size(), witness_nodes.size() * ptrs.size(), false});
            }
            std::swap(last, nodes);
        }
        return pm;
    }
};

// A tree from its largest layer down, as far as its columns are there: a layer's columns have to be enqueued only when it is hashed.
struct MerkleBuilder {
    const Device& d;
    MerkleProver tree;
    int next = -1;         // the layer to hash next; negative: the tree is whole
    size_t count[33];      // columns of each layer
    uint32_t min_log = 32;

    MerkleBuilder(const Device& dev, const size_t (&columns)[33]) : d(dev) {
        for (int log = 0; log <= 32; log++) {
            count[log] = columns[log];
            if (!count[log]) continue;
            next = log;
            min_log = std::min(min_log, (uint32_t)log);
        }
        if (next < 0) {
            tree.layers.push_back(B200Backend::commit_on_layer(d, 0, nullptr, {}));
            return;
        }
        tree.layers.resize((size_t)next + 1);
        tree.layer_col_ptrs.resize((size_t)next + 1);
    }
    // The layer at `next`, whose columns are in tree.layer_col_ptrs, and what follows from it in the same launches.
    void hash_next(HashColumn* leaves = nullptr, const MerkleProver::ChanStep* chan_step = nullptr, bool* chan_done = nullptr) {
        constexpr uint32_t TOP_LOG = MerkleProver::TOP_LOG;
        auto& layers = tree.layers;
        uint32_t log = (uint32_t)next;
        auto top = [&] {  // the rest of the tree is nodes only, built in one launch
            std::vector<uint32_t*> lower;
            for (uint32_t k = 0; k < log; k++) { layers[k] = HashColumn(d, (size_t)8 << k); lower.push_back(layers[k].ptr()); }
            if (chan_step && log >= 1) {
                d.check(zkb_merkle_top_channel(d.ctx(), (int)log, layers[log].ptr(), lower.data(), 1, chan_step->chan, chan_step->alpha, chan_step->root_copy));
                if (chan_done) *chan_done = true;
            } else d.check(zkb_merkle_top(d.ctx(), (int)log, layers[log].ptr(), lower.data(), 1));
            next = -1;
        };
        const bool first = (size_t)log + 1 == layers.size();
        if (first && leaves) layers[log] = std::move(*leaves);
        else {
            layers[log] = HashColumn(d, (size_t)8 << log);
            d.check(zkb_merkle_layer(d.ctx(), (int)log, first ? nullptr : layers[log + 1].ptr(), tree.layer_col_ptrs[log].data(), (int)tree.layer_col_ptrs[log].size(), 1,
                                     layers[log].ptr()));
        }
        const bool all = log <= min_log;  // no columns left below
        if (log > 0 && log <= TOP_LOG && all) return top();
        // The layers below this one that hold no column (down to the next layer that has one, or to the last ones, which
        // the launch above builds): up to nine of them per launch.
        uint32_t floor_log = TOP_LOG;
        if (!all) {
            uint32_t below = log - 1;
            while (!count[below]) below--;
            floor_log = below + 1;
        }
        while (log > floor_log && log >= 9) {
            const uint32_t levels = std::min<uint32_t>(9, log - floor_log);
            std::vector<uint32_t*> outs;
            for (uint32_t j = 1; j <= levels; j++) { layers[log - j] = HashColumn(d, (size_t)8 << (log - j)); outs.push_back(layers[log - j].ptr()); }
            d.check(zkb_merkle_levels(d.ctx(), (int)log, layers[log].ptr(), (int)levels, outs.data(), 1));
            log -= levels;
        }
        if (log > 0 && log <= TOP_LOG && all && layers[log - 1].len() == 0) return top();
        next = (int)log - 1;
    }
    // ... and on to the next layer with columns.
    void hash_to_columns() {
        do hash_next();
        while (next >= 0 && !count[next]);
    }
};

inline MerkleProver MerkleProver::commit(const Device& d, const std::vector<const BaseColumn*>& columns, HashColumn* leaves, const ChanStep* chan_step, bool* chan_done) {
    if (chan_done) *chan_done = false;
    size_t count[33] = {0};
    for (auto c : columns) count[c->log_size()]++;
    MerkleBuilder builder(d, count);
    auto& cols = builder.tree.layer_col_ptrs;
    for (size_t log = 0; log < cols.size(); log++) cols[log].reserve(count[log]);
    for (auto c : columns) cols[c->log_size()].push_back(c->ptr());
    while (builder.next >= 0) builder.hash_next(leaves, chan_step, chan_done);
    return std::move(builder.tree);
}

// ------------------------------------------------------------------ FRI (STWO/prover/fri.rs:87-467)
struct FriConfig {
    uint32_t log_blowup_factor, log_last_layer_degree_bound, n_queries, line_fold_step;
    size_t last_layer_domain_size() const { return (size_t)1 << (log_last_layer_degree_bound + log_blowup_factor); }
};
struct FriLayerProof { std::vector<qm31> fri_witness; MerkleDecommitment decommitment; Hash commitment; };
struct FriProof { FriLayerProof first_layer; std::vector<FriLayerProof> inner_layers; std::vector<qm31> last_layer_poly; };

static cpoint host_circle_point(uint32_t index) {
    cpoint g{2u, 1268011823u}, r{1u, 0u};
    for (int b = 0; b < 31; b++) {
        if ((index >> b) & 1u) r = cpoint_add(r, g);
        g = cpoint_add(g, g);
    }
    return r;
}
template <class T> static void bit_reverse_vec(std::vector<T>& v) {
    uint32_t log = ilog2(v.size());
    for (size_t i = 0; i < v.size(); i++) {
        size_t j = 0;
        for (uint32_t b = 0; b < log; b++) j |= ((i >> b) & 1) << (log - 1 - b);
        if (j > i) std::swap(v[i], v[j]);
    }
}
// LineEvaluation::interpolate on the host (STWO/prover/line.rs:41-66) for the last FRI layer, whose
// domain is Coset::half_odds(log): initial index 2^(29-log), step 2^(31-log).
static std::vector<qm31> line_interpolate(std::vector<qm31> values) {
    uint32_t log = ilog2(values.size());
    bit_reverse_vec(values);
    for (uint32_t k = log; k > 0; k--) {  // domain of the current chunk size 2^k: half_odds(k)
        size_t size = (size_t)1 << k, half = size / 2;
        for (size_t off = 0; off < values.size(); off += size)
            for (size_t i = 0; i < half; i++) {
                uint32_t idx = ((1u << (29 - k)) + ((uint32_t)i << (31 - k))) & 0x7fffffffu;
                uint32_t xinv = m31_inv(host_circle_point(idx).x);
                qm31 a = values[off + i], b = values[off + half + i];
                values[off + i] = a + b;
                values[off + half + i] = qm31_mul_m31(a - b, xinv);
            }
    }
    uint32_t len_inv = m31_inv((uint32_t)values.size());
    for (auto& v : values) v = qm31_mul_m31(v, len_inv);
    return values;
}

static std::vector<qm31> secure_at_batch(const Device& d, const SecureColumnByCoords& col, const std::vector<size_t>& positions) {
    auto flat = B200Backend::batch_at_multi(d, col.refs(), positions);  // secure_column.rs:33-44
    std::vector<qm31> out(positions.size());
    for (size_t j = 0; j < positions.size(); j++) out[j] = {{flat[4 * j], flat[4 * j + 1], flat[4 * j + 2], flat[4 * j + 3]}};
    return out;
}

struct PendingFriLayer {
    std::vector<size_t> eval_slots;  // 4 per decommitment position
    std::vector<bool> is_witness;
    PendingMerkle merkle;
    Hash commitment;
};

// fri.rs:392-436 — positions first, then one gather for all of them (here: joined to the plan).
static PendingFriLayer plan_fri_layer(GatherPlan& plan, const Device& d, const SecureColumnByCoords& column, const MerkleProver& tree,
                                      const std::vector<size_t>& queries, uint32_t fold_step) {
    PendingFriLayer pl;
    std::vector<size_t> positions;
    size_t i = 0;
    while (i < queries.size()) {
        size_t j = i;
        while (j < queries.size() && (queries[j] >> fold_step) == (queries[i] >> fold_step)) j++;
        size_t start = (queries[i] >> fold_step) << fold_step, qi = i;
        for (size_t p = start; p < start + ((size_t)1 << fold_step); p++) {
            positions.push_back(p);
            if (qi < j && queries[qi] == p) { qi++; pl.is_witness.push_back(false); }
            else pl.is_witness.push_back(true);
        }
        i = j;
    }
    for (size_t p : positions)
        for (int k = 0; k < 4; k++) pl.eval_slots.push_back(plan.add(column.columns[k].ptr() + p));
    pl.merkle = tree.plan_decommit(plan, QueriesOf{column.columns[0].log_size(), positions});
    pl.commitment = tree.root(d);
    return pl;
}

struct FriProver {
    FriConfig config;
    const SecureColumnByCoords* first_column = nullptr;
    MerkleProver first_tree;
    struct Inner { SecureColumnByCoords eval; MerkleProver tree; uint32_t fold_step; };
    std::vector<Inner> inner;
    BaseColumn mid_slab, tail_slab;  // trees and layers of the launches that run the middle and the last layers, which `inner` holds views of
    std::vector<qm31> last_layer_poly;

    bool have_nonce = false;  // the proof of work was searched for along with the commitment (grind_bits)
    uint64_t nonce = 0;

    // Memory for n layers from 2^log on that one launch commits and folds: each one's tree and what it folds to (FriTailArgs).
    static std::vector<std::pair<uint32_t*, uint32_t*>> layer_slab(const Device& d, BaseColumn& slab, uint32_t log, size_t n) {
        size_t words = 0;
        for (uint32_t k = 0; k < n; k++) words += ((size_t)16 << (log - k)) + 4 * zk::fri_tail_stride((int)(log - k) - 1);
        slab = BaseColumn(d, words);
        std::vector<std::pair<uint32_t*, uint32_t*>> places;
        uint32_t* at = slab.ptr();
        for (uint32_t k = 0; k < n; k++) {
            uint32_t* const tree = at;
            at += (size_t)16 << (log - k);
            places.push_back({tree, at});
            at += 4 * zk::fri_tail_stride((int)(log - k) - 1);
        }
        return places;
    }
    // Layers `first` and on, of 2^log values, which such a launch has committed; layer: the first of them, and what the last one folds to afterwards.
    void adopt_layers(const Device& d, const SecureColumnByCoords& column, SecureColumnByCoords& layer, size_t first, uint32_t log,
                      const std::vector<std::pair<uint32_t*, uint32_t*>>& places) {
        for (size_t k = 0; k < places.size(); k++, log--) {
            if (first + k == 0) first_tree = tree_view(d, places[k].first, log, column);
            else {
                Inner in{std::move(layer), {}, 1};
                in.tree = tree_view(d, places[k].first, log, in.eval);
                inner.push_back(std::move(in));
            }
            layer = SecureColumnByCoords();
            for (int c = 0; c < 4; c++)
                layer.columns[c] = BaseColumn::view(d, places[k].second + c * zk::fri_tail_stride((int)log - 1), (size_t)1 << (log - 1));
        }
    }

    // A tree in memory laid out as the tail's launch writes it (FriTailArgs::tree).
    static MerkleProver tree_view(const Device& d, uint32_t* tree, uint32_t log, const SecureColumnByCoords& eval) {
        MerkleProver mp;
        for (uint32_t j = 0; j <= log; j++) mp.layers.push_back(HashColumn::view(d, tree + ((size_t)8 << j), (size_t)8 << j));
        mp.layer_col_ptrs.resize(log + 1);
        for (auto p : eval.cptrs()) mp.layer_col_ptrs[log].push_back(p);
        return mp;
    }

    // fri.rs:109-221. grind_bits >= 0: the proof of work of that many bits follows the commitment in the transcript, and its first
    // nonces may be tested in the same round trip (have_nonce says whether one was found).
    static FriProver commit(const Device& d, Channel& ch, FriConfig config, const SecureColumnByCoords& column, int grind_bits = -1) {
        FriProver fp;
        fp.config = config;
        fp.first_column = &column;
        uint32_t first_log = column.columns[0].log_size(), inner_log = first_log - 1;
        uint32_t last_log = ilog2(config.last_layer_domain_size());
        SecureColumnByCoords layer;
        bool last_done = false;
        if (config.line_fold_step == 1) {
            // Device-resident commit phase: every layer's tree, the channel step (mix the root, draw the
            // folding challenge) and the fold are enqueued back to back; the host reads all roots and the
            // channel state once, after the last fold. The last layers, of at most 2^FRI_TAIL_LOG values, run in one launch.
            const size_t n_layers = 1 + (inner_log > last_log ? inner_log - last_log : 0);
            const size_t tail = first_log > (uint32_t)zk::FRI_TAIL_LOG ? std::min<size_t>(n_layers, first_log - zk::FRI_MID_END)
                                : first_log >= 3 && inner_log >= last_log ? 0 : n_layers;  // the first layer of that launch
            const bool last_in_tail = tail < n_layers && last_log <= (uint32_t)zk::FRI_TAIL_MAX_LAST &&
                                      config.log_last_layer_degree_bound <= (uint32_t)zk::FRI_TAIL_MAX_BOUND;
            // Of the layers before that launch those of at most 2^FRI_MID_LOG values are one launch too; the others are launches of their own.
            const size_t launched = first_log > (uint32_t)zk::FRI_MID_LOG ? std::min<size_t>(tail, first_log - zk::FRI_MID_LOG) : first_log > (uint32_t)zk::FRI_TAIL_LOG ? 0 : tail;
            const size_t mid_layers = tail - launched;
            const uint32_t mid_log = first_log - (uint32_t)launched;
            // [the middle launch's meeting place | channel 16 | challenges 4 each (16-byte aligned) | roots 8 each | the tail's results]
            const size_t sync_words = mid_layers ? zk::FRI_MID_SYNC_WORDS : 0;
            const size_t tail_at = 16 + 12 * tail, tail_layers = n_layers - tail;
            BaseColumn fs(d, sync_words + tail_at + zk::fri_tail_out_words((int)tail_layers));
            uint32_t* const sync = fs.ptr();
            uint32_t* const chan = sync + sync_words;
            uint32_t* alphas = chan + 16;
            uint32_t* roots = chan + 16 + 4 * tail;
            bool mid_done = false;
            if (tail > 0) {
                std::vector<uint32_t> st(sync_words + 16, 0u);
                for (int k = 0; k < 8; k++) st[sync_words + k] = ch.digest()[k];
                st[sync_words + 8] = ch.n_draws();
                d.check(zk::upload_small(d.ctx(), sync, st.data(), st.size()));
                HashColumn leaves;
                bool have_leaves = false, stepped = false;
                // Layers [k0, k1) as launches; every fold but the last also hashes the leaves of the layer it produces: that layer is committed next.
                auto launch_layers = [&](size_t k0, size_t k1) {
                    for (size_t k = k0; k < k1; k++) {
                        MerkleProver::ChanStep step{chan, alphas + 4 * k, roots + 8 * k};
                        Inner in{std::move(layer), {}, 1};
                        std::vector<const BaseColumn*> refs = k ? in.eval.refs() : column.refs();
                        MerkleProver tree = MerkleProver::commit(d, refs, have_leaves ? &leaves : nullptr, &step, &stepped);
                        if (!stepped) d.check(zkb_channel_mix_root_draw(d.ctx(), chan, tree.layers[0].ptr(), alphas + 4 * k, roots + 8 * k));
                        have_leaves = k + 1 < k1 && (k > 0 || first_log >= 3);
                        if (k == 0) {
                            layer = SecureColumnByCoords(d, (size_t)1 << inner_log);
                            B200Backend::fold_circle_into_line(d, layer, column, alphas, have_leaves ? &leaves : nullptr);
                            fp.first_tree = std::move(tree);
                            continue;
                        }
                        layer = have_leaves ? B200Backend::fold_line(d, in.eval, alphas + 4 * k, leaves) : B200Backend::fold_line(d, in.eval, alphas + 4 * k);
                        in.tree = std::move(tree);
                        fp.inner.push_back(std::move(in));
                    }
                };
                launch_layers(0, launched);
                if (mid_layers) {
                    zk::FriMidArgs ma;
                    memset(&ma, 0, sizeof(ma));
                    const std::vector<std::pair<uint32_t*, uint32_t*>> places = fp.layer_slab(d, fp.mid_slab, mid_log, mid_layers);
                    for (size_t k = 0; k < mid_layers; k++) { ma.tree[k] = places[k].first; ma.evals[k] = places[k].second; }
                    const auto src = launched ? layer.cptrs() : column.cptrs();
                    for (int c = 0; c < 4; c++) ma.src[c] = src[c];
                    ma.first_log = (int)mid_log;
                    ma.n_layers = (int)mid_layers;
                    ma.circle = launched == 0;
                    ma.chan = chan;
                    ma.roots = roots + 8 * launched;
                    ma.sync = sync;
                    const int rc = zk::fri_mid(d.ctx(), ma);
                    if (rc == zk::FRI_MID_REFUSED) {
                        fp.mid_slab = BaseColumn();
                        launch_layers(launched, tail);
                    } else {
                        d.check(rc);
                        mid_done = true;
                        fp.adopt_layers(d, column, layer, launched, mid_log, places);
                    }
                }
            }
            if (tail_layers > 0) {
                zk::FriTailArgs ta;
                memset(&ta, 0, sizeof(ta));
                const uint32_t log0 = first_log - (uint32_t)tail;
                const std::vector<std::pair<uint32_t*, uint32_t*>> places = fp.layer_slab(d, fp.tail_slab, log0, tail_layers);
                for (size_t k = 0; k < tail_layers; k++) { ta.tree[k] = places[k].first; ta.evals[k] = places[k].second; }
                const auto src = tail ? layer.cptrs() : column.cptrs();
                for (int c = 0; c < 4; c++) ta.src[c] = src[c];
                ta.first_log = (int)log0;
                ta.n_layers = (int)tail_layers;
                ta.circle = tail == 0;
                if (tail) ta.chan = chan;
                for (int k = 0; k < 8; k++) ta.digest[k] = ch.digest()[k];
                ta.n_draws = ch.n_draws();
                ta.out = chan + tail_at;
                ta.last_log = (int)last_log;
                ta.last_bound = last_in_tail ? (int)config.log_last_layer_degree_bound : -1;
                ta.pow_bits = grind_bits > 0 ? (uint32_t)grind_bits : 0u;
                d.check(zk::fri_tail(d.ctx(), ta));
                if (last_in_tail && grind_bits > 0) d.check(zk::grind_first(d.ctx(), ta.out + 16, grind_bits, ta.out + 10));
                fp.adopt_layers(d, column, layer, tail, log0, places);
            }
            const uint32_t* h = nullptr;  // one copy, one synchronisation
            d.check(zk::read_small(d.ctx(), chan, fs.len() - sync_words, &h));
            if (mid_done && (h[zk::FRI_MID_DONE] != 1u || h[zk::FRI_MID_FAILED] != 0u)) throw Error(ZKB_ETIMEOUT, "FRI: a layer's challenge did not arrive");
            const uint32_t* const state = tail_layers ? h + tail_at : h;
            HashWords dg;
            for (int k = 0; k < 8; k++) dg[k] = state[k];
            ch.set_state(dg, state[8]);
            auto root_at = [&](size_t k) {
                const uint32_t* w = k < tail ? h + 16 + 4 * tail + 8 * k : h + tail_at + zk::FRI_TAIL_ROOTS + 8 * (k - tail);
                Hash r;
                for (int i = 0; i < 8; i++) r[i] = w[i];
                return r;
            };
            fp.first_tree.root_cache = root_at(0);
            fp.first_tree.have_root = true;
            for (size_t k = 1; k < n_layers; k++) { fp.inner[k - 1].tree.root_cache = root_at(k); fp.inner[k - 1].tree.have_root = true; }
            if (last_in_tail) {
                if (state[9]) throw Error(ZKB_EINVAL, "FRI: invalid degree");
                for (size_t i = 0; i < (size_t)1 << config.log_last_layer_degree_bound; i++)
                    fp.last_layer_poly.push_back(qm31{{state[32 + 4 * i], state[33 + 4 * i], state[34 + 4 * i], state[35 + 4 * i]}});
                fp.have_nonce = grind_bits == 0 || (grind_bits > 0 && state[10] != 0xffffffffu);
                fp.nonce = grind_bits > 0 ? state[10] : 0;
                last_done = true;
            }
        } else {
            layer = SecureColumnByCoords(d, (size_t)1 << inner_log, true);
            fp.first_tree = MerkleProver::commit(d, column.refs());
            ch.mix_root(fp.first_tree.root(d));
            qm31 alpha = ch.draw_secure_felt();
            B200Backend::fold_circle_into_line(d, layer, column, alpha);
            if (inner_log != last_log) {
                for (;;) {
                    uint32_t cur_log = layer.columns[0].log_size();
                    bool last_fold = !(cur_log > last_log + config.line_fold_step);
                    uint32_t step = last_fold ? cur_log - last_log : config.line_fold_step;
                    Inner in{std::move(layer), {}, step};
                    in.tree = MerkleProver::commit(d, in.eval.refs());
                    ch.mix_root(in.tree.root(d));
                    qm31 a = ch.draw_secure_felt();
                    layer = B200Backend::fold_line(d, in.eval, a);
                    for (uint32_t s2 = 1; s2 < step; s2++) {  // backend/cpu/fri.rs:15-30
                        a = a * a;
                        layer = B200Backend::fold_line(d, layer, a);
                    }
                    fp.inner.push_back(std::move(in));
                    if (last_fold) break;
                }
            }
        }
        if (last_done) return fp;
        // commit_last_layer, fri.rs:193-221
        if (layer.len() != config.last_layer_domain_size()) throw Error(ZKB_EINVAL, "FRI: unexpected last layer size");
        std::vector<size_t> all(layer.len());
        std::iota(all.begin(), all.end(), 0);
        std::vector<qm31> coeffs = line_interpolate(secure_at_batch(d, layer, all));
        bit_reverse_vec(coeffs);
        size_t bound = (size_t)1 << config.log_last_layer_degree_bound;
        for (size_t i = bound; i < coeffs.size(); i++)
            if (!qm31_is_zero(coeffs[i])) throw Error(ZKB_EINVAL, "FRI: invalid degree");
        coeffs.resize(bound);
        bit_reverse_vec(coeffs);
        fp.last_layer_poly = coeffs;
        ch.mix_felts(fp.last_layer_poly);
        return fp;
    }

    // fri.rs:223-281, planned: `finish` is called after the plan has been executed.
    std::vector<PendingFriLayer> plan_decommit(GatherPlan& plan, const Device& d, Channel& ch, std::vector<size_t>& query_positions) const {
        uint32_t first_log = first_column->columns[0].log_size();
        query_positions = sorted_dedup(draw_queries(ch, first_log, config.n_queries));
        std::vector<PendingFriLayer> pending;
        pending.push_back(plan_fri_layer(plan, d, *first_column, first_tree, query_positions, 1));
        std::vector<size_t> q = fold_queries(query_positions, 1);
        for (auto& in : inner) {
            pending.push_back(plan_fri_layer(plan, d, in.eval, in.tree, q, in.fold_step));
            q = fold_queries(q, in.fold_step);
        }
        return pending;
    }
    FriProof finish_decommit(const GatherPlan& plan, const std::vector<PendingFriLayer>& pending) const {
        FriProof proof;
        auto layer = [&](const PendingFriLayer& pl) {
            FriLayerProof lp;
            for (size_t k = 0; k < pl.is_witness.size(); k++)
                if (pl.is_witness[k])
                    lp.fri_witness.push_back({{plan.words[pl.eval_slots[4 * k]], plan.words[pl.eval_slots[4 * k + 1]],
                                               plan.words[pl.eval_slots[4 * k + 2]], plan.words[pl.eval_slots[4 * k + 3]]}});
            lp.decommitment = pl.merkle.finish(plan).second;
            lp.commitment = pl.commitment;
            return lp;
        };
        proof.first_layer = layer(pending[0]);
        for (size_t k = 1; k < pending.size(); k++) proof.inner_layers.push_back(layer(pending[k]));
        proof.last_layer_poly = last_layer_poly;
        return proof;
    }
};

}  // namespace b200

namespace b200 {

// ------------------------------------------------------------------ commitment scheme (STWO/prover/pcs/mod.rs)
struct PcsConfig {
    uint32_t pow_bits;
    FriConfig fri;
    void mix_into(Channel& ch) const {  // STWO/core/pcs/mod.rs:47-69 (lifting_log_size None -> 0)
        qm31 f[2] = {{{pow_bits, fri.log_blowup_factor, fri.n_queries, fri.log_last_layer_degree_bound}}, {{fri.line_fold_step, 0, 0, 0}}};
        ch.mix_felts(f, 2);
    }
};

struct CommitmentTreeProver {  // pcs/mod.rs:466-630
    std::vector<BaseColumn> coeffs;  // views of the caller's columns after interpolation
    BaseColumn coeff_slab;           // host path: the one allocation the coefficient columns are views of
    std::vector<BaseColumn> evals;
    std::vector<BaseColumn> eval_slabs;  // device path: one allocation per column size, which the evals are views of
    MerkleProver commitment;
    uint32_t max_log() const { return (uint32_t)commitment.layers.size() - 1; }
};

static CirclePointQ point_add(CirclePointQ p, CirclePointQ q) {  // STWO/core/circle.rs:103-113
    return {p.x * q.x - p.y * q.y, p.x * q.y + p.y * q.x};
}
static CirclePointQ point_repeated_double(CirclePointQ p, uint32_t n) {
    for (uint32_t i = 0; i < n; i++) p = point_add(p, p);
    return p;
}
static CirclePointQ get_random_point(Channel& ch) {  // circle.rs:147-163
    qm31 t = ch.draw_secure_felt();
    qm31 t2 = t * t;
    qm31 inv = qm31_inv(t2 + qm31_one());
    return {(qm31_one() - t2) * inv, qm31_dbl(t) * inv};
}
static bool point_less(const CirclePointQ& a, const CirclePointQ& b) {
    for (int k = 0; k < 4; k++) if (a.x.c[k] != b.x.c[k]) return a.x.c[k] < b.x.c[k];
    for (int k = 0; k < 4; k++) if (a.y.c[k] != b.y.c[k]) return a.y.c[k] < b.y.c[k];
    return false;
}

// The out-of-domain sample points of all columns, flat (a segment has tens of thousands of columns, most of them with one sample at
// one of a handful of points: a vector a column is an allocation a column). Columns are numbered through the trees; column i has the
// samples first[i] ... first[i + 1] - 1, sample s is at points[point_of[s]].
struct SamplePoints {
    std::vector<CirclePointQ> points;
    std::vector<uint32_t> point_of;
    std::vector<size_t> first{0};
    uint32_t intern(const CirclePointQ& p) {
        for (size_t k = 0; k < points.size(); k++) if (points[k] == p) return (uint32_t)k;
        points.push_back(p);
        return (uint32_t)(points.size() - 1);
    }
    void end_column() { first.push_back(point_of.size()); }
};
// What is evaluated where: a group of columns of one size at one point (doubled as often as its columns are shorter than the tallest), its values one after the
// other in the value array, sample s's at place_of[s]. Made of the trees and of which points are which, not of where they are.
struct SamplePlan {
    struct Group { uint32_t log, point, doublings; size_t first, count; };
    std::vector<Group> groups;
    std::vector<uint32_t> place_of;
    std::vector<const uint32_t*> polys;
};
struct SampledValues {
    std::vector<size_t> tree_first{0};  // the trees' first columns
    std::vector<size_t> first{0};       // the columns' first values
    std::vector<qm31> values;
    const qm31* at(size_t tree, size_t column) const { return values.data() + first[tree_first[tree] + column]; }
};

struct PcsProof {
    std::vector<Hash> commitments;
    SampledValues sampled_values;
    std::vector<MerkleDecommitment> decommitments;
    std::vector<Words> queried_values;
    uint64_t proof_of_work = 0;
    FriProof fri;
    // A sink with the two vector operations the writers use, over a caller's buffer: words past the capacity are counted, not
    // written (the caller compares size() with the capacity afterwards).
    struct RawSink {
        uint32_t* out;
        size_t cap, n = 0;
        int end() const { return 0; }
        void reserve(size_t) {}
        void push_back(uint32_t v) { if (n < cap) out[n] = v; n++; }
        template <class It> void insert(int, It b, It e) {
            const size_t k = (size_t)(e - b);
            if (n + k <= cap && k) {
                if (k < LONG_RUN) memcpy(out + n, &*b, 4 * k);
                else runs.push_back({out + n, &*b, k});
            }
            n += k;
        }
        // Long runs (the queried values of a wide tree's layers; their source outlives the sink) are copied at the end, by eight threads
        // in equal parts: one core moves some 6 GB/s into fresh pages, and the proof of a composed segment is 26 MB and more.
        static constexpr size_t LONG_RUN = 4096;
        struct Run { uint32_t* dst; const uint32_t* src; size_t n; };
        std::vector<Run> runs;
        void finish() {
            size_t total = 0;
            for (auto& r : runs) total += r.n;
            parallel_chunks<8>(total, (size_t)1 << 17, [&](size_t lo, size_t hi, size_t) {
                size_t at = 0;
                for (auto& r : runs) {
                    const size_t a = std::max(lo, at), b = std::min(hi, at + r.n);
                    if (a < b) memcpy(r.dst + (a - at), r.src + (a - at), 4 * (b - a));
                    at += r.n;
                }
            });
            runs.clear();
        }
        size_t size() const { return n; }
    };
    template <class O> static void put_q(O& o, qm31 q) { o.insert(o.end(), q.c, q.c + 4); }
    template <class O> static void put_hash(O& o, const Hash& h) { o.insert(o.end(), h.begin(), h.end()); }
    template <class O> static void put_dec(O& o, const MerkleDecommitment& d) {
        o.push_back((uint32_t)d.hash_witness.size());
        for (auto& h : d.hash_witness) put_hash(o, h);
        o.push_back((uint32_t)d.column_witness.size());
        d.column_witness.append_to(o);
    }
    template <class O> static void put_layer(O& o, const FriLayerProof& l) {
        o.push_back((uint32_t)l.fri_witness.size());
        for (auto q : l.fri_witness) put_q(o, q);
        put_dec(o, l.decommitment);
        put_hash(o, l.commitment);
    }
    std::vector<uint32_t> to_words() const {
        std::vector<uint32_t> o;
        write(o);
        return o;
    }
    template <class O> void write(O& o) const {
        size_t expect = 1 << 16;
        expect += 4 * sampled_values.values.size() + 2 * sampled_values.first.size();
        for (auto& d : decommitments) expect += 8 * d.hash_witness.size() + d.column_witness.size();
        for (auto& t : queried_values) expect += t.size();
        o.reserve(expect);
        o.push_back((uint32_t)commitments.size());
        for (auto& h : commitments) put_hash(o, h);
        const SampledValues& sv = sampled_values;
        for (size_t t = 0; t + 1 < sv.tree_first.size(); t++) {
            o.push_back((uint32_t)(sv.tree_first[t + 1] - sv.tree_first[t]));
            for (size_t c = sv.tree_first[t]; c < sv.tree_first[t + 1]; c++) {
                const size_t n = sv.first[c + 1] - sv.first[c];
                o.push_back((uint32_t)n);
                if (n) o.insert(o.end(), sv.values[sv.first[c]].c, sv.values[sv.first[c]].c + 4 * n);
            }
        }
        for (auto& d : decommitments) put_dec(o, d);
        for (auto& t : queried_values) { o.push_back((uint32_t)t.size()); t.append_to(o); }
        o.push_back((uint32_t)proof_of_work);
        o.push_back((uint32_t)(proof_of_work >> 32));
        put_layer(o, fri.first_layer);
        o.push_back((uint32_t)fri.inner_layers.size());
        for (auto& l : fri.inner_layers) put_layer(o, l);
        o.push_back((uint32_t)fri.last_layer_poly.size());
        for (auto q : fri.last_layer_poly) put_q(o, q);
    }
};

struct CommitmentSchemeProver {
    const Device& d;
    PcsConfig config;
    std::vector<CommitmentTreeProver> trees;
    float* phase_ms;
    int ev = 32;  // event slots 32.. mark phase boundaries
    std::vector<std::pair<int, int>> marks;  // (phase, slot after it)

    CommitmentSchemeProver(const Device& dev, PcsConfig cfg, float* phases) : d(dev), config(cfg), phase_ms(phases) {
        if (phase_ms) { for (int i = 0; i < ZKB_PCS_N_PHASES; i++) phase_ms[i] = 0.f; mark(-1); }
    }
    void mark(int phase) {
        if (!phase_ms || ev >= 63) return;
        d.check(zkb_event_record(d.ctx(), ev));
        marks.push_back({phase, ev++});
    }
    void finish_timing() {
        if (!phase_ms) return;
        for (size_t i = 1; i < marks.size(); i++) {
            float ms = 0.f;
            d.check(zkb_event_elapsed_ms(d.ctx(), marks[i - 1].second, marks[i].second, &ms));
            if (marks[i].first >= 0) phase_ms[marks[i].first] += ms;
        }
    }

    // Trees committed one after the other with nothing drawn in between: their roots are read and mixed in at the end (mix_roots). One of
    // them ends beside the work on the next ones, the first whose short layers hold so many columns that they are a chain of
    // compressions on a handful of warps (20,000 columns of 2^11 rows: a millisecond and a half with most of the chip idle).
    struct SeveralTrees {
        bool more = true;  // trees come after this one
        bool forked = false;
    };
    static constexpr uint32_t NARROW_LOG = 13;  // the tallest such layer
    static bool narrow(const size_t (&columns)[33]) {
        size_t chain = 0;
        for (uint32_t log = 0; log <= NARROW_LOG; log++) chain += columns[log] / 16;
        return chain >= 64;  // some 55 us; a fork and its join cost a few
    }
    void mix_roots(Channel& ch) {
        zk::side_join(d.ctx());
        if (trees.size() > 1) {
            GatherPlan plan;
            for (auto& t : trees) plan.add_hash(t.commitment.layers[0].ptr());
            plan.execute(d);
            for (size_t k = 0; k < trees.size(); k++) {
                trees[k].commitment.root_cache = plan.hash_at(k);
                trees[k].commitment.have_root = true;
            }
        }
        for (auto& t : trees) ch.mix_root(t.commitment.root(d));
    }

    // TreeBuilder::extend_evals + commit (pcs/mod.rs:429-464) -> CommitmentTreeProver::new (:481-537).
    // `columns` are consumed: interpolated in place, per size group.
    // `fence_of` (optional, one entry per column) names the copy fence after which a column's values have
    // arrived from the host; columns are then interpolated and extended fence by fence, while later
    // columns are still in flight.
    void commit_evals(std::vector<BaseColumn> columns, Channel& ch, const std::vector<int>* fence_of = nullptr,
                      BaseColumn* slab = nullptr, bool are_coeffs = false, SeveralTrees* several = nullptr) {
        CommitmentTreeProver t;
        if (slab) t.coeff_slab = std::move(*slab);
        std::map<uint32_t, std::vector<size_t>> by_log;
        {
            size_t count[33] = {0};
            for (auto& c : columns) count[c.log_size()]++;
            std::vector<size_t>* of[33] = {nullptr};
            for (uint32_t log = 0; log <= 32; log++)
                if (count[log]) { of[log] = &by_log[log]; of[log]->reserve(count[log]); }
            for (size_t i = 0; i < columns.size(); i++) of[columns[i].log_size()]->push_back(i);
        }
        t.evals.resize(columns.size());
        HashColumn leaves;
        bool have_leaves = false;
        const bool hashes_later = fence_of && !columns.empty();
        if (hashes_later) {
            mark(0);
            // One column size: the leaf layer is hashed run by run (whole Blake2s blocks of 16 columns) as the
            // extended columns appear, instead of after the last one.
            const bool incremental = by_log.size() == 1 && columns.size() > 16;
            const uint32_t leaf_log = columns[0].log_size() + config.fri.log_blowup_factor;
            size_t hashed = 0, extended = 0;
            if (incremental) leaves = HashColumn(d, (size_t)8 << leaf_log);
            auto hash_ready = [&](bool final) {
                size_t avail = extended - hashed;
                size_t take = final ? avail : (avail > 16 ? (avail - 1) / 16 * 16 : 0);  // keep at least one column for the final call
                if (!take) return;
                std::vector<const uint32_t*> p;
                for (size_t c = hashed; c < hashed + take; c++) p.push_back(t.evals[c].ptr());
                d.check(zkb_merkle_leaves_partial(d.ctx(), (int)leaf_log, p.data(), (int)take, (int)hashed, (int)columns.size(), 1, leaves.ptr()));
                hashed += take;
            };
            std::map<int, std::map<uint32_t, std::vector<size_t>>> by_fence;  // fences in the order they complete
            for (size_t i = 0; i < columns.size(); i++) by_fence[(*fence_of)[i]][columns[i].log_size()].push_back(i);
            for (auto& f : by_fence) {
                d.check(zkb_wait_fence(d.ctx(), f.first));
                for (auto& g : f.second) {
                    std::vector<BaseColumn*> cols;
                    std::vector<const BaseColumn*> ccols;
                    for (auto i : g.second) { cols.push_back(&columns[i]); ccols.push_back(&columns[i]); }
                    B200Backend::interpolate_columns(d, cols);
                    auto ev_cols = B200Backend::evaluate_polynomials(d, ccols, config.fri.log_blowup_factor);
                    for (size_t k = 0; k < g.second.size(); k++) t.evals[g.second[k]] = std::move(ev_cols[k]);
                    if (incremental) { extended = g.second.back() + 1; hash_ready(false); }
                }
            }
            if (incremental) { hash_ready(true); have_leaves = true; }
        } else {
            // From the tallest columns down, each size (small ones together: commit_group) interpolated, extended and hashed before the next: a segment's short columns are tens of thousands,
            // which take the host longer to write down than the device to transform, and the device has the tall ones' hashes meanwhile.
            const uint32_t blowup = config.fri.log_blowup_factor;
            struct Size { uint32_t log; const std::vector<size_t>* of; std::vector<uint32_t*> coeffs, evals; };
            std::vector<Size> sizes;
            size_t count[33] = {0};
            for (auto g = by_log.rbegin(); g != by_log.rend(); ++g) {
                sizes.push_back({g->first, &g->second, {}, {}});
                count[g->first + blowup] = g->second.size();
            }
            MerkleBuilder builder(d, count);
            // The tables of several sizes of few columns go to the device in one copy: a copy between two kernels of a few microseconds costs as much as one. Those of the
            // extended columns go behind the interpolations, which need not wait for their allocations: three trees of 10 columns of 2^6 ... 2^4 rows 344 us with one copy for both,
            // 338 with two; of 2^7 ... 2^4 rows 397 and 393; of 40 columns of 2^9 ... 2^4 rows 642 and 635, 709 with a copy a size and table.
            auto run_end = [&](size_t first) {
                size_t end = first;
                for (size_t n = 0; end < sizes.size() && end < first + 12 && (end == first || n + sizes[end].of->size() <= 4096); end++) n += sizes[end].of->size();
                return end;
            };
            auto stage = [&](std::vector<uint32_t*> Size::*table, size_t first, size_t end) {
                std::vector<std::pair<const uint32_t* const*, size_t>> tables;
                for (size_t k = first; k < end; k++) tables.push_back({(sizes[k].*table).data(), (sizes[k].*table).size()});
                d.check(zk::stage_tables(d.ctx(), tables.data(), tables.size()));
            };
            size_t with_coeffs = 0, with_evals = 0;  // sizes whose tables are made
            auto interpolate = [&](size_t k) {
                if (k == with_coeffs) {
                    for (const size_t end = run_end(k); with_coeffs < end; with_coeffs++) {
                        Size& g = sizes[with_coeffs];
                        g.coeffs.reserve(g.of->size());
                        for (size_t c : *g.of) g.coeffs.push_back(columns[c].ptr());
                    }
                    stage(&Size::coeffs, k, with_coeffs);
                }
                if (are_coeffs) return;  // TreeBuilder::extend_polys (pcs/mod.rs:437-452): the columns are coefficients already
                d.check(zkb_ifft_cols(d.ctx(), sizes[k].coeffs.data(), (int)sizes[k].coeffs.size(), (int)sizes[k].log));
            };
            auto extend = [&](size_t k) {
                if (k == with_evals) {
                    for (const size_t end = run_end(k); with_evals < end; with_evals++) {
                        Size& g = sizes[with_evals];
                        const size_t nc = g.of->size(), stride = std::max<size_t>((size_t)1 << (g.log + blowup), 4);
                        // one allocation for the extended columns of a size (16-byte aligned each)
                        t.eval_slabs.emplace_back(d, nc * stride);
                        g.evals.resize(nc);
                        for (size_t c = 0; c < nc; c++) g.evals[c] = t.eval_slabs.back().ptr() + c * stride;
                    }
                    stage(&Size::evals, k, with_evals);
                }
                Size& g = sizes[k];
                const size_t nc = g.of->size(), n_out = (size_t)1 << (g.log + blowup);
                d.check(zkb_lde_cols(d.ctx(), g.coeffs.data(), (int)nc, (int)g.log, g.evals.data(), (int)(g.log + blowup)));
                for (size_t c = 0; c < nc; c++) t.evals[(*g.of)[c]] = BaseColumn::view(d, g.evals[c], n_out);
                builder.tree.layer_col_ptrs[g.log + blowup].assign(g.evals.begin(), g.evals.end());
            };
            if (phase_ms) {  // phase after phase, to be timed
                for (size_t k = 0; k < sizes.size(); k++) interpolate(k);
                mark(0);
                for (size_t k = 0; k < sizes.size(); k++) extend(k);
                mark(1);
                while (builder.next >= 0) builder.hash_next();
            } else {
                const bool fork = several && several->more && !several->forked && narrow(count);
                size_t stop = 0, k = 0;  // from `stop` on: on the side
                std::vector<size_t> words;
                for (const Size& g : sizes) {
                    words.push_back(g.of->size() << (g.log + blowup));
                    if (!(fork && g.log + blowup <= NARROW_LOG)) stop++;
                }
                while (k < stop) {
                    const size_t end = k + zk::commit_group(&words[k], stop - k);
                    for (size_t j = k; j < end; j++) interpolate(j);
                    for (size_t j = k; j < end; j++) extend(j);
                    for (; k < end; k++) builder.hash_to_columns();
                }
                if (k < sizes.size()) {
                    several->forked = true;
                    for (size_t j = k; j < sizes.size(); j++) interpolate(j);
                    for (size_t j = k; j < sizes.size(); j++) extend(j);
                    // so that the decommitment finds them: a table copied on the side is not there for the work outside
                    for (size_t j = k; j < sizes.size(); j++) {
                        const auto& cols = builder.tree.layer_col_ptrs[sizes[j].log + blowup];
                        d.check(zk::stage_table(d.ctx(), cols.data(), (int)cols.size()));
                    }
                    d.check(zk::side_begin(d.ctx()));
                    while (builder.next >= 0) builder.hash_next();
                    d.check(zk::side_end(d.ctx()));
                }
            }
            t.commitment = std::move(builder.tree);
        }
        t.coeffs = std::move(columns);
        if (hashes_later) {
            mark(1);
            std::vector<const BaseColumn*> refs;
            refs.reserve(t.evals.size());
            for (auto& e : t.evals) refs.push_back(&e);
            t.commitment = MerkleProver::commit(d, refs, have_leaves ? &leaves : nullptr);
        }
        if (!several) ch.mix_root(t.commitment.root(d));
        mark(2);
        trees.push_back(std::move(t));
    }

    // pcs/quotient_ops.rs:73-194 with STWO/core/pcs/quotients.rs:306-345 and :75-104: what is accumulated for which columns. It depends on
    // the columns' sizes and the sample points only, so it is made and uploaded while the samples are evaluated and hashed.
    struct Numerators {
        struct Group { uint32_t log; size_t first_col, n_cols, first_batch, n_batches; };
        std::vector<const uint32_t*> cols, coeffs;  // evaluations and coefficients, by ascending size, in their own order within a size
        std::vector<Group> groups;
        zk::NumeratorEntries entries;       // batch after batch
        std::vector<zk::NumeratorBatch> batches;
        std::vector<uint32_t> batch_point;  // of the points below
        std::vector<CirclePointQ> points;   // the sample points, then the shifted ones
        zk::NumeratorLines lines;
    };
    // place_of[s]: where sample s's value lies in the value array.
    Numerators plan_numerators(const SamplePoints& sp, const std::vector<uint32_t>& place_of, uint32_t lifting_log) const {
        Numerators nu;
        nu.points = sp.points;
        const size_t n_cols = sp.first.size() - 1;
        std::vector<const BaseColumn*> flat, flat_coeffs;
        std::vector<uint8_t> logs;
        flat.reserve(n_cols);
        flat_coeffs.reserve(n_cols);
        logs.reserve(n_cols);
        size_t first_of[34] = {0};
        for (auto& t : trees)
            for (size_t c = 0; c < t.evals.size(); c++) {
                const BaseColumn& e = t.evals[c];
                flat.push_back(&e);
                flat_coeffs.push_back(&t.coeffs[c]);
                logs.push_back((uint8_t)std::min<uint32_t>(e.log_size(), 32));
                first_of[logs.back() + 1]++;
            }
        // Entry j of the flattened list takes random_coeff^j (quotients.rs:306-345 multiplies as it goes): a column with two samples
        // has a third entry before them, its second sample at that point shifted by the column's period.
        std::vector<uint32_t> first_pow(n_cols);
        uint32_t n_pows = 0;
        for (size_t c = 0; c < n_cols; c++) {
            const size_t ns = sp.first[c + 1] - sp.first[c];
            first_pow[c] = n_pows;
            n_pows += (uint32_t)(ns + (ns == 2 ? 1 : 0));
        }
        for (int k = 1; k < 34; k++) first_of[k] += first_of[k - 1];
        std::vector<uint32_t> order(n_cols);
        for (size_t c = 0; c < n_cols; c++) order[first_of[logs[c]]++] = (uint32_t)c;
        // the shifted points: a handful of distinct (size, point) pairs
        struct Shifted { uint32_t log, from, to; };
        std::vector<Shifted> shifted;
        auto shift_of = [&](uint32_t log, uint32_t from) {
            for (auto& s : shifted) if (s.log == log && s.from == from) return s.to;
            cpoint per = host_circle_point(1u << (31 - lifting_log));  // step of CanonicCoset(lifting_log)
            for (uint32_t k = 0; k < log; k++) per = cpoint_add(per, per);
            const CirclePointQ p = point_add(nu.points[from], {qm31_from_m31(per.x), qm31_from_m31(per.y)});
            uint32_t to = 0;
            while (to < nu.points.size() && !(nu.points[to] == p)) to++;
            if (to == nu.points.size()) nu.points.push_back(p);
            shifted.push_back({log, from, to});
            return to;
        };
        // every entry's batch (a size's points in the order they come up), then the batches' entries in place
        struct Raw { uint32_t batch, col, val, pow; };
        std::vector<Raw> raw;
        raw.reserve(n_pows);
        nu.cols.reserve(n_cols);
        nu.coeffs.reserve(n_cols);
        std::vector<uint32_t> batch_of;  // per point, within the size at hand; ~0: none yet
        for (size_t i = 0; i < n_cols;) {
            const uint32_t log = logs[order[i]];
            const size_t first_col = nu.cols.size(), first_batch = nu.batches.size();
            std::fill(batch_of.begin(), batch_of.end(), ~0u);
            for (; i < n_cols && logs[order[i]] == log; i++) {
                const uint32_t c = order[i];
                const uint32_t col = (uint32_t)(nu.cols.size() - first_col);
                nu.cols.push_back(flat[c]->ptr());
                nu.coeffs.push_back(flat_coeffs[c]->ptr());
                uint32_t pow = first_pow[c];
                auto entry = [&](uint32_t point, size_t sample) {
                    if (point >= batch_of.size()) batch_of.resize(point + 1, ~0u);
                    if (batch_of[point] == ~0u) {
                        batch_of[point] = (uint32_t)nu.batches.size();
                        nu.batches.push_back({nu.points[point].y, 0, 0, qm31_zero(), qm31_zero()});
                        nu.batch_point.push_back(point);
                    }
                    nu.batches[batch_of[point]].count++;
                    raw.push_back({batch_of[point], col, place_of[sample], pow++});
                };
                const size_t s0 = sp.first[c], s1 = sp.first[c + 1];
                if (s1 - s0 == 2) entry(shift_of(log, sp.point_of[s0 + 1]), s0 + 1);
                for (size_t s = s0; s < s1; s++) entry(sp.point_of[s], s);
            }
            nu.groups.push_back({log, first_col, nu.cols.size() - first_col, first_batch, nu.batches.size() - first_batch});
        }
        std::vector<size_t> at(nu.batches.size());
        size_t n = 0;
        for (size_t b = 0; b < at.size(); b++) { nu.batches[b].first = at[b] = n; n += nu.batches[b].count; }
        nu.entries.col.resize(n);
        nu.entries.val.resize(n);
        nu.entries.pow.resize(n);
        for (auto& r : raw) {
            const size_t k = at[r.batch]++;
            nu.entries.col[k] = r.col;
            nu.entries.val[k] = r.val;
            nu.entries.pow[k] = r.pow;
        }
        return nu;
    }

    SecureColumnByCoords compute_fri_quotients(Numerators& nu, qm31 random_coeff, const qm31* h_values, const uint32_t* d_values, uint32_t lifting_log) {
        std::unique_ptr<HostClock> hc(new HostClock("pcs.quot.lines"));
        d.check(zk::numerator_lines(d.ctx(), nu.entries, nu.batches, nu.lines, random_coeff, h_values, d_values));
        hc.reset(new HostClock("pcs.quot.numerators"));
        std::vector<AccumulatedNumerators> accs;
        for (auto& g : nu.groups)
            for (size_t b = g.first_batch; b < g.first_batch + g.n_batches; b++) {
                SecureColumnByCoords acc(d, (size_t)1 << g.log);
                auto o = acc.ptrs();
                d.check(zk::numerator_run(d.ctx(), nu.cols.data() + g.first_col, nu.coeffs.data() + g.first_col, (int)g.n_cols, (int)g.log,
                                          (int)(g.log - config.fri.log_blowup_factor), nu.lines, nu.batches[b], o.data()));
                accs.push_back({nu.points[nu.batch_point[b]], std::move(acc), nu.batches[b].first_linear});
            }
        hc.reset(new HostClock("pcs.quot.combine"));
        std::stable_sort(accs.begin(), accs.end(),
                         [](const AccumulatedNumerators& a, const AccumulatedNumerators& b) { return point_less(a.sample_point, b.sample_point); });
        std::vector<AccumulatedNumerators> per_point;
        for (size_t i = 0; i < accs.size();) {
            size_t j = i;
            while (j < accs.size() && accs[j].sample_point == accs[i].sample_point) j++;
            qm31 first = qm31_zero();
            std::vector<SecureColumnByCoords> cols;
            for (size_t k = i; k < j; k++) {
                first = first + accs[k].first_linear_term_acc;
                cols.push_back(std::move(accs[k].partial_numerators_acc));
            }
            CirclePointQ pt = accs[i].sample_point;
            per_point.push_back({pt, B200Backend::lift_and_accumulate(d, std::move(cols)), first});
            i = j;
        }
        return B200Backend::compute_quotients_and_combine(d, per_point, lifting_log);
    }

    // batch out-of-domain evaluation: one call per (coefficient size, transformed point) group (pcs/mod.rs:187-265)
    SamplePlan plan_samples(const SamplePoints& sp, size_t n_points) const {
        HostClock hc("pcs.sample.group");
        // Every column is lifted to the height of the LAST tree (pcs/mod.rs:180: in a proof it is the composition tree, which
        // is the tallest); a taller column in an earlier tree has no lift.
        const uint32_t lifting_log = trees.back().max_log();
        for (auto& t : trees)
            if (!t.evals.empty() && t.max_log() > lifting_log)
                throw Error(ZKB_EINVAL, "pcs: the last tree must hold the tallest column (every column is lifted to its height)");
        SamplePlan plan;
        const size_t n_samples = sp.point_of.size();
        std::vector<int> group_of(n_points * 64, -1);  // by (point, doublings)
        std::vector<uint32_t> sample_group(n_samples);
        plan.place_of.resize(n_samples);
        plan.polys.resize(n_samples);
        size_t flat = 0;
        for (auto& t : trees)
            for (size_t c = 0; c < t.coeffs.size(); c++, flat++) {
                const uint32_t shift = lifting_log - t.evals[c].log_size();
                for (size_t s = sp.first[flat]; s < sp.first[flat + 1]; s++) {
                    int& g = group_of[sp.point_of[s] * 64 + shift];
                    if (g < 0) {
                        g = (int)plan.groups.size();
                        plan.groups.push_back({t.coeffs[c].log_size(), sp.point_of[s], shift, 0, 0});
                    }
                    sample_group[s] = (uint32_t)g;
                    plan.groups[g].count++;
                }
            }
        size_t at = 0;
        for (auto& g : plan.groups) { g.first = at; at += g.count; g.count = 0; }
        flat = 0;
        for (auto& t : trees)
            for (size_t c = 0; c < t.coeffs.size(); c++, flat++)
                for (size_t s = sp.first[flat]; s < sp.first[flat + 1]; s++) {
                    SamplePlan::Group& g = plan.groups[sample_group[s]];
                    plan.place_of[s] = (uint32_t)(g.first + g.count);
                    plan.polys[g.first + g.count++] = t.coeffs[c].ptr();
                }
        return plan;
    }

    // pcs/mod.rs:168-419
    PcsProof prove_values(SamplePoints sp, const SamplePlan& sample_plan, Channel& ch) {
        PcsProof proof;
        const uint32_t lifting_log = trees.back().max_log();
        const size_t n_samples = sp.point_of.size();
        const std::vector<uint32_t>& place_of = sample_plan.place_of;
        for (auto& t : trees) proof.sampled_values.tree_first.push_back(proof.sampled_values.tree_first.back() + t.coeffs.size());
        // The quotient plan of tens of thousands of samples takes as long as hashing them does: it is made on another thread meanwhile.
        const bool aside = n_samples >= 8192;
        std::future<Numerators> planned;
        if (aside) planned = std::async(std::launch::async, [&] { return plan_numerators(sp, place_of, lifting_log); });
        std::unique_ptr<HostClock> hc(new HostClock("pcs.sample.eval"));
        BaseColumn d_values(d, 4 * n_samples);
        for (auto& g : sample_plan.groups) {
            const CirclePointQ p = point_repeated_double(sp.points[g.point], g.doublings);
            uint32_t pt[8];
            memcpy(pt, p.x.c, 16);
            memcpy(pt + 4, p.y.c, 16);
            d.check(zk::eval_at_point_device(d.ctx(), sample_plan.polys.data() + g.first, (int)g.count, (int)g.log, pt, d_values.ptr() + 4 * g.first));
        }
        hc.reset(new HostClock("pcs.quot.plan"));
        Numerators nu;
        BaseColumn lines_block;
        auto stage = [&] {
            d.check(zk::numerator_stage(d.ctx(), nu.entries, nu.batches, nu.lines));
            lines_block = BaseColumn::adopt(d, nu.lines.block);
        };
        if (!aside) {
            nu = plan_numerators(sp, place_of, lifting_log);
            stage();
        }
        hc.reset(new HostClock("pcs.sample.read"));
        qm31* h_values = reinterpret_cast<qm31*>(GatherPlan::arena(4 * n_samples));
        if (n_samples) d.check(zkb_d2h(d.ctx(), h_values, d_values.ptr(), 16 * n_samples));
        std::vector<qm31>& values = proof.sampled_values.values;
        values.resize(n_samples);
        for (size_t s = 0; s < n_samples; s++) values[s] = h_values[place_of[s]];
        mark(3);
        hc.reset(new HostClock("pcs.quot.mix"));
        ch.mix_felts(values);
        qm31 random_coeff = ch.draw_secure_felt();
        if (aside) {
            nu = planned.get();
            stage();
        }
        hc.reset(new HostClock("pcs.quot.compute"));
        SecureColumnByCoords quotients = compute_fri_quotients(nu, random_coeff, h_values, d_values.ptr(), lifting_log);
        proof.sampled_values.first = std::move(sp.first);
        hc.reset();
        mark(4);
        FriProver fri = FriProver::commit(d, ch, config.fri, quotients, (int)config.pow_bits);
        mark(5);
        proof.proof_of_work = fri.have_nonce ? fri.nonce : B200Backend::grind(d, ch.pow_prefixed_digest(config.pow_bits), config.pow_bits);
        ch.mix_u64(proof.proof_of_work);
        mark(6);
        hc.reset(new HostClock("pcs.decommit.plan"));
        std::vector<size_t> query_positions;
        GatherPlan plan;
        std::unique_ptr<HostClock> hc2(new HostClock("pcs.decommit.plan.fri"));
        auto fri_pending = fri.plan_decommit(plan, d, ch, query_positions);
        hc2.reset(new HostClock("pcs.decommit.plan.trees"));
        std::vector<PendingMerkle> tree_pending;
        for (auto& t : trees) {  // STWO/core/pcs/utils.rs:200-218, then pcs/mod.rs:575-630
            const uint32_t tree_max = t.max_log();
            std::vector<size_t> of_log;
            tree_pending.push_back(t.commitment.plan_decommit(plan, [&](uint32_t log) -> const std::vector<size_t>& {
                of_log.clear();
                if (log >= t.commitment.layer_col_ptrs.size() || t.commitment.layer_col_ptrs[log].empty()) return of_log;
                for (auto pos : query_positions) {
                    const size_t q = ((pos >> (lifting_log - tree_max + 1)) << 1) + (pos & 1);
                    of_log.push_back(((q >> (tree_max - log + 1)) << 1) + (q & 1));
                }
                of_log = sorted_dedup(std::move(of_log));
                return of_log;
            }));
        }
        hc2.reset();
        hc.reset(new HostClock("pcs.decommit.gather"));
        plan.execute(d);
        hc.reset(new HostClock("pcs.decommit.finish"));
        proof.fri = fri.finish_decommit(plan, fri_pending);
        for (size_t k = 0; k < trees.size(); k++) {
            auto r = tree_pending[k].finish(plan);
            proof.queried_values.push_back(std::move(r.first));
            proof.decommitments.push_back(std::move(r.second));
            proof.commitments.push_back(trees[k].commitment.root(d));
        }
        hc.reset();
        mark(7);
        return proof;
    }
};

// ------------------------------------------------------------------ GKR (STWO/prover/lookups)
// Dense univariate polynomial over QM31, low coefficient first (lookups/utils.rs:12-146).
struct UniPoly {
    std::vector<qm31> c;
    void trim() { while (!c.empty() && qm31_is_zero(c.back())) c.pop_back(); }
    qm31 eval(qm31 x) const {
        qm31 acc = qm31_zero();
        for (size_t i = c.size(); i-- > 0;) acc = acc * x + c[i];
        return acc;
    }
    static UniPoly mul(UniPoly a, UniPoly b) {
        a.trim(); b.trim();
        if (a.c.empty() || b.c.empty()) return {};
        UniPoly r;
        r.c.assign(a.c.size() + b.c.size() - 1, qm31_zero());
        for (size_t i = 0; i < a.c.size(); i++)
            for (size_t j = 0; j < b.c.size(); j++) r.c[i + j] = r.c[i + j] + a.c[i] * b.c[j];
        r.trim();
        return r;
    }
    static UniPoly add(const UniPoly& a, const UniPoly& b) {
        UniPoly r;
        for (size_t i = 0; i < std::max(a.c.size(), b.c.size()); i++)
            r.c.push_back((i < a.c.size() ? a.c[i] : qm31_zero()) + (i < b.c.size() ? b.c[i] : qm31_zero()));
        return r;
    }
    static UniPoly interpolate_lagrange(const std::vector<qm31>& xs, const std::vector<qm31>& ys) {  // utils.rs:26-54
        UniPoly coeffs;
        for (size_t i = 0; i < xs.size(); i++) {
            qm31 prod = ys[i];
            for (size_t j = 0; j < xs.size(); j++)
                if (i != j) prod = prod * qm31_inv(xs[i] - xs[j]);
            UniPoly term;
            term.c = {prod};
            term.trim();
            for (size_t j = 0; j < xs.size(); j++)
                if (i != j) { UniPoly lin; lin.c = {qm31_neg(xs[j]), qm31_one()}; term = mul(term, lin); }
            coeffs = add(coeffs, term);
        }
        coeffs.trim();
        return coeffs;
    }
};

static qm31 eq1(qm31 x, qm31 y) { return x * y + (qm31_one() - x) * (qm31_one() - y); }  // utils.rs:165-170

// correct_sum_as_poly_in_first_variable (gkr_prover.rs:884-923), split in two.
// The part that depends only on the out-of-domain point y and on the number of
// variables k: every oracle that is active in a round shares it, so it is worked out once per round (two inversions and
// the Lagrange basis on {0, 1, 2, b}) instead of once per instance (a batch has hundreds). The round polynomial of an
// oracle is then r0 L0 + r1 L1 + r2 L2 (the value at b is zero), the same field elements as the interpolation gives.
struct RoundBasis {
    qm31 e0a, e2a;   // eq(0, y[n-k]) / prod_{i <= n-k} eq(0, y_i) and eq(2, y[n-k]) / the same product
    qm31 L[3][4];    // coefficients (low first) of the basis polynomials of the nodes 0, 1, 2
    RoundBasis() = default;
    RoundBasis(const std::vector<qm31>& y, size_t k) {
        size_t n = y.size();
        qm31 a = qm31_one();
        for (size_t i = 0; i < n - k + 1; i++) a = a * eq1(qm31_zero(), y[i]);
        a = qm31_inv(a);
        qm31 two = qm31_from_m31(2);
        qm31 b = (qm31_one() - y[n - k]) * qm31_inv(qm31_one() - qm31_dbl(y[n - k]));
        e0a = eq1(qm31_zero(), y[n - k]) * a;
        e2a = eq1(two, y[n - k]) * a;
        const qm31 xs[4] = {qm31_zero(), qm31_one(), two, b};
        for (int i = 0; i < 3; i++) {
            qm31 denom = qm31_one();
            qm31 poly[4] = {qm31_one(), qm31_zero(), qm31_zero(), qm31_zero()};
            int deg = 0;
            for (int j = 0; j < 4; j++) {
                if (j == i) continue;
                denom = denom * (xs[i] - xs[j]);
                for (int t = ++deg; t > 0; t--) poly[t] = poly[t - 1] - xs[j] * poly[t];  // times (x - xs[j])
                poly[0] = qm31_neg(xs[j] * poly[0]);
            }
            qm31 inv = qm31_inv(denom);
            for (int t = 0; t < 4; t++) L[i][t] = poly[t] * inv;
        }
    }
    // the polynomial with the values r0, r1, r2 at 0, 1, 2 and zero at b
    UniPoly round_poly(qm31 r0, qm31 r1, qm31 r2) const {
        UniPoly p;
        p.c.resize(4);
        for (int t = 0; t < 4; t++) p.c[t] = r0 * L[0][t] + r1 * L[1][t] + r2 * L[2][t];
        p.trim();
        return p;
    }
};

static Layer layer_view(const Device& d, int kind, const uint32_t* num, const uint32_t* den, size_t n) {
    Layer l;
    l.kind = kind;
    l.den.words = BaseColumn::view(d, const_cast<uint32_t*>(den), 4 * n);
    if (kind == ZKB_GKR_LOGUP_GENERIC) l.num.words = BaseColumn::view(d, const_cast<uint32_t*>(num), 4 * n);
    if (kind == ZKB_GKR_LOGUP_MULTIPLICITIES) l.num_base = BaseColumn::view(d, const_cast<uint32_t*>(num), n);
    return l;
}

// The bases of a layer's rounds (variables left: nv, nv - 1 ... 1) with one inversion for all of them. With y the round's
// coordinate and u = 1 - 2y, b = (1 - y) / u, and the denominators of the basis polynomials are -2 (1 - y) / u, y / u and
// 2 (1 - 3y) / u: 0.5 us a round, where five inversions each took 2.3 us with the device waiting.
static std::vector<RoundBasis> round_bases(const std::vector<qm31>& y, size_t nv) {
    std::vector<RoundBasis> out(nv);
    const qm31 one = qm31_one(), three = qm31_from_m31(3);
    const size_t first = y.size() - nv;
    std::vector<qm31> v(4 * nv + 1), inv(4 * nv + 1);  // u, 1 - y, y, 1 - 3y of every round; the product over the coordinates before
    qm31 before = one;
    for (size_t i = 0; i < first; i++) before = before * (one - y[i]);
    v[4 * nv] = before;
    for (size_t r = 0; r < nv; r++) {
        const qm31 c = y[first + r];
        v[4 * r] = one - qm31_dbl(c);
        v[4 * r + 1] = one - c;
        v[4 * r + 2] = c;
        v[4 * r + 3] = one - three * c;
    }
    qm31 acc = one;
    for (size_t i = 0; i < v.size(); i++) { inv[i] = acc; acc = acc * v[i]; }
    if (qm31_is_zero(acc)) {  // a coordinate is 0, 1, 1/2 or 1/3
        for (size_t r = 0; r < nv; r++) out[r] = RoundBasis(y, nv - r);
        return out;
    }
    acc = qm31_inv(acc);
    for (size_t i = v.size(); i-- > 0;) { inv[i] = inv[i] * acc; acc = acc * v[i]; }
    const uint32_t half = m31_inv(2);
    qm31 a = inv[4 * nv];  // 1 / the product of 1 - y over the coordinates so far
    for (size_t r = 0; r < nv; r++) {
        RoundBasis& o = out[r];
        const qm31 c = v[4 * r + 2], u = v[4 * r], b = v[4 * r + 1] * inv[4 * r], b2 = qm31_dbl(b), b3 = b2 + b;
        o.e0a = a;
        a = a * inv[4 * r + 1];
        o.e2a = (three * c - one) * a;
        const qm31 i0 = qm31_neg(qm31_mul_m31(u * inv[4 * r + 1], half)), i1 = u * inv[4 * r + 2], i2 = qm31_mul_m31(u * inv[4 * r + 3], half);
        const qm31 two = qm31_from_m31(2);
        o.L[0][0] = qm31_neg(b2) * i0; o.L[0][1] = (two + b3) * i0; o.L[0][2] = qm31_neg(three + b) * i0; o.L[0][3] = i0;
        o.L[1][0] = qm31_zero();       o.L[1][1] = b2 * i1;         o.L[1][2] = qm31_neg(two + b) * i1;   o.L[1][3] = i1;
        o.L[2][0] = qm31_zero();       o.L[2][1] = b * i2;          o.L[2][2] = qm31_neg(one + b) * i2;   o.L[2][3] = i2;
    }
    return out;
}

// The sum-check of a layer with the transcript on the host, a launch a round: table j of the plan gives the sums of round j (of the layers
// fixed with the challenge before, and of the oracles that enter), the last table the masks (GKR_LAYER_MASK_WORDS per oracle).
static void host_rounds(const Device& d, Channel& ch, zk::GkrLayerPlan& plan, qm31 alpha, qm31 lambda, const std::vector<qm31>& ood_point, const SecureMle& eq_evals,
                        std::vector<qm31>& sc_claims, std::vector<UniPoly>& round_polys, std::vector<qm31>& assignment, std::vector<uint32_t>& mask_words) {
    const size_t K = plan.n_vars.size();
    const int nv = plan.n_rounds;
    const uint32_t half = m31_inv(2);
    std::vector<uint32_t> results;
    std::vector<qm31> rv(3 * K), corr(K, qm31_one());
    std::vector<std::pair<qm31, qm31>> sums(K);
    mask_words.assign(zk::GKR_LAYER_MASK_WORDS * K, 0u);
    auto q_at = [](const uint32_t* w) { return qm31{{w[0], w[1], w[2], w[3]}}; };
    qm31 challenge = qm31_zero();
    for (int round = 0; round <= nv; round++) {
        zk::GkrBatchItem* items = plan.items.data() + plan.table_at[round];
        const size_t n_items = plan.table_at[round + 1] - plan.table_at[round];
        {
            HostClock hc("gkr.round.launch_wait");
            results.resize(n_items * zk::GKR_BATCH_RESULT_WORDS);
            d.check(zk::gkr_batch_round(d.ctx(), items, (int)n_items, challenge.c, eq_evals.words.ptr(), lambda.c, results.data()));
        }
        for (size_t j = 0; j < n_items; j++) {
            const uint32_t* w = results.data() + j * zk::GKR_BATCH_RESULT_WORDS;
            const size_t k = (size_t)items[j].slot;
            if (items[j].mode == 2) memcpy(&mask_words[zk::GKR_LAYER_MASK_WORDS * k], w + 8, 64);
            else sums[k] = {q_at(w), q_at(w + 4)};
        }
        if (round == nv) break;
        // Every active oracle has n_rem variables left, so all their round polynomials are r0 L0 + r1 L1 + r2 L2 over the
        // same basis, and the random linear combination over the batch (sumcheck.rs:139-149, Horner in alpha from the
        // last oracle down) is (sum alpha^k r0_k) L0 + (sum alpha^k r1_k) L1 + (sum alpha^k r2_k) L2 plus the constants of
        // the oracles that wait: eleven multiplications per oracle and round instead of a Lagrange interpolation each.
        // r0 + r1 is the claim by construction, which is the check sumcheck.rs:128-130 makes.
        HostClock hc("gkr.round.algebra");
        const size_t n_rem = (size_t)(nv - round);
        const RoundBasis basis(ood_point, n_rem);
        auto act = [&](size_t k) { return n_rem <= plan.n_vars[k]; };
        qm31 S[3] = {qm31_zero(), qm31_zero(), qm31_zero()}, Sc = qm31_zero();
        for (size_t k = K; k-- > 0;) {
            for (int t = 0; t < 3; t++) S[t] = S[t] * alpha;
            Sc = Sc * alpha;
            if (act(k)) {
                rv[3 * k] = sums[k].first * corr[k] * basis.e0a;
                rv[3 * k + 1] = sc_claims[k] - rv[3 * k];
                rv[3 * k + 2] = sums[k].second * corr[k] * basis.e2a;
                for (int t = 0; t < 3; t++) S[t] = S[t] + rv[3 * k + t];
            } else {
                rv[3 * k] = qm31_mul_m31(sc_claims[k], half);
                Sc = Sc + rv[3 * k];
            }
        }
        UniPoly combined;
        combined.c.resize(4);
        for (int t = 0; t < 4; t++) combined.c[t] = S[0] * basis.L[0][t] + S[1] * basis.L[1][t] + S[2] * basis.L[2][t];
        combined.c[0] = combined.c[0] + Sc;
        if (qm31_is_zero(combined.c[3])) {
            // The combination keeps the length of its longest term. A vanishing leading coefficient does not say which
            // case this is (every term short, or a cancellation), so this round goes term by term.
            combined = UniPoly();
            for (size_t k = K; k-- > 0;) {
                UniPoly rp;
                if (act(k)) rp = basis.round_poly(rv[3 * k], rv[3 * k + 1], rv[3 * k + 2]);
                else { rp.c = {rv[3 * k]}; rp.trim(); }
                for (auto& c : combined.c) c = c * alpha;
                combined = UniPoly::add(combined, rp);
            }
        }
        ch.mix_felts(combined.c);
        challenge = ch.draw_secure_felt();
        qm31 Lc[3];
        for (int t = 0; t < 3; t++) Lc[t] = ((basis.L[t][3] * challenge + basis.L[t][2]) * challenge + basis.L[t][1]) * challenge + basis.L[t][0];
        const qm31 eq_step = eq1(challenge, ood_point[ood_point.size() - n_rem]);  // the same for every active oracle
        for (size_t k = 0; k < K; k++) {
            if (act(k)) {
                sc_claims[k] = rv[3 * k] * Lc[0] + rv[3 * k + 1] * Lc[1] + rv[3 * k + 2] * Lc[2];
                corr[k] = corr[k] * eq_step;
            } else sc_claims[k] = rv[3 * k];
        }
        round_polys.push_back(std::move(combined));
        assignment.push_back(challenge);
    }
}

// An instance of a batch: the input and the layers above it. Level 0 is the input, level l has 2^(log - l) entries; the levels from
// 1 on lie one after the other. A round fixes a level in place (a thread of the fixing kernel reads entries i and i + n/2 and
// writes entry i, and no other thread touches either), but the input, which is the caller's, into the fold arrays.
struct BatchTower {
    int kind, log;
    const uint32_t *num, *den;
    uint32_t *num_levels, *den_levels, *num_fold, *den_fold;  // numerators: null where the kind has none
    int kind_at(int level) const { return level == 0 || kind == ZKB_GKR_GRAND_PRODUCT ? kind : ZKB_GKR_LOGUP_GENERIC; }
    size_t offset(int level) const { return 4 * (((size_t)1 << log) - ((size_t)1 << (log - level + 1))); }
};

// The tables of one layer's sum-check (gkr_batch.hpp). Every oracle is level `level` of its instance's tower: those of at least
// level + 1 levels take part, inst[k] is oracle k's.
static void plan_layer(const std::vector<BatchTower>& towers, int level, int n_rounds, zk::GkrLayerPlan& plan, std::vector<size_t>& inst) {
    inst.clear();
    plan.n_rounds = n_rounds;
    plan.n_vars.clear();
    plan.items.clear();
    plan.table_at.clear();
    for (size_t i = 0; i < towers.size(); i++)
        if (towers[i].log > level) {
            inst.push_back(i);
            plan.n_vars.push_back((uint32_t)(towers[i].log - level - 1));
        }
    if (!n_rounds) return;
    // round q fixes a layer of 2^(n_rounds - q + 1) entries
    for (int j = 0; j <= n_rounds; j++) {
        plan.table_at.push_back(plan.items.size());
        for (int fix = 1; fix >= 0; fix--) {
            const int round = fix ? j - 1 : j;
            if (round < 0 || round == n_rounds) continue;
            const uint32_t n_rem = (uint32_t)(n_rounds - round);
            for (size_t k = 0; k < inst.size(); k++) {
                const bool enters = plan.n_vars[k] == n_rem;
                if (fix ? plan.n_vars[k] < n_rem : !enters) continue;
                const BatchTower& t = towers[inst[k]];
                zk::GkrBatchItem it{};
                it.n = (unsigned long long)2 << n_rem;
                it.kind = (uint32_t)t.kind_at(level);
                it.mode = !fix ? 0u : it.n >= 8 ? 1u : 2u;
                it.slot = k;
                const bool num = it.kind == ZKB_GKR_LOGUP_GENERIC || it.kind == ZKB_GKR_LOGUP_MULTIPLICITIES;
                if (level) {
                    it.den = it.den_out = t.den_levels + t.offset(level);
                    if (num) it.num = it.num_out = t.num_levels + t.offset(level);
                } else {
                    it.den_out = t.den_fold;
                    it.den = enters ? t.den : t.den_fold;
                    if (num) { it.num_out = t.num_fold; it.num = enters ? t.num : t.num_fold; }
                    if (it.kind == ZKB_GKR_LOGUP_MULTIPLICITIES && !enters) it.kind = ZKB_GKR_LOGUP_GENERIC;
                }
                plan.items.push_back(it);
            }
        }
    }
    plan.table_at.push_back(plan.items.size());
}

// gkr_prover.rs:657-882 with sumcheck.rs:96-176. Returns the proof word stream.
static std::vector<uint32_t> gkr_prove_batch(const Device& d, Channel& ch, const std::vector<Layer>& input_layers) {
    const size_t n_inst = input_layers.size();
    std::unique_ptr<HostClock> hc(new HostClock("gkr.towers"));
    std::vector<BatchTower> towers(n_inst);  // gen_layers, :847-852
    int n_layers = 0;
    BaseColumn slab;
    for (int pass = 0; pass < 2; pass++) {  // one allocation for all towers and fold arrays: its size, then the places
        size_t words = 0;
        auto take = [&](size_t n) { uint32_t* p = pass ? slab.ptr() + words : nullptr; words += n; return p; };
        for (size_t i = 0; i < n_inst; i++) {
            const Layer& in = input_layers[i];
            BatchTower& t = towers[i];
            t = {in.kind, (int)in.n_variables(), in.num_ptr(), in.den.words.ptr(), nullptr, nullptr, nullptr, nullptr};
            n_layers = std::max(n_layers, t.log);
            if (!t.log) continue;
            const size_t n = in.len();
            t.den_levels = take(4 * (n - 1));
            t.den_fold = take(2 * n);
            if (t.kind != ZKB_GKR_GRAND_PRODUCT) t.num_levels = take(4 * (n - 1));
            if (t.num) t.num_fold = take(2 * n);
        }
        if (!pass && words) slab = BaseColumn(d, words);
    }
    std::vector<zk::GkrBatchItem> items;
    std::vector<size_t> top_of(n_inst, 0);
    for (size_t i = 0; i < n_inst; i++) {
        const BatchTower& t = towers[i];
        if (!t.log) continue;
        top_of[i] = zk::GKR_TOP_WORDS * items.size();
        zk::GkrBatchItem it{};
        it.num = t.num;
        it.den = t.den;
        it.num_out = t.num_levels;
        it.den_out = t.den_levels;
        it.n = (unsigned long long)1 << t.log;
        it.kind = (uint32_t)t.kind;
        items.push_back(it);
    }
    std::vector<uint32_t> tops(zk::GKR_TOP_WORDS * items.size()), results;
    if (!items.empty()) d.check(zk::gkr_batch_towers(d.ctx(), items.data(), (int)items.size(), tops.data()));
    hc.reset();
    auto q_at = [](const uint32_t* w) { return qm31{{w[0], w[1], w[2], w[3]}}; };

    // claims and masks: num, den of a fraction (2 columns), or the product (1); column c of a mask is (v[2c], v[2c+1])
    struct Claim { uint32_t n_cols = 0; qm31 v[2]; };
    struct MaskRec { uint32_t n_cols; qm31 v[4]; };
    std::vector<std::vector<UniPoly>> sumcheck_round_polys;
    std::vector<std::vector<MaskRec>> masks_by_inst(n_inst);
    for (size_t i = 0; i < n_inst; i++) masks_by_inst[i].reserve((size_t)towers[i].log);
    std::vector<Claim> output_claims(n_inst), claims(n_inst);
    std::vector<qm31> ood_point;

    // Whether the transcript of a layer's rounds stays on the device (gkr_batch_layer_begin; ZKB_GKR_ROUNDS=host: never;
    // ZKB_GKR_ROUNDS=launches: with a launch per round and step instead of one for the layer; =refused: the same, as though the one launch had
    // been refused). The layer's
    // description is staged as one block (an item per oracle and active round, 64 bytes each, and some 52 bytes per oracle): a batch of
    // thousands of tall instances would not fit the staging ring and takes the round-by-round path, which stages one round's items at a time.
    const char* rounds_env = getenv("ZKB_GKR_ROUNDS");
    const bool never = rounds_env && !strcmp(rounds_env, "host");
    auto on_device = [&](const zk::GkrLayerPlan& p) {
        return !never && p.n_rounds > 0 && p.n_rounds <= zk::GKR_LAYER_MAX_ROUNDS &&
               64 * p.items.size() + 64 * p.n_vars.size() + 256 * (size_t)p.n_rounds + 8192 <= ((size_t)2 << 20);
    };
    // A layer's tables depend on the towers' sizes only: they are made and staged while the layer before runs.
    zk::GkrLayerPlan plan, next_plan;
    plan.launches = next_plan.launches = rounds_env && !strcmp(rounds_env, "launches");
    plan.refused = next_plan.refused = rounds_env && !strcmp(rounds_env, "refused");
    std::vector<size_t> inst, next_inst;
    auto make_next = [&](int layer) {
        HostClock hc_plan("gkr.layer.plan");
        plan_layer(towers, n_layers - layer - 1, layer, next_plan, next_inst);
        if (on_device(next_plan)) d.check(zk::gkr_batch_plan(d.ctx(), next_plan));
    };
    if (n_layers) make_next(0);
    std::vector<qm31> alpha_pow, sc_claims;
    std::vector<zk::GkrRoundConst> consts;
    std::vector<uint32_t> mask_words;
    for (int layer = 0; layer < n_layers; layer++) {
        std::swap(plan, next_plan);
        std::swap(inst, next_inst);
        const int n_remaining = n_layers - layer, level = n_remaining - 1, nv = layer;
        const size_t K = inst.size();
        // EqEvals::generate, :235-247
        hc.reset(new HostClock("gkr.layer.eq_evals"));
        SecureMle eq_evals;
        bool have_eq = false;
        auto make_eq = [&] {
            if (ood_point.empty()) eq_evals = B200Backend::gen_eq_evals(d, {}, qm31_one());
            else eq_evals = B200Backend::gen_eq_evals(d, std::vector<qm31>(ood_point.begin() + 1, ood_point.end()), eq1(qm31_zero(), ood_point[0]));
            have_eq = true;
        };
        if (on_device(plan) ? plan.needs_eq : nv > 0) make_eq();
        hc.reset(new HostClock("gkr.layer.claims"));
        for (size_t i : inst) {
            if (towers[i].log == n_remaining) {  // its output layer: one entry per column
                const uint32_t* w = tops.data() + top_of[i];
                Claim& c = claims[i];
                if (towers[i].kind == ZKB_GKR_GRAND_PRODUCT) { c.n_cols = 1; c.v[0] = q_at(w); }
                else { c.n_cols = 2; c.v[0] = q_at(w + 4); c.v[1] = q_at(w); }
                output_claims[i] = c;
            }
            ch.mix_felts(claims[i].v, claims[i].n_cols);
        }
        const qm31 sumcheck_alpha = ch.draw_secure_felt();
        const qm31 lambda = ch.draw_secure_felt();
        alpha_pow.resize(K);
        sc_claims.resize(K);
        for (size_t k = 0; k < K; k++) {
            const Claim& c = claims[inst[k]];
            alpha_pow[k] = k ? alpha_pow[k - 1] * sumcheck_alpha : qm31_one();
            sc_claims[k] = qm31_mul_m31(c.n_cols == 1 ? c.v[0] : c.v[0] + lambda * c.v[1], 1u << (nv - (int)plan.n_vars[k]));
        }
        std::vector<UniPoly> round_polys;
        std::vector<qm31> assignment;
        const uint32_t* masks_at = nullptr;  // GKR_LAYER_MASK_WORDS per oracle that had a round
        if (on_device(plan)) {
            hc.reset(new HostClock("gkr.layer.begin"));
            consts.resize((size_t)nv);
            const std::vector<RoundBasis> bases = round_bases(ood_point, (size_t)nv);
            for (int round = 0; round < nv; round++) {
                const size_t n_rem = (size_t)(nv - round);
                const RoundBasis& basis = bases[round];
                zk::GkrRoundConst& rc = consts[round];
                memset(&rc, 0, sizeof(rc));
                memcpy(rc.e0a, basis.e0a.c, 16);
                memcpy(rc.e2a, basis.e2a.c, 16);
                for (int i = 0; i < 3; i++)
                    for (int t = 0; t < 4; t++) memcpy(rc.L[i][t], basis.L[i][t].c, 16);
                memcpy(rc.y, ood_point[ood_point.size() - n_rem].c, 16);
                rc.n_rem = (uint32_t)n_rem;
            }
            uint32_t chan[9];
            memcpy(chan, ch.digest().data(), 32);
            chan[8] = ch.n_draws();
            for (;;) {
                const int rc = zk::gkr_batch_layer_begin(d.ctx(), plan, alpha_pow[0].c, sc_claims[0].c, consts.data(), have_eq ? eq_evals.words.ptr() : nullptr, lambda.c, chan);
                if (rc != zk::GKR_BATCH_AGAIN) { d.check(rc); break; }
                make_eq();
            }
            hc.reset();
            if (layer + 1 < n_layers) make_next(layer + 1);
            hc.reset(new HostClock("gkr.layer.wait"));
            zk::GkrLayerResult res;
            d.check(zk::gkr_batch_layer_end(d.ctx(), plan, res));
            HashWords digest;
            memcpy(digest.data(), res.channel, 32);
            ch.set_state(digest, res.channel[8]);
            for (int round = 0; round < nv; round++) {
                const uint32_t* w = res.records + zk::GKR_LAYER_OUT_WORDS * (size_t)round;
                UniPoly rp;
                for (uint32_t t = 0; t < w[16] && t < 4; t++) rp.c.push_back(q_at(w + 4 * t));
                round_polys.push_back(std::move(rp));
                assignment.push_back(q_at(w + 20));
            }
            masks_at = res.masks;
        } else {
            if (nv > 0) host_rounds(d, ch, plan, sumcheck_alpha, lambda, ood_point, eq_evals, sc_claims, round_polys, assignment, mask_words);
            masks_at = mask_words.data();
            if (layer + 1 < n_layers) make_next(layer + 1);
        }
        hc.reset(new HostClock("gkr.layer.masks"));
        sumcheck_round_polys.push_back(std::move(round_polys));
        // try_into_mask, :572-597. An oracle that entered with two entries had no sum-check round: its mask came with the towers.
        for (size_t k = 0; k < K; k++) {
            const size_t i = inst[k];
            const bool had_round = plan.n_vars[k] > 0;
            const uint32_t* w = had_round ? masks_at + zk::GKR_LAYER_MASK_WORDS * k : tops.data() + top_of[i] + 8;
            const int kind = towers[i].kind_at(level);
            MaskRec m;
            if (kind == ZKB_GKR_GRAND_PRODUCT) { m.n_cols = 1; m.v[0] = q_at(w); m.v[1] = q_at(w + 4); }
            else {
                if (kind == ZKB_GKR_LOGUP_MULTIPLICITIES && !had_round) throw Error(ZKB_EINVAL, "gkr: a multiplicities layer cannot be a mask");
                m.n_cols = 2;
                m.v[0] = kind == ZKB_GKR_LOGUP_SINGLES ? qm31_one() : q_at(w + 8);
                m.v[1] = kind == ZKB_GKR_LOGUP_SINGLES ? qm31_one() : q_at(w + 12);
                m.v[2] = q_at(w);
                m.v[3] = q_at(w + 4);
            }
            ch.mix_felts(m.v, 2 * m.n_cols);
            masks_by_inst[i].push_back(m);
        }
        const qm31 challenge = ch.draw_secure_felt();
        ood_point = std::move(assignment);
        ood_point.push_back(challenge);
        for (size_t i : inst) {
            const MaskRec& m = masks_by_inst[i].back();
            claims[i].n_cols = m.n_cols;
            for (uint32_t c = 0; c < m.n_cols; c++) claims[i].v[c] = challenge * (m.v[2 * c + 1] - m.v[2 * c]) + m.v[2 * c];
        }
        hc.reset();
    }
    std::vector<uint32_t> o;
    size_t room = 16 + 4 * (ood_point.size() + 1) + 32 * n_inst;
    for (auto& l : sumcheck_round_polys) room += 1 + 17 * l.size();
    for (auto& m : masks_by_inst) room += 17 * m.size();
    o.reserve(room);
    auto put = [&](const qm31* q, size_t n) { for (size_t k = 0; k < n; k++) o.insert(o.end(), q[k].c, q[k].c + 4); };
    o.push_back((uint32_t)sumcheck_round_polys.size());
    for (auto& l : sumcheck_round_polys) {
        o.push_back((uint32_t)l.size());
        for (auto& p : l) { o.push_back((uint32_t)p.c.size()); put(p.c.data(), p.c.size()); }
    }
    for (auto& of : masks_by_inst) {
        o.push_back((uint32_t)of.size());
        for (auto& m : of) { o.push_back(m.n_cols); put(m.v, 2 * m.n_cols); }
    }
    for (auto& c : output_claims) { o.push_back(c.n_cols); put(c.v, c.n_cols); }
    o.push_back((uint32_t)ood_point.size());
    put(ood_point.data(), ood_point.size());
    for (auto& c : claims) { o.push_back(c.n_cols); put(c.v, c.n_cols); }
    return o;
}

// ------------------------------------------------------------------ one PCS proof over G ranks
// The reference has no multi-device code; this is the proof of pcs_prove_impl (one tree of equally sized columns, one
// out-of-domain sample per column) with the data-parallel phases sharded: rank r interpolates and extends ncols / G
// columns; an exchange (the caller's: the library moves no data between devices) turns the column shards into row
// shards [ncols][N / G]; every rank hashes the Merkle subtree over its rows, evaluates its own polynomials at the
// out-of-domain point and computes the quotients of its rows. The Fiat-Shamir channel is replicated: every rank mixes
// the same values in the same order. The quotient column (4 x N words, 1 / (ncols / 4) of the evaluations) is gathered
// by the caller and every rank runs the same FRI commitment, grind and query draw on it; a rank then decommits the
// queried rows it owns, and any rank merges the parts, layer by layer in rank order, into the single-device proof's words.
struct ShardSession {
    zkb_ctx* ctx;
    Device dev;
    int rank, world, log_g, ncols, ncl, n_chunks = 1;
    uint32_t* ext_rows = nullptr;
    std::vector<uint32_t*> peer_rows;  // every rank's receive buffer as this process sees it (own buffer at [rank]); empty: the caller exchanges
    uint32_t log_n, log_out, log_local;
    size_t N, R;
    PcsConfig config;
    Channel ch;
    std::vector<BaseColumn> coeffs;    // views of the caller's local columns, interpolated in place
    BaseColumn evals;                  // [ncl][N]
    BaseColumn rows;                   // [ncols][R]; global column c = source rank * ncl + j
    std::vector<BaseColumn> row_cols;  // views of `rows`
    MerkleProver subtree, top;
    BaseColumn roots;                  // [world][8]
    Hash root{};
    CirclePointQ oods{};
    std::vector<qm31> samples;
    SecureColumnByCoords quot_local, quot_full;
    FriProver fri;
    uint64_t nonce = 0;
    std::vector<size_t> query_positions;
    FriProof fri_proof;
    MerkleDecommitment top_dec;
    ShardSession(zkb_ctx* c) : ctx(c), dev(c) {}
};

}  // namespace b200

struct zkb_shard_pcs { b200::ShardSession s; zkb_shard_pcs(zkb_ctx* c) : s(c) {} };

namespace b200 {

template <class F> static int shard_guard(zkb_ctx* ctx, F&& f) {
    try {
        f();
        return ZKB_OK;
    } catch (const Error& e) {
        return zk_set_error_public(ctx, e.code, e.what());
    } catch (const std::exception& e) {
        return zk_set_error_public(ctx, ZKB_ENOMEM, e.what());
    }
}

}  // namespace b200

using namespace b200;

extern "C" {

int zkb_shard_pcs_begin(zkb_ctx* ctx, int rank, int world, int ncols_total, int log_n, const zkb_pcs_config* cfg, zkb_shard_pcs** out) {
    if (!ctx || !cfg || !out) return ZKB_EINVAL;
    *out = nullptr;
    if (world < 1 || (world & (world - 1)) || rank < 0 || rank >= world || ncols_total < world || ncols_total % world || log_n < 1)
        return zk_set_error_public(ctx, ZKB_EINVAL, "zkb_shard_pcs_begin: the rank count must be a power of two that divides the column count");
    int log_g = 0;
    while ((1 << log_g) < world) log_g++;
    int log_out = log_n + (int)cfg->log_blowup_factor;
    if (log_out > zkb_max_log_size(ctx) || log_out - log_g < 3)
        return zk_set_error_public(ctx, ZKB_EINVAL, "zkb_shard_pcs_begin: every rank needs at least 8 rows and the context must cover the evaluation domain");
    return shard_guard(ctx, [&] {
        auto* h = new zkb_shard_pcs(ctx);
        ShardSession& s = h->s;
        s.rank = rank; s.world = world; s.log_g = log_g; s.ncols = ncols_total; s.ncl = ncols_total / world;
        s.log_n = (uint32_t)log_n; s.log_out = (uint32_t)log_out; s.log_local = (uint32_t)(log_out - log_g);
        s.N = (size_t)1 << log_out; s.R = s.N >> log_g;
        s.config = PcsConfig{cfg->pow_bits, {cfg->log_blowup_factor, cfg->log_last_layer_degree_bound, cfg->n_queries, 1}};
        s.config.mix_into(s.ch);
        *out = h;
    });
}

int zkb_shard_pcs_end(zkb_shard_pcs* h) {
    if (!h) return ZKB_EINVAL;
    zkb_ctx* ctx = h->s.ctx;
    zkb_sync(ctx);
    delete h;
    return ZKB_OK;
}

int zkb_shard_pcs_set_rows(zkb_shard_pcs* h, uint32_t* d_rows) {
    if (!h) return ZKB_EINVAL;
    h->s.ext_rows = d_rows;
    return ZKB_OK;
}

int zkb_shard_pcs_set_peer_rows(zkb_shard_pcs* h, uint32_t* const* peer_rows) {
    if (!h) return ZKB_EINVAL;
    ShardSession& s = h->s;
    s.peer_rows.clear();
    if (!peer_rows) return ZKB_OK;
    for (int r = 0; r < s.world; r++) {
        if (!peer_rows[r]) return zk_set_error_public(s.ctx, ZKB_EINVAL, "zkb_shard_pcs_set_peer_rows: null buffer");
        s.peer_rows.push_back(peer_rows[r]);
    }
    s.ext_rows = s.peer_rows[s.rank];
    return ZKB_OK;
}

int zkb_shard_pcs_extend_begin(zkb_shard_pcs* h, uint32_t* const* d_cols, int n_chunks) {
    if (!h || !d_cols) return ZKB_EINVAL;
    ShardSession& s = h->s;
    if (n_chunks < 1 || s.ncl % n_chunks) return zk_set_error_public(s.ctx, ZKB_EINVAL, "zkb_shard_pcs_extend_begin: the chunk count must divide the local column count");
    return shard_guard(s.ctx, [&] {
        std::vector<BaseColumn*> cols;
        s.coeffs.clear();
        for (int c = 0; c < s.ncl; c++) s.coeffs.push_back(BaseColumn::view(s.dev, d_cols[c], (size_t)1 << s.log_n));
        for (auto& c : s.coeffs) cols.push_back(&c);
        B200Backend::interpolate_columns(s.dev, cols);
        s.n_chunks = n_chunks;
        s.evals = BaseColumn(s.dev, (size_t)s.ncl * s.N);  // [chunk][world][ncl / chunks][R]: block d of a chunk is what rank d receives
        // [chunk][source rank][ncl / chunks][R]; the caller's own buffer when it has given one (a buffer its peers can write)
        s.rows = s.ext_rows ? BaseColumn::view(s.dev, s.ext_rows, (size_t)s.ncols * s.R) : BaseColumn(s.dev, (size_t)s.ncols * s.R);
    });
}

int zkb_shard_pcs_extend_chunk(zkb_shard_pcs* h, int k, uint32_t** d_send, uint32_t** d_recv, size_t* words_per_peer) {
    if (!h || !d_send || !d_recv || !words_per_peer) return ZKB_EINVAL;
    ShardSession& s = h->s;
    if (k < 0 || k >= s.n_chunks || s.coeffs.empty()) return zk_set_error_public(s.ctx, ZKB_EINVAL, "zkb_shard_pcs_extend_chunk: no such chunk");
    return shard_guard(s.ctx, [&] {
        const int cc = s.ncl / s.n_chunks;
        std::vector<const uint32_t*> src;
        std::vector<uint32_t*> dst;
        uint32_t* send = s.evals.ptr() + (size_t)k * s.world * cc * s.R;
        for (int j = 0; j < cc; j++) src.push_back(s.coeffs[k * cc + j].ptr());
        if (zk::lde_blocked_supported((int)s.log_n, (int)s.log_out, (int)s.log_local)) {
            // the transform's last pass writes every row block where the exchange sends it from: no repack
            for (int j = 0; j < cc; j++) dst.push_back(send + (size_t)j * s.R);
            s.dev.check(zk::lde_cols_blocked(s.ctx, src.data(), cc, (int)s.log_n, dst.data(), (int)s.log_out, (int)s.log_local,
                                             (uint32_t)((size_t)cc * s.R)));
        } else {
            BaseColumn plain(s.dev, (size_t)cc * s.N);
            for (int j = 0; j < cc; j++) dst.push_back(plain.ptr() + (size_t)j * s.N);
            s.dev.check(zkb_lde_cols(s.ctx, src.data(), cc, (int)s.log_n, dst.data(), (int)s.log_out));
            s.dev.check(zk::repack_row_blocks(s.ctx, plain.ptr(), send, cc, (int)s.log_out, (int)s.log_local));
        }
        *d_send = send;
        *d_recv = s.rows.ptr() + (size_t)k * s.world * cc * s.R;
        *words_per_peer = (size_t)cc * s.R;
        if (!s.peer_rows.empty()) {
            // block d of the chunk goes to rank d's buffer, into the place of this rank's block there: copy engines, after the
            // transform just enqueued, four copies side by side; every rank starts with a different peer
            const size_t words = (size_t)cc * s.R, at = ((size_t)k * s.world + s.rank) * words;
            for (int j = 0; j < s.world; j++) {
                const int dst = (s.rank + j) % s.world;
                s.dev.check(zkb_copy_to_peer(s.ctx, s.peer_rows[dst] + at, send + (size_t)dst * words, words * 4, j));
            }
        }
    });
}

int zkb_shard_pcs_extend(zkb_shard_pcs* h, uint32_t* const* d_cols, uint32_t** d_send, uint32_t** d_rows) {
    if (!h || !d_cols || !d_send || !d_rows) return ZKB_EINVAL;
    int rc = zkb_shard_pcs_extend_begin(h, d_cols, 1);
    if (rc) return rc;
    size_t words = 0;
    return zkb_shard_pcs_extend_chunk(h, 0, d_send, d_rows, &words);
}

int zkb_shard_pcs_subtree(zkb_shard_pcs* h, uint32_t** d_root, uint32_t** d_roots) {
    if (!h || !d_root || !d_roots) return ZKB_EINVAL;
    ShardSession& s = h->s;
    return shard_guard(s.ctx, [&] {
        s.evals = BaseColumn();  // the column shards have been sent
        s.row_cols.clear();
        // global column c = source rank * ncl + chunk * cc + j lies in block [chunk][source rank] of the received rows
        const int cc = s.ncl / s.n_chunks;
        for (int c = 0; c < s.ncols; c++) {
            const int src = c / s.ncl, k = (c % s.ncl) / cc, j = c % cc;
            s.row_cols.push_back(BaseColumn::view(s.dev, s.rows.ptr() + ((size_t)(k * s.world + src) * cc + j) * s.R, s.R));
        }
        std::vector<const BaseColumn*> refs;
        for (auto& c : s.row_cols) refs.push_back(&c);
        s.subtree = MerkleProver::commit(s.dev, refs);
        s.roots = BaseColumn(s.dev, (size_t)8 * s.world);
        *d_root = s.subtree.layers[0].ptr();
        *d_roots = s.roots.ptr();
    });
}

int zkb_shard_pcs_sample(zkb_shard_pcs* h, uint32_t* h_samples) {
    if (!h || !h_samples) return ZKB_EINVAL;
    ShardSession& s = h->s;
    return shard_guard(s.ctx, [&] {
        // the top log2(G) layers over the gathered subtree roots: the same nodes the single-device tree has there
        s.top = MerkleProver();
        s.top.layers.resize(s.log_g + 1);
        s.top.layers[s.log_g] = BaseColumn::view(s.dev, s.roots.ptr(), (size_t)8 * s.world);
        for (int lg = s.log_g - 1; lg >= 0; lg--) s.top.layers[lg] = B200Backend::commit_on_layer(s.dev, (uint32_t)lg, &s.top.layers[lg + 1], {});
        s.root = s.top.root(s.dev);
        s.ch.mix_root(s.root);
        s.oods = get_random_point(s.ch);
        std::vector<const BaseColumn*> polys;
        for (auto& c : s.coeffs) polys.push_back(&c);
        auto vals = B200Backend::batch_eval_at_point(s.dev, polys, s.oods);
        for (int c = 0; c < s.ncl; c++) memcpy(h_samples + 4 * c, vals[c].c, 16);
    });
}

int zkb_shard_pcs_quotients(zkb_shard_pcs* h, const uint32_t* h_all_samples, uint32_t* d_quot_local[4], uint32_t* d_quot_full[4]) {
    if (!h || !h_all_samples || !d_quot_local || !d_quot_full) return ZKB_EINVAL;
    ShardSession& s = h->s;
    return shard_guard(s.ctx, [&] {
        s.samples.resize(s.ncols);
        for (int c = 0; c < s.ncols; c++) memcpy(s.samples[c].c, h_all_samples + 4 * c, 16);
        s.ch.mix_felts(s.samples);
        qm31 random_coeff = s.ch.draw_secure_felt();
        // compute_fri_quotients for one size group and one sample point, on this rank's rows: the numerators are
        // row-local; the denominators need the rows' domain points (zkb_quot_combine_rows)
        std::vector<const BaseColumn*> refs;
        for (auto& c : s.row_cols) refs.push_back(&c);
        ColumnSampleBatch batch{s.oods, {}};
        qm31 pow = qm31_one();
        for (int c = 0; c < s.ncols; c++) { batch.cols_vals_randpows.push_back({(size_t)c, s.samples[c], pow}); pow = pow * random_coeff; }
        std::vector<AccumulatedNumerators> accs;
        B200Backend::accumulate_numerators(s.dev, refs, {batch}, accs);
        s.quot_local = SecureColumnByCoords(s.dev, s.R);
        s.quot_full = SecureColumnByCoords(s.dev, s.N);
        std::vector<const uint32_t*> cols;
        for (auto p : accs[0].partial_numerators_acc.cptrs()) cols.push_back(p);
        int acc_log = (int)s.log_out;
        uint32_t pts[8];
        memcpy(pts, s.oods.x.c, 16);
        memcpy(pts + 4, s.oods.y.c, 16);
        auto o = s.quot_local.ptrs();
        s.dev.check(zkb_quot_combine_rows(s.ctx, 1, cols.data(), &acc_log, accs[0].first_linear_term_acc.c, pts, (int)s.log_out,
                                          (size_t)s.rank * s.R, s.R, o.data()));
        s.dev.check(zkb_sync(s.ctx));  // the accumulation is freed when this returns; the caller's gather may run on another stream
        auto f = s.quot_full.ptrs();
        for (int k = 0; k < 4; k++) { d_quot_local[k] = o[k]; d_quot_full[k] = f[k]; }
    });
}

// Serialised part of one rank: [layers L][per layer: count, count x 8 words][n value words][values].
int zkb_shard_pcs_fri_and_decommit(zkb_shard_pcs* h, uint32_t* h_part, size_t cap, size_t* n_words) {
    if (!h || !h_part || !n_words) return ZKB_EINVAL;
    ShardSession& s = h->s;
    return shard_guard(s.ctx, [&] {
        s.fri = FriProver::commit(s.dev, s.ch, s.config.fri, s.quot_full);
        s.nonce = B200Backend::grind(s.dev, s.ch.pow_prefixed_digest(s.config.pow_bits), s.config.pow_bits);
        s.ch.mix_u64(s.nonce);
        GatherPlan plan;
        auto fri_pending = s.fri.plan_decommit(plan, s.dev, s.ch, s.query_positions);
        // this rank's rows among the queried ones, and the ranks that own any
        std::vector<size_t> local, owners;
        for (auto q : s.query_positions) {
            if ((q >> s.log_local) == (size_t)s.rank) local.push_back(q - ((size_t)s.rank << s.log_local));
            owners.push_back(q >> s.log_local);
        }
        std::vector<size_t> per_layer;
        local = sorted_dedup(local);
        owners = sorted_dedup(owners);
        PendingMerkle pm = s.subtree.plan_decommit(plan, QueriesOf{s.log_local, local}, &per_layer);
        PendingMerkle pt = s.top.plan_decommit(plan, QueriesOf{(uint32_t)s.log_g, owners});
        plan.execute(s.dev);
        s.fri_proof = s.fri.finish_decommit(plan, fri_pending);
        s.top_dec = pt.finish(plan).second;
        auto mine = pm.finish(plan);
        std::vector<uint32_t> o;
        o.push_back((uint32_t)per_layer.size());
        size_t at = 0;
        for (size_t cnt : per_layer) {
            o.push_back((uint32_t)cnt);
            for (size_t k = 0; k < cnt; k++, at++) o.insert(o.end(), mine.second.hash_witness[at].begin(), mine.second.hash_witness[at].end());
        }
        o.push_back((uint32_t)mine.first.size());
        mine.first.append_to(o);
        *n_words = o.size();
        if (o.size() > cap) throw Error(ZKB_EINVAL, "zkb_shard_pcs_fri_and_decommit: output buffer too small");
        memcpy(h_part, o.data(), o.size() * 4);
    });
}

int zkb_shard_pcs_finish(zkb_shard_pcs* h, const uint32_t* const* h_parts, const size_t* part_words, uint32_t* h_out, size_t cap,
                         size_t* n_words) {
    if (!h || !h_parts || !part_words || !h_out || !n_words) return ZKB_EINVAL;
    ShardSession& s = h->s;
    return shard_guard(s.ctx, [&] {
        PcsProof proof;
        proof.commitments.push_back(s.root);
        proof.sampled_values.values = s.samples;
        for (size_t k = 0; k < s.samples.size(); k++) proof.sampled_values.first.push_back(k + 1);
        proof.sampled_values.tree_first.push_back(s.samples.size());
        MerkleDecommitment dec;
        std::vector<uint32_t> values;
        std::vector<size_t> cursor(s.world, 1);
        size_t n_layers = 0;
        for (int r = 0; r < s.world; r++) {
            if (part_words[r] < 2) throw Error(ZKB_EINVAL, "zkb_shard_pcs_finish: truncated part");
            if (r == 0) n_layers = h_parts[0][0];
            else if (h_parts[r][0] != n_layers) throw Error(ZKB_EINVAL, "zkb_shard_pcs_finish: the parts disagree on the layer count");
        }
        // the single-device decommitment lists a layer's witness hashes in node order: rank order within each layer
        for (size_t l = 0; l < n_layers; l++)
            for (int r = 0; r < s.world; r++) {
                const uint32_t* p = h_parts[r];
                size_t& c = cursor[r];
                if (c >= part_words[r]) throw Error(ZKB_EINVAL, "zkb_shard_pcs_finish: truncated part");
                size_t cnt = p[c++];
                if (c + 8 * cnt > part_words[r]) throw Error(ZKB_EINVAL, "zkb_shard_pcs_finish: truncated part");
                for (size_t k = 0; k < cnt; k++, c += 8) { Hash hh; memcpy(hh.data(), p + c, 32); dec.hash_witness.push_back(hh); }
            }
        dec.hash_witness.insert(dec.hash_witness.end(), s.top_dec.hash_witness.begin(), s.top_dec.hash_witness.end());
        for (int r = 0; r < s.world; r++) {
            const uint32_t* p = h_parts[r];
            size_t c = cursor[r];
            if (c >= part_words[r]) throw Error(ZKB_EINVAL, "zkb_shard_pcs_finish: truncated part");
            size_t cnt = p[c++];
            if (c + cnt > part_words[r]) throw Error(ZKB_EINVAL, "zkb_shard_pcs_finish: truncated part");
            values.insert(values.end(), p + c, p + c + cnt);
        }
        proof.decommitments.push_back(std::move(dec));
        proof.queried_values.push_back(Words{std::move(values), {}});
        proof.proof_of_work = s.nonce;
        proof.fri = s.fri_proof;
        PcsProof::RawSink w{h_out, cap};
        proof.write(w);
        w.finish();
        w.insert(w.end(), s.ch.digest().begin(), s.ch.digest().end());
        *n_words = w.size();
        if (w.size() > cap) throw Error(ZKB_EINVAL, "zkb_shard_pcs_finish: output buffer too small");
    });
}

}  // extern "C"


// Commits the caller's trees in order (TreeBuilder::extend_evals + commit per tree), from device columns or from host
// columns with the upload overlapped.
// meanwhile: what the host has to do that does not depend on the roots; where the trees are on the device it is done while they are hashed.
template <class Meanwhile>
static void commit_input_trees(Device& dev, zkb_ctx* ctx, CommitmentSchemeProver& prover, Channel& ch, int n_trees, const int* tree_ncols,
                               uint32_t* const* d_cols, const uint32_t* const* h_cols, const uint32_t* col_logs, int total, Meanwhile meanwhile) {
        int flat = 0;
        if (d_cols) {
            // (with phases to be timed one tree after the other: their marks are on one stream)
            const bool together = !prover.phase_ms;
            CommitmentSchemeProver::SeveralTrees several;
            zk::SideScope scope(ctx);
            for (int t = 0; t < n_trees; t++) {
                several.more = t + 1 < n_trees;
                std::vector<BaseColumn> columns;
                columns.reserve((size_t)tree_ncols[t]);
                for (int c = 0; c < tree_ncols[t]; c++, flat++)
                    columns.push_back(BaseColumn::view(dev, d_cols[flat], (size_t)1 << col_logs[flat]));
                prover.commit_evals(std::move(columns), ch, nullptr, nullptr, false, together ? &several : nullptr);
            }
            meanwhile();
            if (together) prover.mix_roots(ch);
        } else {
            // Host columns: every copy of every tree is enqueued on the copy stream first, with a fence
            // after each ~1/32 of the bytes, so that the transfer runs at link speed from start to end
            // while the compute stream interpolates and extends what has already arrived.
            size_t total_bytes = 0;
            for (int i = 0; i < total; i++) total_bytes += (size_t)4 << col_logs[i];
            const size_t per_fence = std::max<size_t>(total_bytes / 32, 1);
            // The columns of a tree live in one allocation (each padded to 64 words), so that columns that
            // are adjacent in host memory, as a row-major trace is, go up in one copy per fence.
            std::vector<std::vector<BaseColumn>> tree_cols(n_trees);
            std::vector<std::vector<int>> tree_fences(n_trees);
            std::vector<BaseColumn> slabs;
            for (int t = 0; t < n_trees; t++) {
                size_t words = 0;
                for (int c = 0; c < tree_ncols[t]; c++) words += std::max<size_t>((size_t)1 << col_logs[flat + c], 64);
                if (words) slabs.emplace_back(dev, words);
                else slabs.emplace_back();  // a tree without columns (it is still committed: its root is the hash of nothing)
                size_t off = 0;
                for (int c = 0; c < tree_ncols[t]; c++, flat++) {
                    size_t n = (size_t)1 << col_logs[flat];
                    tree_cols[t].push_back(BaseColumn::view(dev, slabs.back().ptr() + off, n));
                    off += std::max<size_t>(n, 64);
                }
            }
            flat = 0;
            int fence = 0;
            size_t since = 0;
            // a pending run of copies that are contiguous on both sides
            uint32_t* run_dst = nullptr;
            const uint32_t* run_src = nullptr;
            size_t run_bytes = 0;
            auto flush = [&](int fence_id) {
                if (run_bytes) dev.check(zkb_h2d_overlapped(ctx, run_dst, run_src, run_bytes, fence_id));
                else if (fence_id >= 0) dev.check(zkb_h2d_overlapped(ctx, nullptr, nullptr, 0, fence_id));
                run_bytes = 0;
            };
            try {  // from the first enqueued copy on, no column may be freed while the copy stream still writes into it
            for (int t = 0; t < n_trees; t++)
                for (int c = 0; c < tree_ncols[t]; c++, flat++) {
                    size_t bytes = (size_t)4 << col_logs[flat];
                    uint32_t* dst = tree_cols[t][c].ptr();
                    if (run_bytes && (const uint8_t*)run_src + run_bytes == (const uint8_t*)h_cols[flat] &&
                        (uint8_t*)run_dst + run_bytes == (uint8_t*)dst) {
                        run_bytes += bytes;
                    } else {
                        flush(-1);
                        run_dst = dst; run_src = h_cols[flat]; run_bytes = bytes;
                    }
                    since += bytes;
                    bool close = since >= per_fence || flat == total - 1;
                    tree_fences[t].push_back(fence);
                    if (close) { flush(fence); since = 0; if (fence < 63) fence++; }
                }
                for (int t = 0; t < n_trees; t++) prover.commit_evals(std::move(tree_cols[t]), ch, &tree_fences[t], &slabs[t]);
                meanwhile();
            } catch (...) {
                zkb_sync(ctx);
                throw;
            }
        }
}

static int pcs_prove_impl(zkb_ctx* ctx, int n_trees, const int* tree_ncols, uint32_t* const* d_cols, const uint32_t* const* h_cols,
                          const uint32_t* col_logs, const zkb_pcs_config* cfg, int two_sample_every, uint32_t* h_out, size_t cap,
                          size_t* n_words, float* h_phase_ms) {
    if (!ctx) return ZKB_EINVAL;
    if (!tree_ncols || !col_logs || !cfg || !h_out || !n_words || n_trees <= 0 || (!d_cols && !h_cols)) return ZKB_EINVAL;
    try {
        Device dev(ctx);
        PcsConfig config{cfg->pow_bits, {cfg->log_blowup_factor, cfg->log_last_layer_degree_bound, cfg->n_queries, 1}};
        int total = 0;
        uint32_t max_log = 0;
        for (int t = 0; t < n_trees; t++) total += tree_ncols[t];
        for (int i = 0; i < total; i++) max_log = std::max(max_log, col_logs[i]);
        if ((int)(max_log + config.fri.log_blowup_factor) > zkb_max_log_size(ctx)) return ZKB_EINVAL;
        Channel ch;
        config.mix_into(ch);
        CommitmentSchemeProver prover(dev, config, h_phase_ms);
        // Which column is sampled where: all at the out-of-domain point, drawn from the roots, some one trace step back from it too. Points are told apart
        // by their distance from that one.
        SamplePoints points;
        std::vector<cpoint> distance{host_circle_point(0)};
        SamplePlan sample_plan;
        {
            HostClock hcc("pcs.commit_trees");
            commit_input_trees(dev, ctx, prover, ch, n_trees, tree_ncols, d_cols, h_cols, col_logs, total, [&] {
                points.point_of.reserve(2 * (size_t)total);
                points.first.reserve((size_t)total + 1);
                uint32_t step_back[33];  // per column size, the place of its second point
                for (auto& k : step_back) k = ~0u;
                for (int flat = 0; flat < total; flat++) {
                    if (two_sample_every && flat % two_sample_every == 0) {
                        uint32_t& k = step_back[col_logs[flat]];
                        if (k == ~0u) {
                            // the conjugate of the step of CanonicCoset(col_log)
                            const cpoint st = host_circle_point(1u << (31 - col_logs[flat])), back{st.x, m31_neg(st.y)};
                            for (k = 0; k < distance.size() && (distance[k].x != back.x || distance[k].y != back.y);) k++;
                            if (k == distance.size()) distance.push_back(back);
                        }
                        points.point_of.push_back(k);
                    }
                    points.point_of.push_back(0);
                    points.end_column();
                }
                sample_plan = prover.plan_samples(points, distance.size());
            });
        }
        const CirclePointQ oods = get_random_point(ch);
        points.points.push_back(oods);
        for (size_t k = 1; k < distance.size(); k++) points.points.push_back(point_add(oods, {qm31_from_m31(distance[k].x), qm31_from_m31(distance[k].y)}));
        std::unique_ptr<HostClock> hc(new HostClock("pcs.prove_values"));
        PcsProof proof = prover.prove_values(std::move(points), sample_plan, ch);
        prover.finish_timing();
        hc.reset(new HostClock("pcs.write"));
        PcsProof::RawSink w{h_out, cap};  // straight into the caller's buffer: a proof of many columns is tens of megabytes
        proof.write(w);
        w.finish();
        w.insert(w.end(), ch.digest().begin(), ch.digest().end());
        *n_words = w.size();
        hc.reset();
        HostClock::dump("zkb_pcs_prove");
        if (w.size() > cap) return zk_set_error_public(ctx, ZKB_EINVAL, "zkb_pcs_prove: output buffer too small");
        return ZKB_OK;
    } catch (const Error& e) {
        return zk_set_error_public(ctx, e.code, e.what());
    } catch (const std::exception& e) {
        return zk_set_error_public(ctx, ZKB_ENOMEM, e.what());
    }
}

// prove() (STWO/prover/mod.rs:41-173) for a statement of one or more components: commit the trees, draw the random
// coefficient, evaluate every component's constraint quotients on the evaluation domain of twice its trace size
// (zkb_constraint_quotients) into the accumulation of that size, lift and add the accumulations
// (DomainEvaluationAccumulator, prover/air/accumulation.rs), interpolate and split the composition polynomial, commit its
// eight coordinate halves, sample every column at its mask points around a drawn out-of-domain point, and prove the
// samples. The prover's own sanity check - the composition polynomial's value at the point, once from the committed
// halves (core/proof.rs:27-57) and once from the constraints at the sampled mask values (core/air/components.rs:76-94,
// constraint-framework/src/component.rs:374-413, point.rs) - is returned in oods_evals for the caller to compare.
static int stark_prove_impl(zkb_ctx* ctx, int n_trees, const int* tree_ncols, uint32_t* const* d_cols, const uint32_t* const* h_cols,
                            int n_components, const zkb_stark_component* comps, const zkb_pcs_config* cfg, uint32_t* h_out, size_t cap,
                            size_t* n_words, uint32_t* oods_evals, float* h_phase_ms, float* composition_ms) {
    if (!ctx) return ZKB_EINVAL;
    if (!tree_ncols || !cfg || !h_out || !n_words || !comps || !oods_evals || n_trees <= 0 || n_components <= 0 || (!d_cols && !h_cols))
        return ZKB_EINVAL;
    try {
        Device dev(ctx);
        PcsConfig config{cfg->pow_bits, {cfg->log_blowup_factor, cfg->log_last_layer_degree_bound, cfg->n_queries, 1}};
        const uint32_t blowup = config.fri.log_blowup_factor;
        uint32_t max_trace_log = 0;
        size_t n_constraints = 0;
        for (int k = 0; k < n_components; k++) {
            const zkb_stark_component& c = comps[k];
            if (!c.prog || c.trace_log < 1 || (size_t)n_trees != c.prog->tree_base.size() || (c.prog->n_scalars && !c.scalars))
                return zk_set_error_public(ctx, ZKB_EINVAL, "zkb_stark_prove: a component has no program, no scalars, or a program compiled for other trees");
            max_trace_log = std::max(max_trace_log, c.trace_log);
            n_constraints += c.prog->constraints.size();
        }
        if (blowup < 1 || (int)(max_trace_log + blowup) > zkb_max_log_size(ctx)) return ZKB_EINVAL;
        // where each component's columns start in each tree (they follow those of the components before it), column sizes
        auto cols_of = [&](int k, int t) {
            const auto& tb = comps[k].prog->tree_base;
            return (t + 1 < n_trees ? tb[t + 1] : comps[k].prog->n_cols) - tb[t];
        };
        std::vector<std::vector<uint32_t>> first((size_t)n_components, std::vector<uint32_t>((size_t)n_trees, 0));
        std::vector<uint32_t> tree_start((size_t)n_trees, 0), col_logs;
        int total = 0;
        for (int t = 0; t < n_trees; t++) {
            tree_start[t] = (uint32_t)total;
            uint32_t at = 0;
            for (int k = 0; k < n_components; k++) {
                first[k][t] = at;
                at += cols_of(k, t);
                col_logs.insert(col_logs.end(), cols_of(k, t), comps[k].trace_log);
            }
            if ((int)at != tree_ncols[t])
                return zk_set_error_public(ctx, ZKB_EINVAL, "zkb_stark_prove: the trees do not have the columns the programs were compiled for");
            total += tree_ncols[t];
        }
        Channel ch;
        config.mix_into(ch);
        CommitmentSchemeProver prover(dev, config, h_phase_ms);
        commit_input_trees(dev, ctx, prover, ch, n_trees, tree_ncols, d_cols, h_cols, col_logs.data(), total, [] {});

        // ---- composition polynomial
        const qm31 random_coeff = ch.draw_secure_felt();
        dev.check(zkb_event_record(ctx, 28));
        std::vector<qm31> ascending_powers(n_constraints);
        {
            qm31 pw = qm31_one();
            for (size_t i = 0; i < n_constraints; i++) { ascending_powers[i] = pw; pw = pw * random_coeff; }
        }
        size_t remaining = n_constraints;
        std::map<uint32_t, SecureColumnByCoords> sub;  // sub_accumulations by log size
        std::vector<qm31> shifts((size_t)n_components, qm31_zero());
        for (int k = 0; k < n_components; k++) {
            const zkb_stark_component& c = comps[k];
            const size_t n_k = c.prog->constraints.size();
            // columns(): the last n_k powers, reversed so that the component's first constraint takes the highest (component_prover.rs:271)
            std::vector<qm31> powers(n_k);
            for (size_t i = 0; i < n_k; i++) powers[i] = ascending_powers[remaining - 1 - i];
            remaining -= n_k;
            const uint32_t eval_log = c.trace_log + 1;
            // the component's columns on its evaluation domain: the committed evaluations themselves when the blow-up is 2
            std::vector<BaseColumn> extended;
            std::vector<const uint32_t*> col_ptrs;
            for (int t = 0; t < n_trees; t++) {
                const uint32_t cnt = cols_of(k, t);
                if (blowup == 1) {
                    for (uint32_t q = 0; q < cnt; q++) col_ptrs.push_back(prover.trees[t].evals[first[k][t] + q].ptr());
                } else if (cnt) {
                    std::vector<const BaseColumn*> cc;
                    for (uint32_t q = 0; q < cnt; q++) cc.push_back(&prover.trees[t].coeffs[first[k][t] + q]);
                    auto ev = B200Backend::evaluate_polynomials(dev, cc, 1);
                    for (auto& e : ev) { col_ptrs.push_back(e.ptr()); extended.push_back(std::move(e)); }
                }
            }
            if (c.claimed_sum) {
                qm31 claimed;
                for (int q = 0; q < 4; q++) claimed.c[q] = c.claimed_sum[q];
                shifts[k] = claimed * qm31_inv(qm31_from_m31(1u << c.trace_log));  // LogupAtRow::new, logup.rs:33-41
            }
            uint32_t denom_inv[2];
            if (zkb_constraint_denom_inv((int)c.trace_log, (int)eval_log, denom_inv) != ZKB_OK) return ZKB_EINVAL;
            auto it = sub.find(eval_log);
            const bool fresh = it == sub.end();
            if (fresh) it = sub.emplace(eval_log, SecureColumnByCoords(dev, (size_t)1 << eval_log)).first;
            auto accp = it->second.ptrs();
            dev.check(zkb_constraint_quotients(ctx, c.prog, col_ptrs.data(), c.scalars, shifts[k].c, reinterpret_cast<const uint32_t*>(powers.data()),
                                               denom_inv, (int)c.trace_log, (int)eval_log, accp.data(), fresh ? 0 : 1));
        }
        // DomainEvaluationAccumulator::finalize (air/accumulation.rs:89-124): lift and add ascending sizes, interpolate;
        // then split_at_mid and extend_polys + commit
        std::vector<SecureColumnByCoords> ascending;
        for (auto& kv : sub) ascending.push_back(std::move(kv.second));
        sub.clear();
        SecureColumnByCoords acc = B200Backend::lift_and_accumulate(dev, std::move(ascending));
        const uint32_t comp_log = max_trace_log + 1;
        const size_t N = (size_t)1 << comp_log;
        if (acc.len() != N) return zk_set_error_public(ctx, ZKB_EINVAL, "zkb_stark_prove: no component of the largest size");
        {
            std::vector<BaseColumn*> ap = {&acc.columns[0], &acc.columns[1], &acc.columns[2], &acc.columns[3]};
            B200Backend::interpolate_columns(dev, ap);
            std::vector<BaseColumn> halves;
            for (int q = 0; q < 4; q++) halves.push_back(BaseColumn::view(dev, acc.columns[q].ptr(), N / 2));
            for (int q = 0; q < 4; q++) halves.push_back(BaseColumn::view(dev, acc.columns[q].ptr() + N / 2, N / 2));
            dev.check(zkb_event_record(ctx, 29));
            prover.mark(-1);  // the composition is timed on its own, not as part of the next tree's first phase
            prover.commit_evals(std::move(halves), ch, nullptr, nullptr, true);
        }

        // ---- mask points (component.rs:356-368, core/air/components.rs:32-74) and the samples' proof
        CirclePointQ oods = get_random_point(ch);
        const uint32_t lifting_log = prover.trees.back().max_log();
        const uint32_t max_log_degree_bound = lifting_log - blowup;
        // per component: the mask offsets of each of its columns, in the order the program asks for them
        std::vector<std::vector<std::vector<int32_t>>> offsets((size_t)n_components);
        std::vector<std::vector<std::vector<CirclePointQ>>> points((size_t)n_trees + 1);
        for (int t = 0; t < n_trees; t++) points[t].resize((size_t)tree_ncols[t]);
        std::map<int32_t, CirclePointQ> at_offset;  // a handful of distinct ones over all columns
        auto mask_point = [&](int32_t off) {
            auto it = at_offset.find(off);
            if (it != at_offset.end()) return it->second;
            // trace_step.mul_signed(off): the point of index off * 2^(31 - max_log_degree_bound) in the circle group
            const cpoint st = host_circle_point(((uint32_t)off << (31 - max_log_degree_bound)) & 0x7fffffffu);
            return at_offset[off] = point_add(oods, {qm31_from_m31(st.x), qm31_from_m31(st.y)});
        };
        for (int k = 0; k < n_components; k++) {
            const zkb_air_program* prog = comps[k].prog;
            offsets[k].resize(prog->n_cols);
            for (const zkb_air_op& o : prog->ops)
                if (o.op == ZKB_AIR_LOAD) {
                    auto& v = offsets[k][prog->tree_base[o.a] + o.b];
                    if (std::find(v.begin(), v.end(), (int32_t)o.c) == v.end()) v.push_back((int32_t)o.c);
                }
            for (int t = 0; t < n_trees; t++)
                for (uint32_t q = 0; q < cols_of(k, t); q++)
                    for (int32_t off : offsets[k][prog->tree_base[t] + q]) points[t][first[k][t] + q].push_back(mask_point(off));
        }
        points.back().assign(8, {oods});
        SamplePoints flat_points;
        for (auto& tree : points)
            for (auto& column : tree) {
                for (auto& p : column) flat_points.point_of.push_back(flat_points.intern(p));
                flat_points.end_column();
            }
        const SamplePlan sample_plan = prover.plan_samples(flat_points, flat_points.points.size());
        PcsProof proof = prover.prove_values(std::move(flat_points), sample_plan, ch);
        prover.finish_timing();
        if (composition_ms) dev.check(zkb_event_elapsed_ms(ctx, 28, 29, composition_ms));

        // ---- the sanity check of prove_ex
        auto from_partial_evals = [](qm31 e0, qm31 e1, qm31 e2, qm31 e3) {  // qm31.rs:51-57
            const qm31 i{{0, 1, 0, 0}}, u{{0, 0, 1, 0}}, iu{{0, 0, 0, 1}};
            return e0 + e1 * i + e2 * u + e3 * iu;
        };
        auto comp = [&](size_t c) { return *proof.sampled_values.at((size_t)n_trees, c); };
        const qm31 left = from_partial_evals(comp(0), comp(1), comp(2), comp(3));
        const qm31 right = from_partial_evals(comp(4), comp(5), comp(6), comp(7));
        const qm31 committed = left + point_repeated_double(oods, max_log_degree_bound - 1).x * right;
        // coset_vanishing(CanonicCoset(max_log_degree_bound).coset, oods): the shift -initial + step/2 is zero for a canonic coset
        qm31 vanish = oods.x;
        for (uint32_t q = 1; q < max_log_degree_bound; q++) vanish = qm31_double_x(vanish);
        const qm31 denom_inverse = qm31_inv(vanish);
        qm31 at_point = qm31_zero();  // one PointEvaluationAccumulator (core/air/accumulation.rs:12-36) through all components
        for (int k = 0; k < n_components; k++) {
            const zkb_air_program* prog = comps[k].prog;
            // the program at the point: every value is a secure-field element, a LOAD is the sampled mask value
            std::vector<qm31> v(prog->ops.size(), qm31_zero());
            std::vector<std::pair<int, uint32_t>> where(prog->n_cols);
            for (int t = 0; t < n_trees; t++)
                for (uint32_t q = 0; q < cols_of(k, t); q++) where[prog->tree_base[t] + q] = {t, first[k][t] + q};
            for (size_t i = 0; i < prog->ops.size(); i++) {
                const zkb_air_op& o = prog->ops[i];
                switch (o.op) {
                    case ZKB_AIR_LOAD: {
                        const uint32_t col = prog->tree_base[o.a] + o.b;
                        const auto& offs = offsets[k][col];
                        const size_t j = std::find(offs.begin(), offs.end(), (int32_t)o.c) - offs.begin();
                        v[i] = proof.sampled_values.at((size_t)where[col].first, where[col].second)[j];
                        break;
                    }
                    case ZKB_AIR_CONST_M31: v[i] = qm31_from_m31(o.a); break;
                    case ZKB_AIR_SCALAR: for (int q = 0; q < 4; q++) v[i].c[q] = comps[k].scalars[4 * (size_t)o.a + q]; break;
                    case ZKB_AIR_CUMSUM_SHIFT: v[i] = shifts[k]; break;
                    case ZKB_AIR_ADD_B: case ZKB_AIR_ADD_E: v[i] = v[o.a] + v[o.b]; break;
                    case ZKB_AIR_SUB_B: case ZKB_AIR_SUB_E: v[i] = v[o.a] - v[o.b]; break;
                    case ZKB_AIR_MUL_B: case ZKB_AIR_MUL_E: v[i] = v[o.a] * v[o.b]; break;
                    case ZKB_AIR_NEG_B: case ZKB_AIR_NEG_E: v[i] = qm31_neg(v[o.a]); break;
                    case ZKB_AIR_INV_B: v[i] = qm31_is_zero(v[o.a]) ? qm31_zero() : qm31_inv(v[o.a]); break;
                    case ZKB_AIR_PACK: v[i] = from_partial_evals(v[o.a], v[o.b], v[o.c], v[o.d]); break;
                    default: break;
                }
            }
            for (uint32_t cn : prog->constraints) at_point = at_point * random_coeff + denom_inverse * v[cn];
        }
        for (int q = 0; q < 4; q++) { oods_evals[q] = committed.c[q]; oods_evals[4 + q] = at_point.c[q]; }

        std::vector<uint32_t> w = proof.to_words();
        w.insert(w.end(), ch.digest().begin(), ch.digest().end());
        *n_words = w.size();
        if (w.size() > cap) return zk_set_error_public(ctx, ZKB_EINVAL, "zkb_stark_prove: output buffer too small");
        memcpy(h_out, w.data(), w.size() * 4);
        return ZKB_OK;
    } catch (const Error& e) {
        return zk_set_error_public(ctx, e.code, e.what());
    } catch (const std::exception& e) {
        return zk_set_error_public(ctx, ZKB_ENOMEM, e.what());
    }
}

extern "C" {

int zkb_pcs_prove_device(zkb_ctx* ctx, int n_trees, const int* tree_ncols, uint32_t* const* d_cols, const uint32_t* col_logs,
                         const zkb_pcs_config* config, int two_sample_every, uint32_t* h_out, size_t cap, size_t* n_words,
                         float* h_phase_ms) {
    return pcs_prove_impl(ctx, n_trees, tree_ncols, d_cols, nullptr, col_logs, config, two_sample_every, h_out, cap, n_words, h_phase_ms);
}

int zkb_stark_prove_multi_device(zkb_ctx* ctx, int n_trees, const int* tree_ncols, uint32_t* const* d_cols, int n_components,
                                 const zkb_stark_component* components, const zkb_pcs_config* config, uint32_t* h_out, size_t cap,
                                 size_t* n_words, uint32_t* oods_evals, float* h_phase_ms, float* composition_ms) {
    return stark_prove_impl(ctx, n_trees, tree_ncols, d_cols, nullptr, n_components, components, config, h_out, cap, n_words, oods_evals,
                            h_phase_ms, composition_ms);
}

int zkb_stark_prove_multi_host(zkb_ctx* ctx, int n_trees, const int* tree_ncols, const uint32_t* const* h_cols, int n_components,
                               const zkb_stark_component* components, const zkb_pcs_config* config, uint32_t* h_out, size_t cap,
                               size_t* n_words, uint32_t* oods_evals, float* h_phase_ms, float* composition_ms) {
    return stark_prove_impl(ctx, n_trees, tree_ncols, nullptr, h_cols, n_components, components, config, h_out, cap, n_words, oods_evals,
                            h_phase_ms, composition_ms);
}

int zkb_stark_prove_device(zkb_ctx* ctx, int n_trees, const int* tree_ncols, uint32_t* const* d_cols, uint32_t trace_log,
                           zkb_air_program* prog, const uint32_t* scalars, const uint32_t* claimed_sum, const zkb_pcs_config* config,
                           uint32_t* h_out, size_t cap, size_t* n_words, uint32_t* oods_evals, float* h_phase_ms, float* composition_ms) {
    zkb_stark_component c{prog, trace_log, scalars, claimed_sum};
    return stark_prove_impl(ctx, n_trees, tree_ncols, d_cols, nullptr, 1, &c, config, h_out, cap, n_words, oods_evals, h_phase_ms, composition_ms);
}

int zkb_stark_prove_host(zkb_ctx* ctx, int n_trees, const int* tree_ncols, const uint32_t* const* h_cols, uint32_t trace_log,
                         zkb_air_program* prog, const uint32_t* scalars, const uint32_t* claimed_sum, const zkb_pcs_config* config,
                         uint32_t* h_out, size_t cap, size_t* n_words, uint32_t* oods_evals, float* h_phase_ms, float* composition_ms) {
    zkb_stark_component c{prog, trace_log, scalars, claimed_sum};
    return stark_prove_impl(ctx, n_trees, tree_ncols, nullptr, h_cols, 1, &c, config, h_out, cap, n_words, oods_evals, h_phase_ms, composition_ms);
}

int zkb_pcs_prove_host(zkb_ctx* ctx, int n_trees, const int* tree_ncols, const uint32_t* const* h_cols, const uint32_t* col_logs,
                       const zkb_pcs_config* config, int two_sample_every, uint32_t* h_out, size_t cap, size_t* n_words,
                       float* h_phase_ms) {
    return pcs_prove_impl(ctx, n_trees, tree_ncols, nullptr, h_cols, col_logs, config, two_sample_every, h_out, cap, n_words, h_phase_ms);
}

int zkb_gkr_prove_device(zkb_ctx* ctx, int n_inst, const int* kinds, const uint32_t* const* d_nums, const uint32_t* const* d_dens,
                         const uint64_t* ns, uint64_t seed, uint32_t* h_out, size_t cap, size_t* n_words) {
    if (!ctx) return ZKB_EINVAL;
    if (n_inst <= 0 || !kinds || !d_nums || !d_dens || !ns || !h_out || !n_words) return ZKB_EINVAL;
    try {
        Device dev(ctx);
        for (int i = 0; i < n_inst; i++)
            if (kinds[i] < 0 || kinds[i] > 3 || ns[i] < 1 || (ns[i] & (ns[i] - 1))) return ZKB_EINVAL;
        auto layers = [&] {
            std::vector<Layer> v;
            for (int i = 0; i < n_inst; i++) v.push_back(layer_view(dev, kinds[i], d_nums[i], d_dens[i], ns[i]));
            return v;
        };
        Channel ch;
        ch.mix_u64(seed);
        std::vector<uint32_t> w;
        // Two drivers give the same proof. With everything on the device a layer costs no host round trip, but its masks and claims are
        // hashed there, some 2.3 us an instance, its small layers are one CTA's and an instance's large rounds are launches of their
        // own; the batch driver takes a layer's rounds of all instances in one launch and some 40 us of host time. Measured
        // (resident / batch, us): one instance of 2^12 457 / 748, of 2^22 2,266 / 2,787; two of 2^12 710 / 760, of 2^14 1,023 / 1,004, of 2^20
        // 2,691 / 2,176; three of 2^8 373 / 404, of 2^12 784 / 778; four of 2^8 425 / 405. ZKB_GKR_DRIVER=resident|batch overrides the choice.
        uint64_t tallest = 0;
        for (int i = 0; i < n_inst; i++) tallest = std::max(tallest, ns[i]);
        bool resident = gkr_resident_supported(n_inst, ns) && (n_inst == 1 || (n_inst <= 3 && tallest <= (uint64_t)1 << 12));
        if (const char* pick = getenv("ZKB_GKR_DRIVER")) {
            if (!strcmp(pick, "resident")) resident = gkr_resident_supported(n_inst, ns);
            else if (!strcmp(pick, "batch")) resident = false;
        }
        if (resident) {
            // the transcript stays on the device: no host round trip per sum-check round
            uint32_t dg[8], nd = ch.n_draws();
            for (int k = 0; k < 8; k++) dg[k] = ch.digest()[k];
            int rc = gkr_prove_resident(ctx, layers(), dg, &nd, w);
            if (rc) return rc;
            HashWords hw;
            for (int k = 0; k < 8; k++) hw[k] = dg[k];
            ch.set_state(hw, nd);
        } else {
            w = gkr_prove_batch(dev, ch, layers());
        }
        w.insert(w.end(), ch.digest().begin(), ch.digest().end());
        *n_words = w.size();
        if (w.size() > cap) return zk_set_error_public(ctx, ZKB_EINVAL, "zkb_gkr_prove: output buffer too small");
        memcpy(h_out, w.data(), w.size() * 4);
        HostClock::dump("zkb_gkr_prove_device");
        return ZKB_OK;
    } catch (const Error& e) {
        return zk_set_error_public(ctx, e.code, e.what());
    } catch (const std::exception& e) {
        return zk_set_error_public(ctx, ZKB_ENOMEM, e.what());
    }
}

}  // extern "C"
