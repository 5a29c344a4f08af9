// Witness generation on the device, three more families: the shared bf16 tables' preprocessed columns and their
// multiplicity columns, the key tile's layout flags and selector columns, and the residual-stream component.
// Everything is written in committed order (natural row j lands at index coset_perm(j), prover/src/common.rs:76-80).
//
// Host statements these replace: bf16::norm_table / mul_table (prover/src/bf16.rs:130-158, 264-281), the fraction table
// (prover/src/gadgets/residual_stream/mod.rs:1116-1122), the key tile's row predicates
// (prover/src/gadgets/attention/trace.rs:742-790) and residual_stream_component
// (prover/src/gadgets/residual_stream/mod.rs:1418-1760). The reference's device originals are zk_witness_gen_pre_table and
// zk_witness_gen_sel (stwo_cuda/cuda/zk_pre_witness_gen.cu), zk_flags_key_tile (stwo_cuda/cuda/zk_acc.cu:78-97) and
// zk_witness_gen_residual_stream (stwo_cuda/cuda/zk_residual_stream_witness_gen.cu). Their "mutate" arguments
// (deliberate defects for negative controls) are not part of the operators and are not built.
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "count_cache.cuh"

namespace zk {

namespace {

constexpr uint32_t OFF_TABLE = 0xffffffffu;

__device__ __forceinline__ uint32_t committed_to_natural(uint32_t i, uint32_t log_n) {
    uint32_t c = (i & 1u) ? (((2u << log_n) - i - 1u) >> 1) : (i >> 1);
    return __brev(c) >> (32u - log_n);
}
__device__ __forceinline__ uint32_t field_of(long long v) {  // ((v % p) + p) % p, encoding.rs:29-32
    // two folds of 31 bits bring any |v| < 2^62 below 2p (2^31 = 1 mod p); no 64-bit division
    unsigned long long u = (unsigned long long)(v < 0 ? -v : v);
    u = (u & P) + (u >> 31);
    u = (u & P) + (u >> 31);
    uint32_t r = (uint32_t)u;
    if (r >= P) r -= P;
    return (v < 0 && r) ? P - r : r;
}
__device__ __forceinline__ long long signed_of(uint32_t v) { return v > P / 2 ? (long long)v - (long long)P : (long long)v; }

// ---------------------------------------------------------------------------------------------------
// The shared tables. Every row is a function of its own index; no table is uploaded.
// ---------------------------------------------------------------------------------------------------
struct PreCfg {
    uint32_t kind, log_rows, real_rows, kmax, round, sticky, n_cols, n_counters;
};

// One rounding step of an 8-bit significand m in [128, 256) with round bit rb and sticky flag st: the significand
// field (m7) and whether the step carried into the next binade (bf16.rs:81-88 and the renormalisation at :146).
__device__ __forceinline__ void round_significand(uint32_t round, uint32_t m, uint32_t rb, uint32_t st, uint32_t& m7, uint32_t& binade_up) {
    uint32_t up = round == 0 ? (rb & (st | (m & 1u))) : round == 1 ? rb : 0u;
    uint32_t sig = m + up;
    binade_up = sig >> 8;              // 256 only from m = 255 with a carry
    m7 = binade_up ? 0u : sig - 128u;  // 256 renormalises to significand 128
}

template <uint32_t KIND>
__device__ __forceinline__ void table_row(const PreCfg& c, uint32_t d, uint32_t (&o)[6]) {
#pragma unroll
    for (int k = 0; k < 6; k++) o[k] = 0;
    if (KIND == 3) { o[0] = d; o[1] = d != 0; return; }  // q != 0 indicator
    if (KIND == 4) { o[0] = d; return; }                 // a range table is its own index
    if (d >= c.real_rows) return;                        // past the table's own length: zero rows
    if (KIND == 0) {                                     // normalisation: (m2, ph, st, m7, expfield, nz)
        if (d == 0) return;
        if (d < 256u) {  // an integer below 256 is exactly representable: its top bit gives the binade, the rest the fraction
            uint32_t t = 31u - __clz(d);
            o[0] = d; o[1] = 1; o[3] = (d << (7u - t)) - 128u; o[4] = 127u + t; o[5] = 1;
            return;
        }
        uint32_t per_k = 256u << c.sticky, idx = d - 256u, k = idx / per_k, rem = idx - k * per_k;
        uint32_t m2 = 256u + (rem >> c.sticky), st = c.sticky ? (rem & 1u) : 0u, m7, up;
        round_significand(c.round, m2 >> 1, m2 & 1u, st, m7, up);
        o[0] = m2; o[1] = 1u << k; o[2] = st; o[3] = m7; o[4] = k + 1u + up + 134u; o[5] = 1;
        return;
    }
    if (KIND == 1) {  // fraction: (2^k, r, sticky && r != 0) for 2^k <= d < 2^(k+1)
        if (d == 0) return;
        uint32_t k = 31u - __clz(d), r = d - (1u << k);
        o[0] = 1u << k; o[1] = r; o[2] = (c.sticky && r != 0) ? 1u : 0u;
        return;
    }
    // multiply: (a, b, m7, carry) of the significand product (128 + a)(128 + b), a 16-bit integer in [2^14, 2^16)
    uint32_t a = d >> 7, b = d & 127u, p = (128u + a) * (128u + b), carry = p >> 15, shift = 7u + carry, m7, up;
    round_significand(c.round, p >> shift, (p >> (shift - 1u)) & 1u, (p & ((1u << (shift - 1u)) - 1u)) != 0, m7, up);
    o[0] = a; o[1] = b; o[2] = m7; o[3] = carry + up;
}

// One thread per PAIR of committed rows 2q, 2q+1 (natural rows brev(q) and its complement): 8-byte stores per column.
template <uint32_t KIND>
__global__ void __launch_bounds__(256) pre_table_kernel(const uint32_t* const* __restrict__ counters, uint32_t* const* __restrict__ cols,
                                                        uint32_t* __restrict__ m_col, PreCfg c) {
    const uint32_t L = c.log_rows, q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >> (L - 1)) return;
    const uint32_t j0 = __brev(q) >> (32u - L), j1 = (~j0) & ((1u << L) - 1u);
    uint32_t r0[6], r1[6];
    table_row<KIND>(c, j0, r0);
    table_row<KIND>(c, j1, r1);
#pragma unroll
    for (uint32_t k = 0; k < 6; k++)
        if (k < c.n_cols) reinterpret_cast<uint2*>(cols[k])[q] = make_uint2(r0[k], r1[k]);
    if (m_col) {  // the multiplicities: every component that bumped this table kept a counter of its own; the column is their sum
        uint32_t s0 = 0, s1 = 0;
        for (uint32_t k = 0; k < c.n_counters; k++) {
            const uint32_t* cnt = counters[k];
            s0 += __ldg(cnt + j0);
            s1 += __ldg(cnt + j1);
        }
        reinterpret_cast<uint2*>(m_col)[q] = make_uint2(s0, s1);
    }
}

// Rows where this run's own table is not the closed form (the reference's corrupted-table probe; empty otherwise).
__global__ void pre_patch_kernel(const uint32_t* __restrict__ idx, const uint32_t* __restrict__ val, uint32_t n, uint32_t* const* __restrict__ cols,
                                 uint32_t n_cols, uint32_t log_rows) {
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    uint32_t i = committed_to_natural(idx[t], log_rows);  // the permutation is an involution
    for (uint32_t k = 0; k < n_cols; k++) cols[k][i] = val[(size_t)t * n_cols + k];
}

// ---------------------------------------------------------------------------------------------------
// Key tile: per-row layout flags (natural order) and the selector columns built from them (committed order).
// ---------------------------------------------------------------------------------------------------
constexpr uint32_t F_ACTIVE = 1, F_NOFIRST = 2, F_LAST = 4, F_ISTART = 8;
struct TileGrid {
    uint32_t log_rows, groups, chunks, lead, descending;
};
__device__ __forceinline__ bool tile_row(const TileGrid& g, uint32_t j, uint32_t& grp, uint32_t& chunk) {  // layout.rs:141-183
    if (j < g.lead) return false;
    uint32_t idx = j - g.lead, gi = idx / g.chunks;
    grp = g.descending ? g.groups - 1u - gi : gi;
    chunk = g.chunks - 1u - (idx - gi * g.chunks);
    return true;
}
__global__ void tile_flags_kernel(uint32_t* __restrict__ flags, uint32_t shape, TileGrid g, uint32_t modulus, uint32_t rw) {
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x, rows = 1u << g.log_rows;
    if (j >= rows) return;
    uint32_t f = 0;
    if (shape == 2) {  // per-token component: every row active, an instance starts where the row's highest token is S-1 mod S
        unsigned long long hi = (unsigned long long)(rows - 1u - j) * rw + rw;
        f = F_ACTIVE | (j > 0 ? F_NOFIRST : 0u) | ((j > 0 && hi % modulus == 0) ? F_ISTART : 0u);
    } else {
        uint32_t grp = 0, chunk = 0;
        if (tile_row(g, j, grp, chunk)) {
            f = F_ACTIVE | (chunk + 1u < g.chunks ? F_NOFIRST : 0u) | (chunk == 0 ? F_LAST : 0u);
            if (j > 0 && chunk + 1u == g.chunks && grp % modulus == modulus - 1u) f |= F_ISTART;
        }
    }
    flags[j] = f;
}

struct SelCfg {
    uint32_t shape;  // 0 channel, 1 key, 2 per-token
    TileGrid g;
    uint32_t ctx, with_scale, n_cols;
};
__global__ void selectors_kernel(const uint32_t* __restrict__ flags, const uint32_t* __restrict__ scale, uint32_t* const* __restrict__ cols, SelCfg c) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, rows = 1u << c.g.log_rows;
    if (i >= rows) return;
    uint32_t j = committed_to_natural(i, c.g.log_rows), f = __ldg(flags + j);
    uint32_t act = f & F_ACTIVE ? 1u : 0u, nofirst = f & F_NOFIRST ? 1u : 0u, last = f & F_LAST ? 1u : 0u, istart = f & F_ISTART ? 1u : 0u;
    uint32_t pos = j > 0, end = j + 1u == rows;
    if (c.shape == 2) { cols[0][i] = pos; cols[1][i] = end; cols[2][i] = istart; return; }
    cols[0][i] = nofirst; cols[1][i] = last; cols[2][i] = pos; cols[3][i] = end;
    if (c.shape == 0) { cols[4][i] = istart; return; }
    cols[4][i] = pos & (last ^ 1u); cols[5][i] = pos & last; cols[6][i] = istart;
    uint32_t sc = 1;  // the master exp table's key scale, inverted, per instance; an inert row takes 1
    if (c.with_scale) {
        uint32_t grp = 0, chunk = 0;
        if (tile_row(c.g, j, grp, chunk)) sc = __ldg(scale + grp / c.ctx);
    }
    cols[7][i] = sc;
    if (c.n_cols > 8) cols[8][i] = act;
}


// ---------------------------------------------------------------------------------------------------
// The residual-stream component: a row is a small program over bf16 values held as (signed significand, exponent
// field) pairs: committed leaves (optionally with a tabulated unary image), then slots that each add or multiply two
// earlier values with one bf16 rounding, every intermediate being a committed cell and every table read a counted
// lookup. One thread owns one committed row. A slot's operands are cells the same thread wrote earlier, read back
// from the columns (plain loads, program order), so no per-row state is kept however long the program is.
// ---------------------------------------------------------------------------------------------------
struct RsGroup { uint32_t n, leaf_col, width, un, flat; };
struct RsSlot { uint32_t a_sm, a_ef, b_sm, b_ef, base, o_sm, o_ef, from_slot; };
using RsMult = CountTable;
struct RsArgs {
    const uint32_t* wit;
    const RsGroup* groups;
    const RsSlot* slots;
    const uint32_t* norm3;
    const int32_t* smul3;
    const int32_t* const* un2;
    const uint32_t* out_slot;
    const uint32_t* level_start;  // the slots lie level by level: n_levels + 1 offsets
    uint32_t* const* cols;
    uint32_t* col0;               // evenly spaced columns: the first one, and the distance in words
    long long col_step;
    uint32_t* out_pat;
    int32_t* out_nat;
    int32_t* in_nat;
    RsMult m_pow, m_norm, m_val, m_frac, m_smul;
    const RsMult* m_un;
    uint32_t* counts;
    uint32_t n_norm, n_smul, n_val, log_rows, live, n_groups, n_leaves, n_slots, n_levels, kmax, out_w, teams, flush_every, leaves_by_four, outs_by_four;
};
constexpr uint32_t RS_DMAX = 12, RS_UMIN = 260, RS_BIAS = 134, RS_POW_ROWS = RS_DMAX + 1 + RS_UMIN;

// One lookup: bump the table's multiplicity, or count the lookup as off the table (OFF_TABLE is larger than any table).
__device__ __forceinline__ void lookup(const RsMult& t, uint32_t idx, uint32_t& off) {
    if (idx >= t.n) off++; else count_in_memory(t.m, idx);
}
template <int LOG>
__device__ __forceinline__ void lookup(uint32_t* cache, const RsMult& t, uint32_t idx, uint32_t& off, bool whole = false) {
    if (idx >= t.n) off++; else count_cached<LOG>(cache, t.m, idx, whole);
}
template <class I>
__device__ __forceinline__ uint32_t value_index(I sm, I ef) {  // val_table's row order: zero, then (ef, m7, sign)
    if (sm == 0 && ef == 0) return 0;
    const I a = sm < 0 ? -sm : sm;
    if (ef <= 0 || ef >= 0xff || a < 128 || a >= 256) return OFF_TABLE;
    return 1u + (((uint32_t)ef - 1u) * 128u + (uint32_t)(a - 128)) * 2u + (sm < 0 ? 1u : 0u);
}
template <class I>
__device__ __forceinline__ uint32_t pow_index(I u) {  // [0, DMAX], then [-UMIN, -1]
    if (u >= 0 && u <= (I)RS_DMAX) return (uint32_t)u;
    if (u < 0 && u >= -(I)RS_UMIN) return RS_DMAX + (uint32_t)(-u);
    return OFF_TABLE;
}
__device__ __forceinline__ uint32_t signed_significand_index(long long v) {
    if (v == 0) return 0;
    unsigned long long a = (unsigned long long)(v < 0 ? -v : v);
    return (a < 128 || a >= 256) ? OFF_TABLE : 1u + (v < 0 ? 128u : 0u) + (uint32_t)(a - 128);
}
// Where a column begins. A program's columns usually are one allocation, evenly spaced: their addresses are then computed. Otherwise
// they come from the table, which the kernel never writes: through the read-only path, so that the loads of a slot's
// fourteen column addresses are independent of the stores between them (a plain load would have to be ordered after every
// earlier store, one address at a time).
template <bool EVEN>
__device__ __forceinline__ uint32_t* column(const RsArgs& a, uint32_t c) {
    if (EVEN) return a.col0 + (long long)c * a.col_step;
    return reinterpret_cast<uint32_t*>(__ldg(reinterpret_cast<const unsigned long long*>(a.cols) + c));
}
// A cell as the exponent it encodes, negative ones as 0: no larger than 2^31 for any word, so no sign is needed.
__device__ __forceinline__ uint32_t exponent_of(uint32_t v) { return v <= P / 2 ? v : v < P ? 0u : v - P; }
// An operand's words: its significand cell, and the exponent it encodes. A slot's output exponent is clamped to [0, 0xfe] on the way
// out of the slot while its cell keeps the unclamped value, so the clamp applies to slot sources only.
struct RsOperand {
    uint32_t sm, ef;
    __device__ __forceinline__ int small_sm() const { return (int)(sm <= P / 2 ? sm : sm - P); }  // of an operand that is_small
    __device__ __forceinline__ bool is_small() const { return (uint32_t)(small_sm() + (1 << 17)) < (2u << 17) && ef < (1u << 20); }
};
template <bool EVEN>
__device__ __forceinline__ RsOperand operand(const RsArgs& a, uint32_t i, uint32_t c_sm, uint32_t c_ef, bool from_slot) {
    if (c_sm == OFF_TABLE) return {0u, 0u};
    const uint32_t e = exponent_of(column<EVEN>(a, c_ef)[i]);
    return {column<EVEN>(a, c_sm)[i], from_slot ? umin32(e, 0xfeu) : e};
}

// What an addition writes and which rows of the tables it looks up.
struct RsAddition { uint32_t fa, fb, etop, mag, sg, m2, ph, r, st, m7, ef, nz, c_sm, c_ef, pa, pb, ni, frac, val, lost, bad_exp; };
// Both operands aligned to the larger exponent (a shift of up to DMAX bits is kept, a smaller operand is dropped), added, the magnitude normalised
// to a 9-bit M2 with its round-bit weight ph, rounded through the table. In 32 bits for operands that are small (a significand below 2^17 times
// 2^DMAX) and table rows of less than 2^16, which are all that well-formed tables and cells hold; false for other rows. In 64 bits for any.
template <class I, bool STICKY>
__device__ __forceinline__ bool add_slot(const RsArgs& a, I a_sm, I a_ef, I b_sm, I b_ef, RsAddition& o) {
    constexpr bool WIDE = sizeof(I) == 8;
    const I etop = a_ef > b_ef ? a_ef : b_ef, ua = a_ef - etop + (I)RS_DMAX, ub = b_ef - etop + (I)RS_DMAX;
    o.pa = pow_index(ua);
    o.pb = pow_index(ub);
    o.fa = ua >= 0 ? 1u << ua : 0u;
    o.fb = ub >= 0 ? 1u << ub : 0u;
    const I acc = a_sm * (I)o.fa + b_sm * (I)o.fb, mag = acc < 0 ? -acc : acc;
    I r = 0;
    uint32_t k = 0;
    o.sg = acc < 0;
    o.m2 = o.ph = o.st = o.lost = 0;
    if (mag) {
        const uint32_t bits = WIDE ? 64u - (uint32_t)__clzll((long long)mag) : 32u - (uint32_t)__clz((int)mag);
        k = bits > 9u ? bits - 9u : 0u;
        if (k > a.kmax) o.lost = 1;  // a round-bit weight the table does not carry
        else { o.ph = 1u << k; o.m2 = (uint32_t)(mag >> k); r = mag & (((I)1 << k) - 1); o.st = STICKY && r != 0; }
    }
    // the normalisation table's row: zero row, 255 exact small magnitudes, then (k, m2, st) ascending
    if (o.m2 == 0 && o.ph == 0) o.ni = 0;
    else if (o.ph == 1 && o.m2 < 256u) o.ni = o.m2;
    else if (o.m2 >= 256u && o.m2 < 512u) o.ni = 256u + (k * 256u + (o.m2 - 256u)) * (STICKY ? 2u : 1u) + o.st;
    else o.ni = OFF_TABLE;
    o.m7 = o.ef = o.nz = 0;
    if (o.ni >= a.n_norm) o.lost++;
    else {
        o.m7 = __ldg(a.norm3 + 3 * (size_t)o.ni); o.ef = __ldg(a.norm3 + 3 * (size_t)o.ni + 1); o.nz = __ldg(a.norm3 + 3 * (size_t)o.ni + 2);
        if (!WIDE && (o.m7 >= 1u << 16 || o.ef >= 1u << 16 || o.nz >= 256u)) return false;
    }
    o.frac = o.ph == 0 ? (r == 0 ? 0u : OFF_TABLE) : o.ph + (uint32_t)r;
    const I c_sm = (I)(128u * o.nz + o.m7) * (o.sg ? -1 : 1), c_ef = o.nz == 1 ? (I)o.ef + etop - (I)(RS_DMAX + RS_BIAS) : 0;
    o.bad_exp = o.nz == 1 && !(c_ef >= 1 && c_ef < 0xff);
    o.val = (c_ef >= 0 && c_ef < 0xff) ? value_index(c_sm, c_ef) : OFF_TABLE;  // the slot's own output is a looked-up pair too
    if (WIDE) {
        o.etop = field_of(etop); o.mag = field_of(mag); o.r = field_of(r); o.c_sm = field_of(c_sm); o.c_ef = field_of(c_ef);
    } else {
        o.etop = (uint32_t)etop; o.mag = (uint32_t)mag; o.r = (uint32_t)r;
        o.c_sm = c_sm < 0 ? (uint32_t)(c_sm + (I)P) : (uint32_t)c_sm;
        o.c_ef = c_ef < 0 ? (uint32_t)(c_ef + (I)P) : (uint32_t)c_ef;
    }
    return true;
}
template <bool STICKY>
__device__ __noinline__ void add_slot_wide(const RsArgs& a, RsOperand x, RsOperand y, RsAddition* o) {
    add_slot<long long, STICKY>(a, signed_of(x.sm), (long long)x.ef, signed_of(y.sm), (long long)y.ef, *o);
}

// A team of warps owns 32 consecutive committed rows at a time: lane = row, so that every column access of a warp is one 128-byte
// line. The warps share the rows' work: the leaves, then the slots level by level (a level holds the slots whose operands are
// leaves or outputs of earlier levels), with a barrier of the team between levels, since a slot's operand may be a cell
// another warp of the team wrote.
//
// What bounded it were the counts (count_cache.cuh), then the latency of a slot, a chain of loads (its record, the operands' cells, a
// row of the table) before its stores, then its instructions, 990 a slot with its two leaves. So one CTA an SM keeps the counters and takes rows until none
// are left, in two teams of sixteen warps; column addresses are computed where they can be (fourteen of them were 28 registers), four leaves are loaded at a
// time, additions are worked out in 32 bits, the power table's one busy row is counted in a register, tables that have a counter a row need no tags (of the
// fraction table's 2^14 rows a third of the lookups went to memory while they shared 2^12 counters), a slot's operands are asked for a slot before.
// 2^15 rows of 128 additions: 690 us with the counts as atomics in L2, 257 us with them in shared memory, 204 us with four leaves or outputs of a row to
// an access, 170 us as it is now (650 instructions a slot, issue slots at 46 %, the LSU's data path too). The normalisation table in shared memory, a word
// a row, gained nothing (173). 2^13 rows: 53 -> 48 us; four teams of eight warps instead of two of sixteen: 193.
constexpr uint32_t RS_LANES = 16, RS_TEAMS = 2, RS_LEAVES = 4;
constexpr int RS_VAL_LOG = 13, RS_NORM_LOG = 13, RS_FRAC_LOG = 14, RS_FRAC_FEW_LOG = 12, RS_SMUL_LOG = 14;
constexpr uint32_t RS_MUL_WORDS = (1u << RS_VAL_LOG) + (1u << RS_SMUL_LOG);
constexpr uint32_t rs_add_words(int frac_log) { return (1u << RS_VAL_LOG) + (1u << RS_NORM_LOG) + (1u << frac_log); }
// From how many additions a CTA on the fraction table has 2^RS_FRAC_LOG counters: those are 48 KB more to clear and to look through at the end, a microsecond.
// With 2^12 and with 2^14, kmax 13: 2^13 rows of 4 additions, 256 a CTA: 18.1 and 19.4 us; 2^14 rows, 443 a CTA: 25.0 and 24.1; 32 rows of 128, 4,096: 40.7 and 38.4;
// 2^15 rows of 128: 179 and 176.
constexpr uint64_t RS_FRAC_ADDITIONS = 384;
template <bool MUL, bool STICKY, bool EVEN, int FRAC_LOG>
__global__ void __launch_bounds__(32 * RS_LANES * RS_TEAMS, 1) residual_stream_kernel(const __grid_constant__ RsArgs a) {
    // The power table has 273 rows and every addition hits row DMAX with its larger operand: that row is counted in a register, the others per CTA in
    // shared memory, and added to the global array once at the end.
    __shared__ uint32_t pow_hist[RS_POW_ROWS];
    extern __shared__ __align__(16) uint32_t counts_sm[];
    uint32_t *const val_counts = counts_sm, *const norm_counts = counts_sm + (1u << RS_VAL_LOG), *const frac_counts = norm_counts + (1u << RS_NORM_LOG);
    uint32_t* const smul_counts = norm_counts;  // a program adds or multiplies
    const bool norm_whole = count_is_whole<RS_NORM_LOG>(a.m_norm), frac_whole = count_is_whole<FRAC_LOG>(a.m_frac);
    count_clear<RS_VAL_LOG>(val_counts, false, threadIdx.x, blockDim.x);
    if (MUL) count_clear<RS_SMUL_LOG>(smul_counts, false, threadIdx.x, blockDim.x);
    else {
        count_clear<RS_NORM_LOG>(norm_counts, norm_whole, threadIdx.x, blockDim.x);
        count_clear<FRAC_LOG>(frac_counts, frac_whole, threadIdx.x, blockDim.x);
    }
    for (uint32_t k = threadIdx.x; k < RS_POW_ROWS; k += blockDim.x) pow_hist[k] = 0;
    __syncthreads();
    auto flush = [&](uint32_t thread, uint32_t threads) {
        count_flush<RS_VAL_LOG>(val_counts, a.m_val.m, thread, threads);
        if (MUL) count_flush<RS_SMUL_LOG>(smul_counts, a.m_smul.m, thread, threads);
        else {
            count_flush<RS_NORM_LOG>(norm_counts, a.m_norm.m, thread, threads);
            count_flush<FRAC_LOG>(frac_counts, a.m_frac.m, thread, threads);
        }
    };
    const uint32_t lanes = blockDim.x / (32u * a.teams), team = (threadIdx.x >> 5) / lanes, t = (threadIdx.x >> 5) - team * lanes;
    auto team_sync = [&] {
        __syncwarp();  // lanes without a row come here by another way than those with one, and the barrier takes whole warps
        asm volatile("bar.sync %0, %1;" ::"r"(team + 1u), "r"(32u * lanes) : "memory");
    };
    uint32_t off = 0, bad_exp = 0, un_off = 0, top = 0, since_flush = 0;
    // (a CTA's first team takes its rows before any CTA's second: what is left for a last pass is one team's a CTA)
    for (uint32_t block = blockIdx.x + gridDim.x * team; (block << 5 >> a.log_rows) == 0; block += gridDim.x * a.teams) {
    const uint32_t i = block * 32u + (threadIdx.x & 31u);
    const bool in_range = (i >> a.log_rows) == 0;
    const uint32_t j = in_range ? committed_to_natural(i, a.log_rows) : 0u;
    const bool live = j < a.live;
    const size_t leaf0 = (size_t)j * a.n_leaves;

    if (in_range)
    for (uint32_t g = 0; g < a.n_groups; g++) {
        const RsGroup gr = a.groups[g];
        for (uint32_t k0 = t * RS_LEAVES; k0 < gr.n; k0 += lanes * RS_LEAVES) {
            // What is in natural row order lies n_leaves words apart from lane to lane: a sector a lane and access, whatever its width.
            const size_t at = leaf0 + gr.flat + k0;
            const bool four = a.leaves_by_four && k0 + RS_LEAVES <= gr.n;
            uint32_t pats[RS_LEAVES];
            if (four) {
                const uint4 p = live ? __ldg(reinterpret_cast<const uint4*>(a.wit + at)) : make_uint4(0u, 0u, 0u, 0u);
                pats[0] = p.x; pats[1] = p.y; pats[2] = p.z; pats[3] = p.w;
            } else {
#pragma unroll
                for (uint32_t u = 0; u < RS_LEAVES; u++) pats[u] = live && k0 + u < gr.n ? __ldg(a.wit + at + u) : 0u;
            }
            int2 held = make_int2(0, 0);
#pragma unroll
            for (uint32_t u = 0; u < RS_LEAVES; u++) {
                const uint32_t k = k0 + u, pat = pats[u];
                if (k >= gr.n) break;
                // a bf16 pattern as (sm, ef); both zeros, infinities and NaNs collapse to (0, 0)
                const uint32_t e = (pat >> 7) & 0xffu;
                const bool finite = e != 0 && e != 0xffu;
                const int mag = 128 + (int)(pat & 0x7fu);
                const int sm = finite ? ((pat >> 15) & 1u ? -mag : mag) : 0;
                const uint32_t ef = finite ? e : 0u;
                const uint32_t b = gr.leaf_col + k * gr.width;
                column<EVEN>(a, b)[i] = sm < 0 ? (uint32_t)(sm + (int)P) : (uint32_t)sm;
                column<EVEN>(a, b + 1)[i] = ef;
                if (!four) reinterpret_cast<int2*>(a.in_nat)[at + u] = make_int2(sm, (int)ef);
                else if (u & 1) reinterpret_cast<int4*>(a.in_nat)[(at + u) >> 1] = make_int4(held.x, held.y, sm, (int)ef);
                else held = make_int2(sm, (int)ef);
                const uint32_t v = value_index(sm, (int)ef);
                if (gr.un == 0) { lookup<RS_VAL_LOG>(val_counts, a.m_val, v, off); continue; }
                uint32_t *c2 = column<EVEN>(a, b + 2), *c3 = column<EVEN>(a, b + 3);
                lookup(a.m_un[gr.un - 1], v, off);
                int2 img = make_int2(0, 0);  // the unary image, tabulated over the value table's rows
                if (v < a.n_val) img = __ldg(reinterpret_cast<const int2*>(a.un2[gr.un - 1]) + v);
                else un_off++;
                c2[i] = field_of(img.x);
                c3[i] = field_of(img.y);
            }
        }
    }

    for (uint32_t level = 0; level < a.n_levels; level++) {
      team_sync();
      if (!in_range) continue;
      // A slot's operands are cells of levels before: the next slot's are on their way while this one is worked out, and the record after it.
      const uint32_t end = a.level_start[level + 1];
      uint32_t at = a.level_start[level] + t;
      if (at >= end) continue;
      RsSlot sl = a.slots[at];
      RsOperand x = operand<EVEN>(a, i, sl.a_sm, sl.a_ef, sl.from_slot & 1u), y = operand<EVEN>(a, i, sl.b_sm, sl.b_ef, sl.from_slot & 2u);
      uint32_t b = sl.base;
      if (at + lanes < end) sl = a.slots[at + lanes];
      while (true) {
        RsOperand next_x{0u, 0u}, next_y{0u, 0u};
        const uint32_t next_b = sl.base;
        if (at + lanes < end) {
            next_x = operand<EVEN>(a, i, sl.a_sm, sl.a_ef, sl.from_slot & 1u);
            next_y = operand<EVEN>(a, i, sl.b_sm, sl.b_ef, sl.from_slot & 2u);
        }
        if (at + 2 * lanes < end) sl = a.slots[at + 2 * lanes];
        uint32_t* const first = EVEN ? column<EVEN>(a, b) + i : nullptr;
        auto put = [&](uint32_t k, uint32_t v) { (EVEN ? first + (long long)k * a.col_step : column<EVEN>(a, b + k) + i)[0] = v; };
        if (!MUL) {
            RsAddition o;
            if (!(x.is_small() && y.is_small() && add_slot<int, STICKY>(a, x.small_sm(), (int)x.ef, y.small_sm(), (int)y.ef, o))) {
                RsAddition wide;
                add_slot_wide<STICKY>(a, x, y, &wide);
                o = wide;
            }
            constexpr uint32_t kk = STICKY ? 9u : 8u;
            put(0, o.fa); put(1, o.fb); put(2, o.etop); put(3, o.mag); put(4, o.sg); put(5, o.m2); put(6, o.ph); put(7, o.r);
            if (STICKY) put(8, o.st);
            put(kk, o.m7); put(kk + 1, o.ef); put(kk + 2, o.nz); put(kk + 3, o.c_sm); put(kk + 4, o.c_ef);
            off += o.lost;
            bad_exp += o.bad_exp;
            for (const uint32_t u : {o.pa, o.pb}) {
                if (u >= a.m_pow.n) off++;
                else if (u == RS_DMAX) top++;
                else atomicAdd(pow_hist + u, 1u);
            }
            lookup<RS_NORM_LOG>(norm_counts, a.m_norm, o.ni, off, norm_whole);
            lookup<FRAC_LOG>(frac_counts, a.m_frac, o.frac, off, frac_whole);
            lookup<RS_VAL_LOG>(val_counts, a.m_val, o.val, off);
        } else {
            // the signed significands' correctly rounded product and binade carry come from one table row
            const uint32_t ia = signed_significand_index(signed_of(x.sm)), ib = signed_significand_index(signed_of(y.sm));
            const uint32_t si = (ia == OFF_TABLE || ib == OFF_TABLE) ? OFF_TABLE : ia * 257u + ib;
            int32_t prod = 0, cy = 0, nzc = 0;
            if (si < a.n_smul) { prod = __ldg(a.smul3 + 3 * (size_t)si); cy = __ldg(a.smul3 + 3 * (size_t)si + 1); nzc = __ldg(a.smul3 + 3 * (size_t)si + 2); }
            else off++;
            lookup<RS_SMUL_LOG>(smul_counts, a.m_smul, si, off);
            const long long c_sm = prod, c_ef = nzc == 1 ? (long long)x.ef + y.ef + cy - 127 : 0;
            bad_exp += nzc == 1 && !(c_ef >= 1 && c_ef < 0xff);
            put(0, field_of(c_sm));
            put(1, (uint32_t)cy);
            put(2, (uint32_t)nzc);
            put(3, field_of(c_ef));
            lookup<RS_VAL_LOG>(val_counts, a.m_val, (c_ef >= 0 && c_ef < 0xff) ? value_index(c_sm, c_ef) : OFF_TABLE, off);
        }
        at += lanes;
        if (at >= end) break;
        x = next_x;
        y = next_y;
        b = next_b;
      }
    }
    team_sync();

    // what the bindings and the next component read, in natural row order
    if (in_range)
    for (uint32_t k0 = t * 4; k0 < a.out_w; k0 += lanes * 4) {
        uint32_t pats[4];
        int2 held = make_int2(0, 0);
        const size_t at = (size_t)j * a.out_w + k0;
        const bool four = a.outs_by_four;
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            if (k0 + u >= a.out_w) break;
            const RsSlot sl = a.slots[a.out_slot[k0 + u]];
            // (as words: of the magnitude the low bits count, and what is below 0 is known from the cell)
            const uint32_t c_sm = column<EVEN>(a, sl.o_sm)[i], c_ef = column<EVEN>(a, sl.o_ef)[i];
            const uint32_t sm = c_sm > P / 2 ? c_sm - P : c_sm, e = c_ef > P / 2 ? c_ef - P : c_ef;
            const bool negative = c_sm > P / 2 && c_sm < P;
            uint32_t pat = 0;
            if (sm != 0) pat = ((negative ? 1u << 15 : 0u) | (umin32(exponent_of(c_ef), 0xfeu) << 7) | ((negative ? 0u - sm : sm) - 128u)) & 0xffffu;
            pats[u] = pat;
            if (!four) {
                a.out_pat[at + u] = pat;
                reinterpret_cast<int2*>(a.out_nat)[at + u] = make_int2((int)sm, (int)e);
            } else if (u & 1) {
                reinterpret_cast<int4*>(a.out_nat)[(at + u) >> 1] = make_int4(held.x, held.y, (int)sm, (int)e);
            } else {
                held = make_int2((int)sm, (int)e);
            }
        }
        if (four) *reinterpret_cast<uint4*>(a.out_pat + at) = make_uint4(pats[0], pats[1], pats[2], pats[3]);
    }
    team_sync();  // the next rows' cells are other memory, but a warp must not be two passes ahead of its team's barrier
    if (++since_flush == a.flush_every) {
        flush(threadIdx.x - team * 32u * lanes, 32u * lanes);
        since_flush = 0;
    }
    }
    __syncthreads();
    flush(threadIdx.x, blockDim.x);
    if (!MUL)
        for (uint32_t k = threadIdx.x; k < RS_POW_ROWS && k < a.m_pow.n; k += blockDim.x)
            if (pow_hist[k]) atomicAdd(a.m_pow.m + k, pow_hist[k]);
    top = __reduce_add_sync(0xffffffffu, top);
    off = __reduce_add_sync(0xffffffffu, off);
    bad_exp = __reduce_add_sync(0xffffffffu, bad_exp);
    un_off = __reduce_add_sync(0xffffffffu, un_off);
    if ((threadIdx.x & 31u) == 0) {
        if (top) atomicAdd(a.m_pow.m + RS_DMAX, top);
        if (off) atomicAdd(a.counts, off);
        if (bad_exp) atomicAdd(a.counts + 1, bad_exp);
        if (un_off) atomicAdd(a.counts + 2, un_off);
    }
}

}  // namespace
}  // namespace zk

using namespace zk;

namespace {
// Host arrays the kernels index (groups, slots, pointer tables) go up through the context's staging ring, 8 bytes a word.
template <class T> size_t array_slots(size_t n) { return (n * sizeof(T) + 7) / 8 + 1; }
template <class T> int stage_array(zkb_ctx* ctx, const T* src, size_t n, const T** out) {
    std::vector<uint64_t> blob(array_slots<T>(n), 0);
    if (n) memcpy(blob.data(), src, n * sizeof(T));
    void** d = nullptr;
    int rc = stage_ptrs(ctx, reinterpret_cast<const void* const*>(blob.data()), (int)blob.size(), &d);
    *out = reinterpret_cast<const T*>(d);
    return rc;
}
}  // namespace

extern "C" {

int zkb_witness_pre_table(zkb_ctx* ctx, uint32_t kind, uint32_t log_rows, uint32_t kmax, uint32_t round, const uint32_t* const* counters,
                          uint32_t n_counters, const uint32_t* patch_idx, const uint32_t* patch_val, uint32_t n_patch, uint32_t* const* cols,
                          uint32_t n_cols, uint32_t* m_col) {
    if (!ctx) return ZKB_EINVAL;
    static const uint32_t width[5] = {6, 3, 4, 2, 1};
    ZKB_CHECK_ARG(ctx, kind <= 4 && round <= 2 && cols && n_cols == width[kind] && log_rows >= 1 && log_rows <= 30 && kmax <= 21);
    ZKB_CHECK_ARG(ctx, (n_counters == 0 || counters) && n_counters <= 4096 && (n_patch == 0 || (patch_idx && patch_val)));
    ZKB_CHECK_ARG(ctx, m_col == nullptr || ((uintptr_t)m_col & 7) == 0);
    for (uint32_t k = 0; k < n_cols; k++) ZKB_CHECK_ARG(ctx, cols[k] != nullptr && ((uintptr_t)cols[k] & 7) == 0);
    for (uint32_t k = 0; k < n_counters; k++) ZKB_CHECK_ARG(ctx, counters[k] != nullptr);
    const uint32_t sticky = round == 0;
    uint64_t real = kind == 0 ? 256ull + (uint64_t)(kmax + 1) * (256u << sticky) : kind == 1 ? 1ull << (kmax + 1) : kind == 2 ? 1ull << 14 : 1ull << log_rows;
    // The table must fit the committed height (the rows above its own length commit zero).
    ZKB_CHECK_ARG(ctx, real <= (1ull << log_rows));
    DeviceGuard g(ctx);
    void **d_cnt = nullptr, **d_cols = nullptr;
    int rc = stage_reserve(ctx, (size_t)n_cols + n_counters);
    if (rc) return rc;
    rc = stage_ptrs(ctx, (const void* const*)cols, (int)n_cols, &d_cols);
    if (rc) return rc;
    if (n_counters && m_col) {
        rc = stage_ptrs(ctx, (const void* const*)counters, (int)n_counters, &d_cnt);
        if (rc) return rc;
    }
    PreCfg c{kind, log_rows, (uint32_t)real, kmax, round, sticky, n_cols, m_col ? n_counters : 0u};
    const uint32_t pairs = 1u << (log_rows - 1), grid = (pairs + 255) / 256;
    {
        ProfScope prof(ctx, "pre_table_kernel");
        auto cnt = (const uint32_t* const*)d_cnt;
        auto cl = (uint32_t* const*)d_cols;
        switch (kind) {
            case 0: pre_table_kernel<0><<<grid, 256, 0, ctx->stream>>>(cnt, cl, m_col, c); break;
            case 1: pre_table_kernel<1><<<grid, 256, 0, ctx->stream>>>(cnt, cl, m_col, c); break;
            case 2: pre_table_kernel<2><<<grid, 256, 0, ctx->stream>>>(cnt, cl, m_col, c); break;
            case 3: pre_table_kernel<3><<<grid, 256, 0, ctx->stream>>>(cnt, cl, m_col, c); break;
            default: pre_table_kernel<4><<<grid, 256, 0, ctx->stream>>>(cnt, cl, m_col, c); break;
        }
        ZKB_LAUNCH_CHECK(ctx);
    }
    if (n_patch) {
        pre_patch_kernel<<<(n_patch + 255) / 256, 256, 0, ctx->stream>>>(patch_idx, patch_val, n_patch, (uint32_t* const*)d_cols, n_cols, log_rows);
        ZKB_LAUNCH_CHECK(ctx);
    }
    return ZKB_OK;
}

static int check_tile(zkb_ctx* ctx, uint32_t shape, uint32_t log_rows, uint32_t groups, uint32_t chunks, uint32_t lead) {
    ZKB_CHECK_ARG(ctx, shape <= 2 && log_rows <= 30);
    if (shape != 2) ZKB_CHECK_ARG(ctx, groups >= 1 && chunks >= 1 && (uint64_t)groups * chunks + lead == (1ull << log_rows));
    return ZKB_OK;
}

int zkb_key_tile_flags(zkb_ctx* ctx, uint32_t shape, uint32_t log_rows, uint32_t groups, uint32_t chunks, uint32_t lead, uint32_t descending,
                       uint32_t modulus, uint32_t rw, uint32_t* flags) {
    if (!ctx) return ZKB_EINVAL;
    int rc = check_tile(ctx, shape, log_rows, groups, chunks, lead);
    if (rc) return rc;
    ZKB_CHECK_ARG(ctx, flags && modulus >= 1 && (shape != 2 || rw >= 1));
    DeviceGuard g(ctx);
    const uint32_t rows = 1u << log_rows;
    ProfScope prof(ctx, "tile_flags_kernel");
    tile_flags_kernel<<<(rows + 255) / 256, 256, 0, ctx->stream>>>(flags, shape, TileGrid{log_rows, groups, chunks, lead, descending ? 1u : 0u}, modulus, rw);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

int zkb_witness_selectors(zkb_ctx* ctx, uint32_t shape, uint32_t log_rows, uint32_t groups, uint32_t chunks, uint32_t lead, uint32_t descending,
                          const uint32_t* flags, const uint32_t* scale, uint32_t ctx_len, uint32_t n_insts, int with_scale, uint32_t* const* cols,
                          uint32_t n_cols) {
    if (!ctx) return ZKB_EINVAL;
    int rc = check_tile(ctx, shape, log_rows, groups, chunks, lead);
    if (rc) return rc;
    ZKB_CHECK_ARG(ctx, flags && cols && n_cols == (shape == 0 ? 5u : shape == 2 ? 3u : n_cols) && (shape != 1 || n_cols == 8 || n_cols == 9));
    // every group's instance must have a scale entry
    if (shape == 1 && with_scale) ZKB_CHECK_ARG(ctx, scale && ctx_len >= 1 && (groups - 1) / ctx_len < n_insts);
    for (uint32_t k = 0; k < n_cols; k++) ZKB_CHECK_ARG(ctx, cols[k] != nullptr);
    DeviceGuard g(ctx);
    void** d_cols = nullptr;
    rc = stage_ptrs(ctx, (const void* const*)cols, (int)n_cols, &d_cols);
    if (rc) return rc;
    const uint32_t rows = 1u << log_rows;
    SelCfg c{shape, TileGrid{log_rows, groups, chunks, lead, descending ? 1u : 0u}, ctx_len, (shape == 1 && with_scale) ? 1u : 0u, n_cols};
    ProfScope prof(ctx, "selectors_kernel");
    selectors_kernel<<<(rows + 255) / 256, 256, 0, ctx->stream>>>(flags, scale, (uint32_t* const*)d_cols, c);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

int zkb_witness_residual_stream(zkb_ctx* ctx, const zkb_rs_program* prog, const zkb_rs_tables* tables, const uint32_t* wit, uint32_t live_rows,
                                uint32_t log_rows, uint32_t* const* cols, uint32_t n_cols, uint32_t* out_pat, int32_t* out_nat, int32_t* in_nat,
                                const zkb_rs_mults* mults, uint32_t* counts) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, prog && tables && mults && wit && cols && out_pat && out_nat && in_nat && counts && log_rows <= 30);
    const zkb_rs_program& p = *prog;
    ZKB_CHECK_ARG(ctx, p.kind <= 1 && p.sticky <= 1 && p.kmax <= 21 && p.groups && p.n_groups >= 1 && (p.n_slots == 0 || p.slots) && (p.out_w == 0 || p.out_slot));
    ZKB_CHECK_ARG(ctx, live_rows <= (1u << log_rows) && n_cols >= 1 && n_cols <= 65536);
    ZKB_CHECK_ARG(ctx, ((uintptr_t)out_nat & 7) == 0 && ((uintptr_t)in_nat & 7) == 0);
    ZKB_CHECK_ARG(ctx, p.kind == 1 ? (tables->smul3 != nullptr && mults->smul.m != nullptr) : (tables->norm3 != nullptr && mults->pow.m && mults->norm.m && mults->frac.m));
    ZKB_CHECK_ARG(ctx, mults->val.m != nullptr && (tables->n_un == 0 || (tables->un2 && mults->un)));
    // every column index a row touches is checked here, so that the kernel needs no bounds tests
    const uint32_t slot_w = p.kind == 0 ? 13u + p.sticky : 4u;
    uint64_t n_leaves = 0;
    for (uint32_t g = 0; g < p.n_groups; g++) {
        const zkb_rs_group& gr = p.groups[g];
        ZKB_CHECK_ARG(ctx, gr.un <= tables->n_un && gr.width == (gr.un ? 4u : 2u) && gr.flat == n_leaves);
        ZKB_CHECK_ARG(ctx, (uint64_t)gr.leaf_col + (uint64_t)gr.n * gr.width <= n_cols);
        n_leaves += gr.n;
    }
    ZKB_CHECK_ARG(ctx, n_leaves >= 1 && n_leaves <= (1u << 20));
    auto col_ok = [&](uint32_t c) { return c == OFF_TABLE || c < n_cols; };
    for (uint32_t s = 0; s < p.n_slots; s++) {
        const zkb_rs_slot& sl = p.slots[s];
        ZKB_CHECK_ARG(ctx, (uint64_t)sl.base + slot_w <= n_cols && sl.o_sm < n_cols && sl.o_ef < n_cols && sl.from_slot <= 3);
        ZKB_CHECK_ARG(ctx, col_ok(sl.a_sm) && col_ok(sl.b_sm) && (sl.a_sm == OFF_TABLE || sl.a_ef < n_cols) && (sl.b_sm == OFF_TABLE || sl.b_ef < n_cols));
    }
    for (uint32_t k = 0; k < p.out_w; k++) ZKB_CHECK_ARG(ctx, p.out_slot[k] < p.n_slots);
    // Levels: a slot that reads a cell of another slot comes one level after it, and that slot must come earlier in
    // evaluation order (an operand inside a later slot's cells would be read before it is written).
    std::vector<uint32_t> level(p.n_slots, 0), owner(n_cols, OFF_TABLE);
    for (uint32_t s = 0; s < p.n_slots; s++)
        for (uint32_t c = 0; c < slot_w; c++) {
            ZKB_CHECK_ARG(ctx, owner[p.slots[s].base + c] == OFF_TABLE);  // two slots' cells overlap
            owner[p.slots[s].base + c] = s;
        }
    for (uint32_t g = 0; g < p.n_groups; g++)
        for (uint64_t c = p.groups[g].leaf_col; c < (uint64_t)p.groups[g].leaf_col + (uint64_t)p.groups[g].n * p.groups[g].width; c++)
            ZKB_CHECK_ARG(ctx, owner[c] == OFF_TABLE);  // a leaf inside a slot's cells
    uint32_t n_levels = 0;
    for (uint32_t s = 0; s < p.n_slots; s++) {
        const zkb_rs_slot& sl = p.slots[s];
        ZKB_CHECK_ARG(ctx, owner[sl.o_sm] == s && owner[sl.o_ef] == s);
        const uint32_t ops[4] = {sl.a_sm, sl.a_ef, sl.b_sm, sl.b_ef};
        for (int o = 0; o < 4; o++) {
            if (ops[o & 2] == OFF_TABLE || owner[ops[o]] == OFF_TABLE) continue;
            ZKB_CHECK_ARG(ctx, owner[ops[o]] < s);
            level[s] = std::max(level[s], level[owner[ops[o]]] + 1u);
        }
        n_levels = std::max(n_levels, level[s] + 1u);
    }
    // the slots level by level, in their own order within a level (a counting sort)
    std::vector<uint32_t> level_start(n_levels + 1, 0), place(p.n_slots), out_slot(p.out_w);
    for (uint32_t s = 0; s < p.n_slots; s++) level_start[level[s] + 1]++;
    for (uint32_t l = 0; l < n_levels; l++) level_start[l + 1] += level_start[l];
    std::vector<uint32_t> next(level_start.begin(), level_start.end());
    std::vector<zkb_rs_slot> slots(p.n_slots);
    for (uint32_t s = 0; s < p.n_slots; s++) {
        place[s] = next[level[s]]++;
        slots[place[s]] = p.slots[s];
    }
    for (uint32_t k = 0; k < p.out_w; k++) out_slot[k] = place[p.out_slot[k]];
    for (uint32_t u = 0; u < tables->n_un; u++) ZKB_CHECK_ARG(ctx, tables->un2[u] && ((uintptr_t)tables->un2[u] & 7) == 0 && mults->un[u].m);
    for (uint32_t k = 0; k < n_cols; k++) ZKB_CHECK_ARG(ctx, cols[k] != nullptr);
    DeviceGuard g(ctx);
    RsArgs a{};
    void** d_cols = nullptr;
    int rc = stage_reserve(ctx, (size_t)n_cols + array_slots<RsGroup>(p.n_groups) + array_slots<RsSlot>(p.n_slots) + array_slots<uint32_t>(p.out_w) +
                                    array_slots<uint32_t>(level_start.size()) + array_slots<uint32_t*>(tables->n_un) + array_slots<RsMult>(tables->n_un));
    if (rc) return rc;
    rc = stage_ptrs(ctx, (const void* const*)cols, (int)n_cols, &d_cols);
    if (rc) return rc;
    static_assert(sizeof(zkb_rs_group) == sizeof(RsGroup) && sizeof(zkb_rs_slot) == sizeof(RsSlot) && sizeof(zkb_rs_mult) == sizeof(RsMult), "layout");
    if ((rc = stage_array(ctx, reinterpret_cast<const RsGroup*>(p.groups), p.n_groups, &a.groups))) return rc;
    if ((rc = stage_array(ctx, reinterpret_cast<const RsSlot*>(slots.data()), p.n_slots, &a.slots))) return rc;
    if ((rc = stage_array(ctx, out_slot.data(), p.out_w, &a.out_slot))) return rc;
    if ((rc = stage_array(ctx, level_start.data(), level_start.size(), &a.level_start))) return rc;
    if ((rc = stage_array(ctx, tables->un2, tables->n_un, &a.un2))) return rc;
    if ((rc = stage_array(ctx, reinterpret_cast<const RsMult*>(mults->un), tables->n_un, &a.m_un))) return rc;
    a.wit = wit; a.norm3 = tables->norm3; a.smul3 = tables->smul3; a.cols = (uint32_t* const*)d_cols;
    a.out_pat = out_pat; a.out_nat = out_nat; a.in_nat = in_nat; a.counts = counts;
    auto mult = [](const zkb_rs_mult& m) { return RsMult{m.m, m.m ? m.n : 0u}; };
    a.m_pow = mult(mults->pow); a.m_norm = mult(mults->norm); a.m_val = mult(mults->val); a.m_frac = mult(mults->frac); a.m_smul = mult(mults->smul);
    a.n_norm = tables->norm3 ? tables->n_norm : 0; a.n_smul = tables->smul3 ? tables->n_smul : 0; a.n_val = tables->n_val;
    a.log_rows = log_rows; a.live = live_rows; a.n_groups = p.n_groups; a.n_leaves = (uint32_t)n_leaves; a.n_slots = p.n_slots;
    a.kmax = p.kmax; a.out_w = p.out_w; a.n_levels = n_levels;
    // four leaves, or outputs, of a row in one access where all of them start on 16 bytes
    bool by_four = n_leaves % 4 == 0 && ((uintptr_t)wit & 15) == 0 && ((uintptr_t)in_nat & 15) == 0;
    for (uint32_t g = 0; g < p.n_groups; g++) by_four = by_four && p.groups[g].flat % 4 == 0;
    a.leaves_by_four = by_four;
    a.outs_by_four = p.out_w % 4 == 0 && ((uintptr_t)out_pat & 15) == 0 && ((uintptr_t)out_nat & 15) == 0;
    // evenly spaced columns need no table
    bool even = true;
    a.col0 = cols[0];
    a.col_step = n_cols > 1 ? (long long)(reinterpret_cast<intptr_t>(cols[1]) - reinterpret_cast<intptr_t>(cols[0])) / 4 : 0;
    for (uint32_t k = 0; k < n_cols && even; k++) even = cols[k] == cols[0] + (long long)k * a.col_step;
    // 32 rows a team of warps; two teams a CTA and a CTA an SM where there are so many rows, sixteen warps a team (eight where a row
    // has too little for them).
    const uint32_t rows = 1u << log_rows, blocks = (rows + 31) / 32;
    a.teams = blocks > 148 ? RS_TEAMS : 1u;
    const uint32_t grid = std::min((blocks + a.teams - 1) / a.teams, 148u);
    const uint32_t lanes = n_leaves + p.n_slots < 64 ? RS_LANES / 2 : RS_LANES, threads = 32 * lanes * a.teams;
    // A counter holds 2^27 - 1: the teams send them to memory long before one could be full.
    a.flush_every = (uint32_t)std::max<uint64_t>(1, ((uint64_t)1 << 24) / (32 * (n_leaves + p.n_slots)));
    ProfScope prof(ctx, "residual_stream_kernel");
    cudaError_t e = cudaSuccess;
    auto launch = [&](auto kernel, uint32_t words) {
        // the most any call of the kernel takes: another thread's call must not lower it in between
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(4 * words));
        if (e == cudaSuccess) kernel<<<grid, threads, 4 * words, ctx->stream>>>(a);
    };
    auto add = [&](auto frac_log) {
        constexpr int LOG = decltype(frac_log)::value;
        if (p.sticky) even ? launch(residual_stream_kernel<false, true, true, LOG>, rs_add_words(LOG)) : launch(residual_stream_kernel<false, true, false, LOG>, rs_add_words(LOG));
        else even ? launch(residual_stream_kernel<false, false, true, LOG>, rs_add_words(LOG)) : launch(residual_stream_kernel<false, false, false, LOG>, rs_add_words(LOG));
    };
    if (p.kind == 1) even ? launch(residual_stream_kernel<true, false, true, 0>, RS_MUL_WORDS) : launch(residual_stream_kernel<true, false, false, 0>, RS_MUL_WORDS);
    else if ((uint64_t)rows * p.n_slots < grid * RS_FRAC_ADDITIONS) add(std::integral_constant<int, RS_FRAC_FEW_LOG>{});
    else add(std::integral_constant<int, RS_FRAC_LOG>{});
    ZKB_CUDA(ctx, e);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

}  // extern "C"
