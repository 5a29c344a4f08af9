// Multiplicities counted per CTA in shared memory before they reach the global tables.
//
// A witness generator looks up a handful of tables millions of times, most often in a few thousand rows of them: as
// atomics in L2 the counts bound it (2^15 rows of 128 additions, 21 million lookups: 450 of 690 us). The tables are larger than shared
// memory, so a CTA keeps 2^LOG counters that serve whichever rows come first: row r's counter is r mod 2^LOG, which holds the
// quotient's tag from its first lookup on; a row that finds another's tag there is counted in memory as before.
#pragma once
#include "common.cuh"

namespace zk {

struct CountTable { uint32_t* m; uint32_t n; };  // a table's global counters

constexpr uint32_t COUNT_TAG_SHIFT = 27, COUNT_MASK = (1u << COUNT_TAG_SHIFT) - 1u;

// Lanes of a warp that hit the same entry are merged into one atomic.
__device__ __forceinline__ void count_in_memory(uint32_t* m, uint32_t idx) {
    uint32_t peers = __match_any_sync(__activemask(), idx);
    if ((threadIdx.x & 31u) == (uint32_t)(__ffs(peers) - 1)) atomicAdd(m + idx, (uint32_t)__popc(peers));
}

// A table of at most 2^LOG rows has a counter a row, and every counter its tag from the start: a lookup is one addition.
template <int LOG>
__device__ __forceinline__ bool count_is_whole(const CountTable& t) { return t.n <= (1u << LOG); }
// (four counters at a time: a call of few rows spends most of its time here; cache: 16-byte aligned)
template <int LOG>
__device__ __forceinline__ void count_clear(uint32_t* cache, bool whole, uint32_t thread, uint32_t threads) {
    const uint32_t v = whole ? 1u << COUNT_TAG_SHIFT : 0u;
    for (uint32_t k = thread; k < (1u << LOG) / 4; k += threads) reinterpret_cast<uint4*>(cache)[k] = make_uint4(v, v, v, v);
}

template <int LOG>
__device__ __forceinline__ void count_cached(uint32_t* cache, uint32_t* m, uint32_t idx, bool whole = false) {
    if (whole) {
        atomicAdd(cache + idx, 1u);
        return;
    }
    const uint32_t tag = (idx >> LOG) + 1u;
    uint32_t* const w = cache + (idx & ((1u << LOG) - 1u));
    uint32_t have = *reinterpret_cast<volatile uint32_t*>(w) >> COUNT_TAG_SHIFT;
    if (have == 0u && tag < 32u) {
        have = atomicCAS(w, 0u, tag << COUNT_TAG_SHIFT) >> COUNT_TAG_SHIFT;
        if (have == 0u) have = tag;
    }
    if (have == tag) {
        atomicAdd(w, 1u);
        return;
    }
    count_in_memory(m, idx);
}

// By `threads` threads (thread = 0 ... threads - 1), beside others that count if need be: what has been counted goes to memory.
template <int LOG>
__device__ __forceinline__ void count_flush(uint32_t* cache, uint32_t* m, uint32_t thread, uint32_t threads) {
    for (uint32_t k = thread; k < (1u << LOG); k += 4 * threads) {
        uint32_t have[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) have[u] = k + u * threads < (1u << LOG) ? *reinterpret_cast<volatile uint32_t*>(cache + k + u * threads) : 0u;
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            if (!(have[u] & COUNT_MASK)) continue;
            const uint32_t at = k + u * threads, w = atomicAnd(cache + at, ~COUNT_MASK);
            if (w & COUNT_MASK) atomicAdd(m + ((((w >> COUNT_TAG_SHIFT) - 1u) << LOG) | at), w & COUNT_MASK);
        }
    }
}

// A row of the normalisation table (m7, expfield, nz) in a word, where it fits one: in shared memory a random row is then one access of a few
// cycles, where the table in memory takes three of a line a lane each.
__device__ __forceinline__ bool pack_norm(const uint32_t* __restrict__ norm3, uint32_t ni, uint32_t& w) {
    const uint32_t m7 = __ldg(norm3 + 3 * (size_t)ni), ef = __ldg(norm3 + 3 * (size_t)ni + 1), nz = __ldg(norm3 + 3 * (size_t)ni + 2);
    w = m7 | ef << 8 | nz << 24;
    return m7 < 256u && ef < 65536u && nz < 256u;
}
}  // namespace zk
