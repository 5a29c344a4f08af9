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

template <int LOG>
__device__ __forceinline__ void count_cached(uint32_t* cache, uint32_t* m, uint32_t idx) {
    const uint32_t tag = (idx >> LOG) + 1u;
    uint32_t* const w = cache + (idx & ((1u << LOG) - 1u));
    if (tag < 32u) {
        uint32_t have = *reinterpret_cast<volatile uint32_t*>(w);
        if (have == 0u) {
            have = atomicCAS(w, 0u, tag << COUNT_TAG_SHIFT);
            if (have == 0u) have = tag << COUNT_TAG_SHIFT;
        }
        if (have >> COUNT_TAG_SHIFT == tag) {
            atomicAdd(w, 1u);
            return;
        }
    }
    count_in_memory(m, idx);
}

// By `threads` threads (thread = 0 ... threads - 1), beside others that count if need be: what has been counted goes to memory.
template <int LOG>
__device__ __forceinline__ void count_flush(uint32_t* cache, uint32_t* m, uint32_t thread, uint32_t threads) {
    for (uint32_t k = thread; k < (1u << LOG); k += threads) {
        if (!(*reinterpret_cast<volatile uint32_t*>(cache + k) & COUNT_MASK)) continue;
        const uint32_t w = atomicAnd(cache + k, ~COUNT_MASK);
        if (w & COUNT_MASK) atomicAdd(m + ((((w >> COUNT_TAG_SHIFT) - 1u) << LOG) | k), w & COUNT_MASK);
    }
}

}  // namespace zk
