// Towers: up to ten levels of a layer's halvings per launch (gen_layers, nitroo/crates/stwo/src/prover/lookups/gkr_prover.rs:847-852).
// A level's entries come from adjacent pairs, so a CTA that takes 2^10 consecutive entries builds its share of every level above
// them; the levels stay in shared memory for the next one and every one is written. One launch per level read each level back from
// memory and cost a launch for the many short ones (a 2^24 tower: 24 launches, 290 us; now three, 218 us).
#pragma once
#include "common.cuh"

namespace zk {

constexpr int TOWER_LEVELS = 10, TOWER_THREADS = 256;

template <int KIND>
__device__ __forceinline__ void tower_pair(qm31 n0, qm31 n1, qm31 d0, qm31 d1, qm31& n, qm31& d) {
    d = qm31_mul(d0, d1);
    if (KIND == ZKB_GKR_LOGUP_SINGLES) n = qm31_add(d0, d1);
    else if (KIND == ZKB_GKR_LOGUP_MULTIPLICITIES) n = qm31_dot2_m31(d1, n0.c[0], d0, n1.c[0]);
    else if (KIND == ZKB_GKR_LOGUP_GENERIC) n = qm31_dot2(d1, n0, d0, n1);
    else n = qm31_zero();
}
__device__ __forceinline__ qm31 tower_ld(const void* p, size_t i) {
    const uint4 v = static_cast<const uint4*>(p)[i];
    return {{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ void tower_st(void* p, size_t i, qm31 v) { static_cast<uint4*>(p)[i] = make_uint4(v.c[0], v.c[1], v.c[2], v.c[3]); }

// CTA `block` of the flat grid over a layer of KIND: takes 2^cta_log of its entries through `levels` <= cta_log levels. outs(l, num, den)
// gives level l's arrays; tops (or null: the launch does not end the tower) gets, from the CTA that makes the last entry, the
// output's denominator and numerator and the two denominators and numerators below it. sd, sn: 512 entries each.
template <int KIND, class Outs>
__device__ __forceinline__ void tower_cta(const uint32_t* num, const uint32_t* den, uint32_t block, int cta_log, int levels, uint4* sd, uint4* sn, Outs outs, uint32_t* tops) {
    constexpr bool HAS_NUM_OUT = KIND != ZKB_GKR_GRAND_PRODUCT;
    constexpr int KIND2 = HAS_NUM_OUT ? ZKB_GKR_LOGUP_GENERIC : ZKB_GKR_GRAND_PRODUCT;
    const uint32_t half = 1u << (cta_log - 1);
    const size_t first = (size_t)block * half;
    uint32_t *num_out, *den_out;
    outs(0, num_out, den_out);
    auto top = [&](qm31 n0, qm31 n1, qm31 d0, qm31 d1, qm31 n, qm31 d) {
        const qm31 v[6] = {d, n, d0, d1, n0, n1};
#pragma unroll
        for (int k = 0; k < 6; k++) tower_st(tops, k, v[k]);
    };
    for (uint32_t i = threadIdx.x; i < half; i += TOWER_THREADS) {
        const size_t o = first + i;
        qm31 n0 = qm31_zero(), n1 = qm31_zero(), n, d;
        if (KIND == ZKB_GKR_LOGUP_GENERIC) { n0 = tower_ld(num, 2 * o); n1 = tower_ld(num, 2 * o + 1); }
        if (KIND == ZKB_GKR_LOGUP_MULTIPLICITIES) { n0.c[0] = num[2 * o]; n1.c[0] = num[2 * o + 1]; }
        const qm31 d0 = tower_ld(den, 2 * o), d1 = tower_ld(den, 2 * o + 1);
        tower_pair<KIND>(n0, n1, d0, d1, n, d);
        tower_st(den_out, o, d);
        tower_st(sd, i, d);
        if (HAS_NUM_OUT) { tower_st(num_out, o, n); tower_st(sn, i, n); }
        if (tops && levels == 1) top(n0, n1, d0, d1, n, d);
    }
    for (int l = 1; l < levels; l++) {
        const uint32_t m = half >> l;
        __syncthreads();
        qm31 n0 = qm31_zero(), n1 = qm31_zero(), d0, d1, n, d;
        const uint32_t i = threadIdx.x;  // at most 256 from the second level on
        if (i < m) {
            if (HAS_NUM_OUT) { n0 = tower_ld(sn, 2 * i); n1 = tower_ld(sn, 2 * i + 1); }
            d0 = tower_ld(sd, 2 * i);
            d1 = tower_ld(sd, 2 * i + 1);
            tower_pair<KIND2>(n0, n1, d0, d1, n, d);
        }
        __syncthreads();
        if (i < m) {
            const size_t o = (size_t)block * m + i;
            outs(l, num_out, den_out);
            tower_st(den_out, o, d);
            tower_st(sd, i, d);
            if (HAS_NUM_OUT) { tower_st(num_out, o, n); tower_st(sn, i, n); }
            if (tops && l + 1 == levels) top(n0, n1, d0, d1, n, d);
        }
    }
}

}  // namespace zk
