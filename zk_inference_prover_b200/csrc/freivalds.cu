// The Freivalds attention-witness component on the device: the committed / preprocessed columns
// (scatter of int8 activations and weights into M31 columns in committed order, with the 8-bit
// range multiplicities), and the Horner accumulators v, u_m, acc_m with their claims.
//
// Rows are laid out by a grid over input channels (prover/src/layout.rs:141-183): coset-order
// row j >= lead belongs to group (= input channel) groups-1-(j-lead)/chunks and chunk
// chunks-1-(j-lead)%chunks; a column stores row j at committed index coset_perm(j)
// (prover/src/common.rs:76-80; the permutation is an involution). Semantics follow
// prover/src/gadgets/freivalds/trace.rs:43-162 (columns) and claims.rs:37-109 (accumulators):
//   v[j]   = [chunk+1 < chunks] v[j-1] s^pq + sum_p s^p (act[p][j] - 128)
//   u_m[j] = [chunk+1 < chunks] u_m[j-1] rv^pk + sum_p rv^p w_m[p][j]
//   acc_m[j] = acc_m[j-1] + [chunk == 0] u_m[j] v[j]
// The Horner restarts at every group, so each group is scanned independently and acc_m is a prefix
// sum over the groups' totals. Kernels: per-row inner products (coalesced column reads, results in
// coset order), per-group scan, prefix over groups, split into coordinate columns.
#include <algorithm>
#include <vector>

#include "common.cuh"

namespace zk {

struct FGrid { uint32_t log_rows, groups, chunks, lead; };

__device__ __forceinline__ uint32_t coset_perm(uint32_t i, uint32_t log_n) {
    uint32_t n = 1u << log_n;
    uint32_t c = (i & 1u) ? (2u * n - i - 1u) >> 1 : i >> 1;
    return __brev(c) >> (32 - log_n);
}
__device__ __forceinline__ uint32_t m31_of_i32(int v) { return v < 0 ? (uint32_t)(v + (int)P) : (uint32_t)v; }

// Which rows a thread of the passes over all rows takes: i and rows - 1 - i. Their places in coset order are neighbours (an even row's
// place is twice the reversal of i / 2, the mirrored odd one's the one after it), so what is read or written there, 16 bytes a
// row, is a whole 32-byte sector at once; with one row a thread the halves of a sector came far apart in time and the memory
// behind L2 saw them twice. The warps of a CTA take rows an eighth of the half apart, whose places are neighbours again.
// block: of rows / 512 (at least one); false: no such row.
__device__ __forceinline__ bool row_pair(uint32_t block, uint32_t rows, uint32_t& i) {
    const uint32_t half = rows >> 1;
    i = half >= 256u ? (threadIdx.x >> 5) * (half >> 3) + block * 32u + (threadIdx.x & 31u) : threadIdx.x;
    return i < half;
}
static unsigned row_pair_blocks(size_t rows) { return rows >= 512 ? (unsigned)(rows / 512) : 1u; }

// ---- F1: columns ------------------------------------------------------------------------------
// Consecutive threads' rows lie far apart in coset order (the permutation is a bit reversal), so every weight load touches 32 sectors a
// warp: with one load a byte those, not the columns' stores, were the pass (16 of them a row and matrix). A row's weights of one
// matrix are consecutive: they are loaded 16 at a time where their addresses allow it, else four. A CTA takes several pieces of rows, so
// that its range histogram reaches memory once. 2^20 rows, 2 x 16 weights and an activation: 100 us before.
constexpr int SCATTER_THREADS = 256;
__global__ void __launch_bounds__(SCATTER_THREADS, 5) freivalds_scatter_kernel(const int8_t* __restrict__ qx, const int8_t* const* __restrict__ qw,
                                                                const uint32_t* __restrict__ n_out, FGrid g, uint32_t pq, uint32_t pk,
                                                                uint32_t n_in, uint32_t tokens, uint32_t n_mats,
                                                                uint32_t* const* __restrict__ base_cols,
                                                                uint32_t* const* __restrict__ pre_cols, uint32_t* __restrict__ m_r8,
                                                                uint32_t table_len, unsigned long long* __restrict__ off_table) {
    extern __shared__ uint32_t hist[];  // table_len counters
    for (uint32_t t = threadIdx.x; t < table_len; t += blockDim.x) hist[t] = 0;
    __syncthreads();
    const uint32_t rows = 1u << g.log_rows;
    for (uint32_t block = blockIdx.x; block < (rows >= 512u ? rows >> 9 : 1u); block += gridDim.x) {
      uint32_t i0;
      if (!row_pair(block, rows, i0)) continue;
      for (uint32_t side = 0; side < 2; side++) {
        const uint32_t i = side ? rows - 1u - i0 : i0;
        const uint32_t j = coset_perm(i, g.log_rows);
        const bool some = j >= g.lead;
        uint32_t k = 0, chunk = 0;
        if (some) {
            uint32_t idx = j - g.lead;
            k = g.groups - 1 - idx / g.chunks;
            chunk = g.chunks - 1 - idx % g.chunks;
        }
        uint32_t off = 0;
        for (uint32_t p = 0; p < pq; p++) {
            int v = 128;
            uint32_t t = chunk * pq + p;
            if (some && t < tokens) v = (int)qx[(size_t)t * n_in + k] + 128;
            base_cols[p][i] = (uint32_t)v;
            if ((uint32_t)v < table_len) atomicAdd(&hist[v], 1u); else off++;
        }
        if (off) atomicAdd(off_table, (unsigned long long)off);
        for (uint32_t m = 0; m < n_mats; m++) {
            const uint32_t no = n_out[m];
            const int8_t* __restrict__ w = qw[m] + (size_t)k * no;
            uint32_t* const* __restrict__ cols = pre_cols + m * pk;
            const uint32_t c0 = chunk * pk, fit = (uint32_t)reinterpret_cast<uintptr_t>(qw[m]) | no | pk;  // aligned and whole: every load of the row is
            if ((fit & 15u) == 0) {
                for (uint32_t p = 0; p < pk; p += 16) {
                    const uint4 x = some && c0 + p < no ? __ldg(reinterpret_cast<const uint4*>(w + c0 + p)) : make_uint4(0, 0, 0, 0);
                    const uint32_t q[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (uint32_t u = 0; u < 16; u++) cols[p + u][i] = m31_of_i32((int)(int8_t)(q[u >> 2] >> (8 * (u & 3))));
                }
            } else {
                // four at a time from aligned words; a word that is not wholly the matrix's comes in bytes
                const uintptr_t lo = reinterpret_cast<uintptr_t>(qw[m]), hi = lo + (uintptr_t)g.groups * no;
                auto word = [&](uintptr_t x) -> uint32_t {
                    if (x >= lo && x + 4 <= hi) return __ldg(reinterpret_cast<const uint32_t*>(x));
                    uint32_t v = 0;
                    for (uint32_t u = 0; u < 4; u++)
                        if (x + u >= lo && x + u < hi) v |= (uint32_t)__ldg(reinterpret_cast<const uint8_t*>(x + u)) << (8 * u);
                    return v;
                };
                const uintptr_t at = reinterpret_cast<uintptr_t>(w + c0);
                const bool any = some && c0 < no;
                uintptr_t x = at & ~(uintptr_t)3;
                uint32_t cur = any ? word(x) : 0u;
                for (uint32_t p = 0; p < pk; p += 4, x += 4) {
                    const uint32_t next = any ? word(x + 4) : 0u, v = __funnelshift_r(cur, next, 8u * (uint32_t)(at & 3u));
                    cur = next;
#pragma unroll
                    for (uint32_t u = 0; u < 4; u++)
                        if (p + u < pk) cols[p + u][i] = (some && c0 + p + u < no) ? m31_of_i32((int)(int8_t)(v >> (8 * u))) : 0u;
                }
            }
        }
        uint32_t* const* sel = pre_cols + n_mats * pk;
        sel[0][i] = (some && chunk + 1 < g.chunks) ? 1u : 0u;
        sel[1][i] = (some && chunk == 0) ? 1u : 0u;
        sel[2][i] = j > 0 ? 1u : 0u;
        sel[3][i] = j + 1 == rows ? 1u : 0u;
      }
    }
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < table_len; t += blockDim.x)
        if (hist[t]) atomicAdd(&m_r8[t], hist[t]);
}

// ---- F2: inner products per row -----------------------------------------------------------------
// lanes[l][j] (QM31, coset order): l = 0 is v_in, l = 1 + m is u_in of matrix m. Eight loads are on their way at a time (a load
// a row, behind that of its column address, one after the other: 107 us at 2^20 rows of 33 columns).
// sum of pow[p] (cols[p][row] - bias) for two rows
struct RowSums { uint4 a, b; };
__device__ __forceinline__ RowSums inner_pair(const uint32_t* const* __restrict__ cols, const uint4* __restrict__ pow, uint32_t n, uint32_t bias, uint32_t i, uint32_t i2) {
    uint64_t a[4] = {0, 0, 0, 0}, b[4] = {0, 0, 0, 0};
    for (uint32_t p0 = 0; p0 < n; p0 += 4) {
        uint32_t x[4], y[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            const bool there = p0 + u < n;
            const uint32_t* const col = there ? cols[p0 + u] : nullptr;
            x[u] = there ? __ldcs(col + i) : bias;
            y[u] = there ? __ldcs(col + i2) : bias;
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {  // four products below 2^62 on top of a folded accumulator fit 64 bits
            const uint4 c = p0 + u < n ? __ldg(pow + p0 + u) : make_uint4(0, 0, 0, 0);
            const uint32_t v = m31_sub(x[u], bias), w = m31_sub(y[u], bias);
            a[0] += (uint64_t)c.x * v; a[1] += (uint64_t)c.y * v; a[2] += (uint64_t)c.z * v; a[3] += (uint64_t)c.w * v;
            b[0] += (uint64_t)c.x * w; b[1] += (uint64_t)c.y * w; b[2] += (uint64_t)c.z * w; b[3] += (uint64_t)c.w * w;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) { a[q] = m31_fold64(a[q]); b[q] = m31_fold64(b[q]); }
    }
    return {make_uint4(m31_reduce64(a[0]), m31_reduce64(a[1]), m31_reduce64(a[2]), m31_reduce64(a[3])),
            make_uint4(m31_reduce64(b[0]), m31_reduce64(b[1]), m31_reduce64(b[2]), m31_reduce64(b[3]))};
}
__global__ void __launch_bounds__(256, 4) freivalds_inner_kernel(const uint32_t* const* __restrict__ base_cols,
                                                                 const uint32_t* const* __restrict__ pre_cols,
                                                                 const uint4* __restrict__ s_pow, const uint4* __restrict__ rv_pow, FGrid g,
                                                                 uint32_t pq, uint32_t pk, uint32_t n_mats, uint4* __restrict__ lanes) {
    const uint32_t rows = 1u << g.log_rows;
    uint32_t i;
    if (!row_pair(blockIdx.x, rows, i)) return;
    const uint32_t i2 = rows - 1u - i, j = coset_perm(i, g.log_rows), j2 = coset_perm(i2, g.log_rows);
    for (uint32_t l = 0; l <= n_mats; l++) {
        const RowSums r = l ? inner_pair(pre_cols + (size_t)(l - 1) * pk, rv_pow, pk, 0u, i, i2) : inner_pair(base_cols, s_pow, pq, 128u, i, i2);
        uint4* const out = lanes + (size_t)l * rows;
        out[j] = j >= g.lead ? r.a : make_uint4(0, 0, 0, 0);
        out[j2] = j2 >= g.lead ? r.b : make_uint4(0, 0, 0, 0);
    }
}

// The same, four rows a thread: two neighbours and the two that mirror them, whose places in coset order are two whole sectors. What a column costs
// beside its products (its address, the power, the checks) is paid for four rows, column addresses and powers come from shared memory,
// and the activations' bias is taken off the finished sums. 2^20 rows of 33 columns: 24 instructions a row and column, 52 us; now 15 and
// 42.
constexpr uint32_t INNER_TILE = 64;
__global__ void __launch_bounds__(256, 4) freivalds_inner_quad_kernel(const uint32_t* const* __restrict__ base_cols, const uint32_t* const* __restrict__ pre_cols,
                                                                      const uint4* __restrict__ s_pow, const uint4* __restrict__ rv_pow, FGrid g, uint32_t pq,
                                                                      uint32_t pk, uint32_t n_mats, qm31 bias, uint4* __restrict__ lanes) {
    __shared__ const uint32_t* s_col[INNER_TILE];
    __shared__ uint4 s_c[INNER_TILE];
    const uint32_t rows = 1u << g.log_rows, n_threads = rows >> 2;  // at least 256
    const uint32_t i = 2u * ((threadIdx.x >> 5) * (n_threads >> 3) + blockIdx.x * 32u + (threadIdx.x & 31u)), i2 = rows - 2u - i;
    for (uint32_t l = 0; l <= n_mats; l++) {
        const uint32_t* const* __restrict__ cols = l ? pre_cols + (size_t)(l - 1) * pk : base_cols;
        const uint4* __restrict__ pow = l ? rv_pow : s_pow;
        const uint32_t n = l ? pk : pq;
        uint64_t a[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int q = 0; q < 4; q++) a[r][q] = 0;
        auto add = [&](const uint4& c, const uint2& x, const uint2& y) {
            const uint32_t e[4] = {x.x, x.y, y.x, y.y};
#pragma unroll
            for (int r = 0; r < 4; r++) {
                a[r][0] += (uint64_t)c.x * e[r]; a[r][1] += (uint64_t)c.y * e[r]; a[r][2] += (uint64_t)c.z * e[r]; a[r][3] += (uint64_t)c.w * e[r];
            }
        };
        // four products below 2^62 on top of a folded sum fit 64 bits
        auto fold = [&] {
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int q = 0; q < 4; q++) a[r][q] = m31_fold64(a[r][q]);
        };
        for (uint32_t tile = 0; tile < n; tile += INNER_TILE) {
            const uint32_t here = n - tile < INNER_TILE ? n - tile : INNER_TILE;
            __syncthreads();
            if (threadIdx.x < here) {
                s_col[threadIdx.x] = cols[tile + threadIdx.x];
                s_c[threadIdx.x] = pow[tile + threadIdx.x];
            }
            __syncthreads();
            uint32_t p = 0;
            for (; p + 4 <= here; p += 4) {
                uint2 x[4], y[4];
#pragma unroll
                for (uint32_t u = 0; u < 4; u++) {
                    x[u] = __ldcs(reinterpret_cast<const uint2*>(s_col[p + u] + i));
                    y[u] = __ldcs(reinterpret_cast<const uint2*>(s_col[p + u] + i2));
                }
#pragma unroll
                for (uint32_t u = 0; u < 4; u++) add(s_c[p + u], x[u], y[u]);
                fold();
            }
            for (; p < here; p++) add(s_c[p], __ldcs(reinterpret_cast<const uint2*>(s_col[p] + i)), __ldcs(reinterpret_cast<const uint2*>(s_col[p] + i2)));
            fold();
        }
        uint4* const out = lanes + (size_t)l * rows;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const uint32_t j = coset_perm(r < 2 ? i + r : i2 + r - 2, g.log_rows);
            uint32_t w[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t v = m31_reduce64(a[r][q]);
                w[q] = l ? v : m31_sub(v, bias.c[q]);
            }
            out[j] = j >= g.lead ? make_uint4(w[0], w[1], w[2], w[3]) : make_uint4(0, 0, 0, 0);
        }
    }
}

// ---- F3: per-group Horner, prefix over groups, split ------------------------------------------------
__device__ __forceinline__ qm31 q_of(uint4 v) { return {{v.x, v.y, v.z, v.w}}; }
__device__ __forceinline__ uint4 u_of(qm31 v) { return make_uint4(v.c[0], v.c[1], v.c[2], v.c[3]); }

// x_r = x_{r-1} step + in_r over the group's `chunks` rows, one WARP a group, 256 rows at a time: lane l takes rows 8l .. 8l+7, runs
// them from a zero carry into registers, the lanes' values are combined by a shuffle scan (a lane of eight rows multiplies what
// comes before it by step^8, so the multipliers of the scan are constants), and each lane then adds its carry times the running power
// of the step. All lanes (v, then the u_m) of the group go through the same warp one after the other, so that the product
// u_m v of the group's last row (what the prefix over groups sums) is at hand and is written to prod[m][slot]. Bound by its products,
// 22 a lane and eight rows (with the multipliers scanned too: 26). One thread per (group, lane) walking 256 rows in sequence
// kept 6% of the warp slots busy and took as long as the pass over all the input columns.
struct ScanSteps {
    qm31 pw[2][9];    // pw[kind][k] = step^k for k = 0..8; kind 0 is lane 0 (v, step s^pq), kind 1 the lanes u_m (step rv^pk)
    qm31 wide[2][6];  // step^(8 2^k)
};
// `left` rows of a group (at most 256 are taken), by a warp; end: the value before them, on return that after the last of them.
// get(r): row r's input; put(r, x): its value. IN_PLACE: get reads what put wrote cheaply, so the sums from a zero carry are kept there
// instead of in 32 registers.
template <bool IN_PLACE, class Get, class Put>
__device__ __forceinline__ void scan_rows(uint32_t left, bool first, const qm31* pw, const qm31* wide, qm31& end, Get get, Put put) {
    const uint32_t lane = threadIdx.x & 31u, r0 = lane * 8u, n_here = r0 >= left ? 0u : (left - r0 < 8u ? left - r0 : 8u);
    const qm31 step = pw[1];
    qm31 y[IN_PLACE ? 1 : 8];
    qm31 acc = qm31_zero();
#pragma unroll
    for (uint32_t k = 0; k < 8; k++)
        if (k < n_here) {
            acc = qm31_mul_add(acc, step, q_of(get(r0 + k)));
            if (IN_PLACE) put(r0 + k, u_of(acc));
            else y[IN_PLACE ? 0 : k] = acc;
        }
    // The value after a lane's rows, exact for lanes whose rows before them are all there: only the last lane with rows may
    // have fewer than eight, and nothing is taken from it or from the ones after.
    qm31 B = lane == 0 && !first ? qm31_mul_add(end, pw[n_here], acc) : acc;
#pragma unroll
    for (int k = 0; k < 5; k++) {
        qm31 b1;
#pragma unroll
        for (int c = 0; c < 4; c++) b1.c[c] = __shfl_up_sync(0xffffffffu, B.c[c], 1 << k);
        if ((int)lane >= (1 << k)) B = qm31_mul_add(b1, wide[k], B);
    }
    qm31 carry;  // into this lane: the value at the end of the previous one
#pragma unroll
    for (int c = 0; c < 4; c++) carry.c[c] = __shfl_up_sync(0xffffffffu, B.c[c], 1);
    if (lane == 0) carry = end;
#pragma unroll
    for (uint32_t k = 0; k < 8; k++)
        if (k < n_here) {
            acc = qm31_mul_add(carry, pw[k + 1], IN_PLACE ? q_of(get(r0 + k)) : y[IN_PLACE ? 0 : k]);
            put(r0 + k, u_of(acc));
        }
    const int from = (int)((left < 256u ? left : 256u) - 1u) >> 3;  // the lane of the last row
#pragma unroll
    for (int c = 0; c < 4; c++) end.c[c] = __shfl_sync(0xffffffffu, acc.c[c], from);
}
__global__ void __launch_bounds__(256) freivalds_group_scan_kernel(uint4* __restrict__ lanes, FGrid g, uint32_t n_mats, const __grid_constant__ ScanSteps st,
                                                                   uint4* __restrict__ prod) {
    const uint32_t slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (slot >= g.groups) return;
    qm31 v_last = qm31_zero();
    for (uint32_t l = 0; l <= n_mats; l++) {
        uint4* p = lanes + ((size_t)l << g.log_rows) + g.lead + (size_t)slot * g.chunks;
        qm31 end = qm31_zero();  // the value after the last row so far
        for (uint32_t base = 0; base < g.chunks; base += 256, p += 256)
            scan_rows<false>(g.chunks - base, base == 0, st.pw[l ? 1 : 0], st.wide[l ? 1 : 0], end, [&](uint32_t r) { return p[r]; }, [&](uint32_t r, uint4 x) { p[r] = x; });
        if (l == 0) v_last = end;
        else if (lane == 0) prod[(size_t)(l - 1) * g.groups + slot] = u_of(qm31_mul(end, v_last));
    }
}

// Scan and split in one, where a group is 256 rows, what a warp scans at a time: then it is an aligned block of coset order, and in committed
// order the blocks whose numbers, bits reversed, are neighbours lie next to each other: with c = (row in the block, bits reversed) 2^L + c_low, c_low
// the block's number reversed, an even row is at 2 c and an odd one at 2 n - 1 - 2 c. A CTA takes the blocks c0 ... c0 + 7 (A) and their complements
// (B), a warp each; for an even row r and either of the two segments below, sixteen consecutive words hold eight blocks' values at row r and eight
// of the others' at row 255 - r, so a lane's values cross shared memory once and go out in whole 64-byte pieces. A block of lead rows is zeros and is
// not scanned. 2^20 rows, v and two u: scan and split one after the other 45 + 35 us, this and the accumulators' columns 47 + 10.
constexpr uint32_t BLOCK_LOG = 8, BLOCK_ROWS = 1u << BLOCK_LOG;
constexpr int SCAN_OUT_THREADS = 512, SCAN_OUT_GROUPS = SCAN_OUT_THREADS / 32;
constexpr uint32_t SCAN_OUT_PITCH = BLOCK_ROWS + 32;  // of a group in shared memory: a gap every eight rows, which the lanes write at a time
constexpr size_t SCAN_OUT_SMEM = (size_t)SCAN_OUT_GROUPS * SCAN_OUT_PITCH * 16;
__global__ void __launch_bounds__(SCAN_OUT_THREADS, 2) freivalds_scan_out_kernel(const uint4* __restrict__ lanes, FGrid g, uint32_t n_mats,
                                                                                 const __grid_constant__ ScanSteps st, uint4* __restrict__ prod,
                                                                                 uint32_t* const* __restrict__ out) {
    extern __shared__ uint4 tile[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, L = g.log_rows - BLOCK_LOG, mask = (1u << L) - 1u, c0 = blockIdx.x * 8u;
    const uint32_t c_low = warp < 8 ? c0 + warp : mask - (c0 + warp - 8u), block = __brev(c_low) >> (32 - L);
    const uint32_t lead_blocks = g.lead >> BLOCK_LOG;
    const bool live = block >= lead_blocks;
    uint4* const mine = tile + warp * SCAN_OUT_PITCH;
    auto at = [](uint32_t r) { return r + (r >> 3); };
    if (!live)
        for (uint32_t k = lane; k < SCAN_OUT_PITCH; k += 32u) mine[k] = make_uint4(0, 0, 0, 0);
    qm31 v_last = qm31_zero();
    for (uint32_t l = 0; l <= n_mats; l++) {
        if (live) {
            qm31 end = qm31_zero();
            const uint4* const rows_in = lanes + ((size_t)l << g.log_rows) + ((size_t)block << BLOCK_LOG);
            uint4 in[8];
#pragma unroll
            for (uint32_t k = 0; k < 8; k++) in[k] = rows_in[32u * k + lane];
#pragma unroll
            for (uint32_t k = 0; k < 8; k++) mine[at(32u * k + lane)] = in[k];
            __syncwarp();
            scan_rows<true>(BLOCK_ROWS, true, st.pw[l ? 1 : 0], st.wide[l ? 1 : 0], end, [&](uint32_t r) { return mine[at(r)]; }, [&](uint32_t r, uint4 x) { mine[at(r)] = x; });
            if (l == 0) v_last = end;
            else if (lane == 0) prod[(size_t)(l - 1) * g.groups + block - lead_blocks] = u_of(qm31_mul(end, v_last));
        }
        __syncthreads();
        uint32_t* const* const o = out + (l ? 8 * l - 4 : 0);
        uint32_t *const o0 = o[0], *const o1 = o[1], *const o2 = o[2], *const o3 = o[3];
        for (uint32_t k = threadIdx.x; k < 16u * BLOCK_ROWS; k += SCAN_OUT_THREADS) {
            const uint32_t w = k & 15u, t = w >> 1, odd = w & 1u, seg = (k >> 4) & 1u, h = k >> 5, r = __brev(h) >> (32 - BLOCK_LOG);
            const uint32_t from = seg == odd ? (seg ? 7u - t : t) : 8u + (seg ? 7u - t : t);  // A in even words of the first segment, odd ones of the second
            const uint32_t row = odd ? BLOCK_ROWS - 1u - r : r;
            const uint4 x = tile[from * SCAN_OUT_PITCH + at(row)];
            const size_t i = 2u * ((h << L) + (seg ? mask - (c0 + 7u) : c0)) + w;
            o0[i] = x.x; o1[i] = x.y; o2[i] = x.z; o3[i] = x.w;
        }
        __syncthreads();
    }
}
// The accumulators' columns for the same grids: the prefix up to the row's block, in its last row (odd, the odd words' first) with it. Where a row
// lies in committed order modulo 2^(L + 1) says which block it is of: a thread has the prefixes of four neighbouring places and writes them to
// every row of its share.
constexpr uint32_t ACC_RUN = 16;
static_assert(BLOCK_ROWS / 2 % ACC_RUN == 0, "whole runs");
__global__ void __launch_bounds__(128) freivalds_acc_columns_kernel(const uint4* __restrict__ prefix, FGrid g, uint32_t n_mats, uint32_t* const* __restrict__ out) {
    const uint32_t L = g.log_rows - BLOCK_LOG, low = 4u * (blockIdx.x * blockDim.x + threadIdx.x), lead_blocks = g.lead >> BLOCK_LOG;
    if (low >> (L + 1)) return;
    const uint32_t h0 = blockIdx.y * ACC_RUN;
    uint32_t upto[4];  // slots in the sum of a place's rows
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) {
        const uint32_t block = coset_perm(low + u, g.log_rows) >> BLOCK_LOG;
        upto[u] = block < lead_blocks ? 0u : block - lead_blocks;
    }
    for (uint32_t m = 0; m < n_mats; m++) {
        const uint4* const pre = prefix + (size_t)m * g.groups;
        auto sum = [&](uint32_t n) { return n ? pre[n - 1u] : make_uint4(0, 0, 0, 0); };
        uint32_t* const* const o = out + 8 + 8 * m;
        uint32_t *const o0 = o[0] + low, *const o1 = o[1] + low, *const o2 = o[2] + low, *const o3 = o[3] + low;
        auto write = [&](size_t h, uint4 a, uint4 b, uint4 c, uint4 d) {
            const size_t i = h << (L + 1);
            *reinterpret_cast<uint4*>(o0 + i) = make_uint4(a.x, b.x, c.x, d.x);
            *reinterpret_cast<uint4*>(o1 + i) = make_uint4(a.y, b.y, c.y, d.y);
            *reinterpret_cast<uint4*>(o2 + i) = make_uint4(a.z, b.z, c.z, d.z);
            *reinterpret_cast<uint4*>(o3 + i) = make_uint4(a.w, b.w, c.w, d.w);
        };
        const uint4 a = sum(upto[0]), b = sum(upto[1]), c = sum(upto[2]), d = sum(upto[3]);
        for (uint32_t h = h0; h < h0 + ACC_RUN; h++)
            if (h) write(h, a, b, c, d);
        if (h0 == 0) {
            const uint32_t b1 = coset_perm(low + 1u, g.log_rows) >> BLOCK_LOG, d1 = coset_perm(low + 3u, g.log_rows) >> BLOCK_LOG;
            write(0, a, sum(b1 < lead_blocks ? 0u : upto[1] + 1u), c, sum(d1 < lead_blocks ? 0u : upto[3] + 1u));
        }
    }
}

// In place: prefix[m][slot] = sum over slots <= slot of what is there; a CTA a matrix, a thread a run of slots. The whole sum is the
// matrix's claim: it goes to page-locked memory as well. (One CTA for all matrices, 1,024 slots at a time: 16 us for 2 x 4,096.)
__global__ void __launch_bounds__(1024) freivalds_prefix_kernel(uint4* __restrict__ prefix, uint32_t groups, uint4* __restrict__ claims) {
    __shared__ qm31 warp_tot[32];
    const uint32_t run = (groups + 1023u) / 1024u, first = threadIdx.x * run, last = first + run < groups ? first + run : groups;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint4* __restrict__ p = prefix + (size_t)blockIdx.x * groups;
    auto shift = [&](qm31 v, int off) {
        qm31 o;
#pragma unroll
        for (int k = 0; k < 4; k++) o.c[k] = __shfl_up_sync(0xffffffffu, v.c[k], off);
        return o;
    };
    qm31 sum = qm31_zero();
#pragma unroll 4
    for (uint32_t s = first; s < last; s++) sum = qm31_add(sum, q_of(p[s]));
    auto scan = [&](qm31 x) {  // inclusive, over the warp
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const qm31 o = shift(x, off);
            if (lane >= off) x = qm31_add(x, o);
        }
        return x;
    };
    const qm31 mine = scan(sum);
    if (lane == 31) warp_tot[warp] = mine;
    __syncthreads();
    if (warp == 0) warp_tot[lane] = scan(warp_tot[lane]);
    __syncthreads();
    qm31 acc = shift(mine, 1);
    if (lane == 0) acc = qm31_zero();
    if (warp) acc = qm31_add(acc, warp_tot[warp - 1]);
    for (uint32_t s = first; s < last; s++) {
        acc = qm31_add(acc, q_of(p[s]));
        p[s] = u_of(acc);
    }
    if (first < last && last == groups) claims[blockIdx.x] = u_of(acc);
}

// out: (1 + 2 n_mats) secure columns of 4 coordinate columns each, committed order.
__global__ void __launch_bounds__(256) freivalds_split_kernel(const uint4* __restrict__ lanes, const uint4* __restrict__ prefix, FGrid g,
                                                              uint32_t n_mats, uint32_t* const* __restrict__ out) {
    const uint32_t rows = 1u << g.log_rows;
    uint32_t i0;
    if (!row_pair(blockIdx.x, rows, i0)) return;
#pragma unroll
    for (uint32_t side = 0; side < 2; side++) {
    const uint32_t i = side ? rows - 1u - i0 : i0;
    const uint32_t j = coset_perm(i, g.log_rows);
    const bool some = j >= g.lead;
    uint32_t slot = 0;
    bool last = false;
    if (some) {
        slot = (j - g.lead) / g.chunks;
        last = (j - g.lead) % g.chunks == g.chunks - 1;
    }
    uint4 v = lanes[j];
    out[0][i] = v.x; out[1][i] = v.y; out[2][i] = v.z; out[3][i] = v.w;
    for (uint32_t m = 0; m < n_mats; m++) {
        uint4 u = lanes[(size_t)(1 + m) * rows + j];
        uint32_t* const* ou = out + 4 + 8 * m;
        ou[0][i] = u.x; ou[1][i] = u.y; ou[2][i] = u.z; ou[3][i] = u.w;
        uint4 a = make_uint4(0, 0, 0, 0);
        if (some) {
            if (last) a = prefix[(size_t)m * g.groups + slot];
            else if (slot > 0) a = prefix[(size_t)m * g.groups + slot - 1];
        }
        uint32_t* const* oa = out + 8 + 8 * m;
        oa[0][i] = a.x; oa[1][i] = a.y; oa[2][i] = a.z; oa[3][i] = a.w;
    }
    }
}

static bool grid_ok(const zkb_grid* g) {
    if (!g || g->log_rows < 1 || g->log_rows > 28 || g->groups == 0 || g->chunks == 0) return false;
    uint64_t rows = 1ull << g->log_rows;
    return (uint64_t)g->groups * g->chunks + g->lead == rows;
}

}  // namespace zk

using namespace zk;

extern "C" {

int zkb_freivalds_scatter(zkb_ctx* ctx, const int8_t* qx, const int8_t* const* qw, const uint32_t* h_n_out, const zkb_grid* grid,
                          uint32_t pq, uint32_t pk, uint32_t n_in, uint32_t tokens, uint32_t n_mats, uint32_t* const* base_cols,
                          uint32_t* const* pre_cols, uint32_t* m_r8, uint32_t table_len, unsigned long long* off_table) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, grid_ok(grid) && grid->groups == n_in);
    ZKB_CHECK_ARG(ctx, qx && qw && h_n_out && base_cols && pre_cols && m_r8 && off_table && pq >= 1 && pk >= 1 && n_mats >= 1);
    ZKB_CHECK_ARG(ctx, table_len >= 1 && table_len <= 8192 && n_mats <= 64);
    ZKB_CHECK_ARG(ctx, (uint64_t)grid->chunks * pq >= tokens);
    for (uint32_t m = 0; m < n_mats; m++) ZKB_CHECK_ARG(ctx, qw[m] != nullptr && (uint64_t)grid->chunks * pk >= h_n_out[m]);
    DeviceGuard g(ctx);
    void **d_base, **d_pre, **d_qw;
    int rc = stage_reserve(ctx, (size_t)pq + (size_t)n_mats * pk + 4 + n_mats + blob_slots(n_mats * 4));
    if (rc) return rc;
    rc = stage_ptrs(ctx, (const void* const*)base_cols, (int)pq, &d_base);
    if (rc) return rc;
    rc = stage_ptrs(ctx, (const void* const*)pre_cols, (int)(n_mats * pk + 4), &d_pre);
    if (rc) return rc;
    rc = stage_ptrs(ctx, (const void* const*)qw, (int)n_mats, &d_qw);
    if (rc) return rc;
    void* d_nout = nullptr;
    rc = stage_blob(ctx, h_n_out, n_mats * 4, &d_nout);
    if (rc) return rc;
    FGrid fg{grid->log_rows, grid->groups, grid->chunks, grid->lead};
    uint32_t rows = 1u << grid->log_rows;
    ProfScope prof(ctx, "freivalds_scatter_kernel");
    const uint32_t grid_ctas = std::min(row_pair_blocks(rows), 148u * 8u);
    freivalds_scatter_kernel<<<grid_ctas, SCATTER_THREADS, table_len * 4, ctx->stream>>>(
        qx, (const int8_t* const*)d_qw, (const uint32_t*)d_nout, fg, pq, pk, n_in, tokens, n_mats, (uint32_t* const*)d_base, (uint32_t* const*)d_pre,
        m_r8, table_len, off_table);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

int zkb_freivalds_acc(zkb_ctx* ctx, const uint32_t* const* base_cols, const uint32_t* const* pre_cols, const zkb_grid* grid, uint32_t pq,
                      uint32_t pk, uint32_t n_mats, const uint32_t h_s[4], const uint32_t h_rv[4], uint32_t* const* out_cols,
                      uint32_t* h_claims) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, grid_ok(grid) && base_cols && pre_cols && h_s && h_rv && out_cols && h_claims);
    ZKB_CHECK_ARG(ctx, pq >= 1 && pk >= 1 && n_mats >= 1 && n_mats <= 64 && (size_t)(pq + pk) * 4 <= ctx->scratch_words);
    DeviceGuard g(ctx);
    const size_t rows = (size_t)1 << grid->log_rows;
    const uint32_t n_lanes = 1 + n_mats;
    // powers of the two challenges, and their steps s^pq, rv^pk (prover/src/relations.rs:85-93)
    std::vector<qm31> pows;
    qm31 s{{h_s[0], h_s[1], h_s[2], h_s[3]}}, rv{{h_rv[0], h_rv[1], h_rv[2], h_rv[3]}};
    qm31 cur = qm31_one();
    for (uint32_t p = 0; p < pq; p++) { pows.push_back(cur); cur = qm31_mul(cur, s); }
    qm31 s_step = cur;
    cur = qm31_one();
    for (uint32_t p = 0; p < pk; p++) { pows.push_back(cur); cur = qm31_mul(cur, rv); }
    qm31 rv_step = cur;
    // the powers go up through the pinned staging ring: no synchronisation with the work before
    void **d_base, **d_pre, **d_out;
    void* d_pw;
    int rc = stage_reserve(ctx, blob_slots(pows.size() * sizeof(qm31)) + (size_t)pq + (size_t)n_mats * pk + (1 + 2 * (size_t)n_mats) * 4);
    if (rc) return rc;
    rc = stage_blob(ctx, pows.data(), pows.size() * sizeof(qm31), &d_pw);
    if (rc) return rc;
    uint4* d_pows = reinterpret_cast<uint4*>(d_pw);
    rc = stage_ptrs(ctx, (const void* const*)base_cols, (int)pq, &d_base);
    if (rc) return rc;
    rc = stage_ptrs(ctx, (const void* const*)pre_cols, (int)(n_mats * pk), &d_pre);
    if (rc) return rc;
    rc = stage_ptrs(ctx, (const void* const*)out_cols, (int)((1 + 2 * n_mats) * 4), &d_out);
    if (rc) return rc;
    auto aligned = [](const uint32_t* const* p, size_t n) {
        for (size_t k = 0; k < n; k++) if ((uintptr_t)p[k] & 15) return false;
        return true;
    };
    // Scan and split in one takes groups of 256 rows, what a warp scans at a time, from 2^19 rows on (two CTAs on nearly every SM): a group is an aligned
    // block of coset order, since lead, the rest of a power of two, is a multiple of 256 too. Two passes -> one, this call alone, two matrices of 16
    // columns: 2^19 rows without lead 100.7 -> 93.1 us, with half of it lead 93.4 -> 89.6; 2^20 157.6 -> 138.8 and 133.5 -> 124.2; 2^22 506 -> 413 and
    // 427 -> 350. One matrix of two columns gains 4 to 20 %, three of 16 5 to 21 %. Below, a CTA's barriers have no other CTA's work to hide behind
    // and two passes, a warp a group without any, are ahead: 2^18 77.0 -> 83.6, 2^16 68.3 -> 79.0. So they are with shorter groups, where a CTA has as many
    // barriers for fewer rows (with the block's size a parameter, 2^20 rows of 128, 64 and 32 to a group: 172 -> 178, 224 -> 241, 336 -> 394).
    const bool blocks = grid->chunks == BLOCK_ROWS && grid->log_rows >= 19 && aligned(out_cols, (1 + 2 * (size_t)n_mats) * 4);
    if (blocks) ZKB_CUDA(ctx, cudaFuncSetAttribute(freivalds_scan_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SCAN_OUT_SMEM));
    // work buffers from the stream-ordered pool: lanes in coset order, prefix over groups
    uint4 *lanes = nullptr, *prefix = nullptr;
    ZKB_CUDA(ctx, cudaMallocAsync((void**)&lanes, (size_t)n_lanes * rows * 16, ctx->stream));
    cudaError_t e = cudaMallocAsync((void**)&prefix, (size_t)n_mats * grid->groups * 16, ctx->stream);
    if (e != cudaSuccess) { cudaFreeAsync(lanes, ctx->stream); return set_error(ctx, ZKB_ENOMEM, "zkb_freivalds_acc: %s", cudaGetErrorString(e)); }
    FGrid fg{grid->log_rows, grid->groups, grid->chunks, grid->lead};
    auto even = [](const uint32_t* const* p, size_t n) {
        for (size_t k = 0; k < n; k++) if ((uintptr_t)p[k] & 7) return false;
        return true;
    };
    // Four rows a thread from 2^19 rows (512 CTAs) and eight columns a matrix on. The whole call, two rows a thread -> four: 2^20 rows, one matrix of 40
    // columns 132 -> 120 us, three of 8 175 -> 172; 2^19, three of 8 116 -> 112. Two rows a thread keep what is smaller, where the chip isn't full
    // (2^18, three of 8: 82.7 -> 82.9; 2^16: 69.1 -> 71.3) or a thread has few columns to share its work (2^20, three of 1: 190 -> 196).
    if (rows >= (1u << 19) && pk >= 8 && even(base_cols, pq) && even(pre_cols, (size_t)n_mats * pk)) {
        qm31 bias = qm31_zero();
        for (uint32_t p = 0; p < pq; p++) bias = qm31_add(bias, qm31_mul_m31(pows[p], 128u));
        ProfScope prof(ctx, "freivalds_inner_quad_kernel");
        freivalds_inner_quad_kernel<<<(unsigned)(rows / 1024), 256, 0, ctx->stream>>>(
            (const uint32_t* const*)d_base, (const uint32_t* const*)d_pre, d_pows, d_pows + pq, fg, pq, pk, n_mats, bias, lanes);
    } else {
        ProfScope prof(ctx, "freivalds_inner_kernel");
        freivalds_inner_kernel<<<row_pair_blocks(rows), 256, 0, ctx->stream>>>(
            (const uint32_t* const*)d_base, (const uint32_t* const*)d_pre, d_pows, d_pows + pq, fg, pq, pk, n_mats, lanes);
    }
    ScanSteps scan_steps;
    for (int kind = 0; kind < 2; kind++) {
        scan_steps.pw[kind][0] = qm31_one();
        for (int k = 1; k <= 8; k++) scan_steps.pw[kind][k] = qm31_mul(scan_steps.pw[kind][k - 1], kind ? rv_step : s_step);
        scan_steps.wide[kind][0] = scan_steps.pw[kind][8];
        for (int k = 1; k < 6; k++) scan_steps.wide[kind][k] = qm31_mul(scan_steps.wide[kind][k - 1], scan_steps.wide[kind][k - 1]);
    }
    if (blocks) {
        ProfScope prof(ctx, "freivalds_scan_out_kernel");
        freivalds_scan_out_kernel<<<1u << (grid->log_rows - BLOCK_LOG - 4), SCAN_OUT_THREADS, SCAN_OUT_SMEM, ctx->stream>>>(lanes, fg, n_mats, scan_steps, prefix, (uint32_t* const*)d_out);
    } else {
        ProfScope prof(ctx, "freivalds_group_scan_kernel");
        freivalds_group_scan_kernel<<<(unsigned)(((size_t)grid->groups * 32 + 255) / 256), 256, 0, ctx->stream>>>(lanes, fg, n_mats, scan_steps, prefix);
    }
    {
        ProfScope prof(ctx, "freivalds_prefix_kernel");
        freivalds_prefix_kernel<<<n_mats, 1024, 0, ctx->stream>>>(prefix, grid->groups, reinterpret_cast<uint4*>(ctx->h_small));
    }
    if (blocks) {
        ProfScope prof(ctx, "freivalds_acc_columns_kernel");
        const dim3 ctas(((2u << (grid->log_rows - BLOCK_LOG)) / 4 + 127) / 128, BLOCK_ROWS / 2 / ACC_RUN);
        freivalds_acc_columns_kernel<<<ctas, 128, 0, ctx->stream>>>(prefix, fg, n_mats, (uint32_t* const*)d_out);
    } else {
        ProfScope prof(ctx, "freivalds_split_kernel");
        freivalds_split_kernel<<<row_pair_blocks(rows), 256, 0, ctx->stream>>>(lanes, prefix, fg, n_mats, (uint32_t* const*)d_out);
    }
    e = cudaGetLastError();
    cudaFreeAsync(lanes, ctx->stream);
    cudaFreeAsync(prefix, ctx->stream);
    if (e != cudaSuccess) return set_error(ctx, ZKB_ECUDA, "zkb_freivalds_acc: %s", cudaGetErrorString(e));
    ZKB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    memcpy(h_claims, ctx->h_small, (size_t)n_mats * 16);
    return ZKB_OK;
}

}  // extern "C"
