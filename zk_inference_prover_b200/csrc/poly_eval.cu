// PolyOps::eval_at_point / batch_eval_at_point: the value of each column's polynomial (FFT-basis
// coefficients) at one QM31 circle point.
//
// The reference folds the coefficient array as a binary tree
// (nitroo/crates/stwo/src/prover/backend/cpu/circle.rs:82-100, core/poly/utils.rs:11-23):
// level k joins blocks of 2^k values as lhs + rhs * m_k with m_0 = y, m_1 = x, m_{k+1} = pi(m_k).
// Field arithmetic is exact and distributive, so the tree equals sum_i c_i * prod_{k: bit k of i} m_k.
// The lowest 11 levels are evaluated as that weighted sum: a CTA takes 2048 coefficients, every
// thread multiplies its 8 coefficients (M31) by weights it keeps in registers (QM31), accumulating
// unreduced in 64 bits, and the CTA adds the 256 partial sums. What remains per column is a short
// array of partials, folded level by level in shared memory with the remaining factors.
#include <vector>

#include "common.cuh"
#include "quot_lines.hpp"

namespace zk {

constexpr int EVAL_CHUNK_LOG = 11;
constexpr int EVAL_MAX_LEVELS = 32;

struct EvalFactors { qm31 m[EVAL_MAX_LEVELS]; };

// weights[i] = prod over set bits k of i of m_k, i < 2^EVAL_CHUNK_LOG, and behind them the same of the run_bits factors that follow.
__global__ void eval_weights_kernel(EvalFactors f, int run_bits, uint32_t* __restrict__ weights) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, n = 1u << EVAL_CHUNK_LOG;
    if (i >= n + (1u << run_bits)) return;
    const int first = i < n ? 0 : EVAL_CHUNK_LOG, bits = i < n ? EVAL_CHUNK_LOG : run_bits;
    qm31 w = qm31_one();
    for (int k = 0; k < bits; k++)
        if (((i < n ? i : i - n) >> k) & 1u) w = qm31_mul(w, f.m[first + k]);
    reinterpret_cast<uint4*>(weights)[i] = make_uint4(w.c[0], w.c[1], w.c[2], w.c[3]);
}

// out[col][chunk] = sum_{e < 2048} cols[col][2048 chunk + e] * weights[e]
// Thread t owns elements 4t..4t+3 and 1024+4t..1024+4t+3 of every chunk (two 16-byte loads) and keeps
// their eight weights in registers. DOT_CHUNKS chunks are in flight per iteration; their per-warp sums
// use the hardware warp reduction on 16-bit halves (32 x 2^16 fits a word) and meet in shared memory
// once per iteration.
constexpr int DOT_CHUNKS = 4;
__global__ void __launch_bounds__(256) eval_dot_kernel(const uint32_t* const* __restrict__ cols, int ncols, int log_n,
                                                       const uint32_t* __restrict__ weights, uint32_t* __restrict__ out) {
    __shared__ uint32_t red[DOT_CHUNKS][4][2][8];  // [chunk][component][lo/hi][warp]
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    uint4 w[8];
#pragma unroll
    for (int u = 0; u < 8; u++) w[u] = reinterpret_cast<const uint4*>(weights)[(u >> 2) * 1024 + 4 * t + (u & 3)];
    const size_t chunks = (size_t)1 << (log_n - EVAL_CHUNK_LOG);
    const size_t groups = (chunks + DOT_CHUNKS - 1) / DOT_CHUNKS;
    // persistent CTAs over (column, group of chunks): the weights are read once per CTA
    for (size_t item = blockIdx.x; item < groups * (size_t)ncols; item += gridDim.x) {
        const size_t col = item / groups, chunk0 = (item % groups) * DOT_CHUNKS;
        const uint32_t* __restrict__ c = cols[col];
        uint4 v[DOT_CHUNKS][2];
#pragma unroll
        for (int g = 0; g < DOT_CHUNKS; g++) {
            if (chunk0 + g < chunks) {
                const uint4* p = reinterpret_cast<const uint4*>(c + ((chunk0 + g) << EVAL_CHUNK_LOG));
                v[g][0] = __ldcs(p + t);
                v[g][1] = __ldcs(p + 256 + t);
            } else {
                v[g][0] = v[g][1] = make_uint4(0, 0, 0, 0);
            }
        }
#pragma unroll
        for (int g = 0; g < DOT_CHUNKS; g++) {
            const uint32_t e[8] = {v[g][0].x, v[g][0].y, v[g][0].z, v[g][0].w, v[g][1].x, v[g][1].y, v[g][1].z, v[g][1].w};
            uint64_t a0 = 0, a1 = 0, a2 = 0, a3 = 0;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                a0 += (uint64_t)e[u] * w[u].x; a1 += (uint64_t)e[u] * w[u].y;
                a2 += (uint64_t)e[u] * w[u].z; a3 += (uint64_t)e[u] * w[u].w;
                if (u == 3) { a0 = m31_fold64(a0); a1 = m31_fold64(a1); a2 = m31_fold64(a2); a3 = m31_fold64(a3); }
            }
            const uint32_t r[4] = {m31_reduce64(a0), m31_reduce64(a1), m31_reduce64(a2), m31_reduce64(a3)};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                uint32_t lo = __reduce_add_sync(0xffffffffu, r[k] & 0xffffu);
                uint32_t hi = __reduce_add_sync(0xffffffffu, r[k] >> 16);
                if (lane == 0) { red[g][k][0][warp] = lo; red[g][k][1][warp] = hi; }
            }
        }
        __syncthreads();
        if (t < 4 * DOT_CHUNKS) {
            const int g = t >> 2, k = t & 3;
            if (chunk0 + g < chunks) {
                uint64_t lo = 0, hi = 0;
#pragma unroll
                for (int wv = 0; wv < 8; wv++) { lo += red[g][k][0][wv]; hi += red[g][k][1][wv]; }
                out[4 * ((size_t)col * chunks + chunk0 + g) + k] = m31_reduce64(lo + (hi << 16));
            }
        }
        __syncthreads();
    }
}

// The same for runs of 2^run_log chunks: out[col][run] = sum_e weights[e] sum_g weights[2048 + g] cols[col][2048 (2^run_log run + g) + e].
// eval_dot_kernel is bound by what a chunk costs beside its products, the reduction of four words over the CTA; here a thread keeps the inner sums of
// its eight elements through a run (64-bit sums folded every four chunks) and the weights and the reduction come once a run. 256 columns of
// 2^20: 396 us with a reduction a chunk, 210 with one in 64.
constexpr int RUN_MIN_LOG = 4, RUN_MAX_LOG = 6, RUN_CTAS = 2, RUN_MIN_RUNS = 80;
__global__ void __launch_bounds__(256, RUN_CTAS) eval_runs_kernel(const uint32_t* const* __restrict__ cols, int ncols, int log_n, int run_log,
                                                                  const uint32_t* __restrict__ weights, uint32_t* __restrict__ out) {
    __shared__ uint4 of_chunk[1 << RUN_MAX_LOG];
    __shared__ uint32_t red[2][4][2][8];  // [run mod 2][component][lo/hi][warp]
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const uint4* const w = reinterpret_cast<const uint4*>(weights);
    if (t < (1 << run_log)) of_chunk[t] = w[(1 << EVAL_CHUNK_LOG) + t];
    __syncthreads();
    const int runs_log = log_n - EVAL_CHUNK_LOG - run_log;
    const size_t items = (size_t)ncols << runs_log;
    const int chunks = 1 << run_log;
    int side = 0;
    for (size_t item = blockIdx.x; item < items; item += gridDim.x, side ^= 1) {
        const uint4* __restrict__ c = reinterpret_cast<const uint4*>(cols[item >> runs_log] + ((item & (((size_t)1 << runs_log) - 1)) << (EVAL_CHUNK_LOG + run_log))) + t;
        uint64_t a[8][4];
#pragma unroll
        for (int u = 0; u < 8; u++)
#pragma unroll
            for (int q = 0; q < 4; q++) a[u][q] = 0;
        uint4 next[4];  // two chunks
#pragma unroll
        for (int g = 0; g < 4; g++) next[g] = __ldcs(c + 256 * g);
        for (int g0 = 0; g0 < chunks; g0 += 4) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint4 v[4];
#pragma unroll
                for (int g = 0; g < 4; g++) v[g] = next[g];
                c += 1024;
                if (g0 + 2 * h + 2 < chunks) {
#pragma unroll
                    for (int g = 0; g < 4; g++) next[g] = __ldcs(c + 256 * g);
                }
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    const uint4 f = of_chunk[g0 + 2 * h + g], x = v[2 * g], y = v[2 * g + 1];
                    const uint32_t e[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        a[u][0] += (uint64_t)e[u] * f.x; a[u][1] += (uint64_t)e[u] * f.y;
                        a[u][2] += (uint64_t)e[u] * f.z; a[u][3] += (uint64_t)e[u] * f.w;
                    }
                }
            }
            // four 62-bit products on top of a folded (< 2^34) sum fit in 64 bits
#pragma unroll
            for (int u = 0; u < 8; u++)
#pragma unroll
                for (int q = 0; q < 4; q++) a[u][q] = m31_fold64(a[u][q]);
        }
        qm31 r = qm31_zero();
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const uint4 x = w[(u >> 2) * 1024 + 4 * t + (u & 3)];
            r = qm31_add(r, qm31_mul(qm31{{m31_reduce64(a[u][0]), m31_reduce64(a[u][1]), m31_reduce64(a[u][2]), m31_reduce64(a[u][3])}}, qm31{{x.x, x.y, x.z, x.w}}));
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t lo = __reduce_add_sync(0xffffffffu, r.c[k] & 0xffffu), hi = __reduce_add_sync(0xffffffffu, r.c[k] >> 16);
            if (lane == 0) { red[side][k][0][warp] = lo; red[side][k][1][warp] = hi; }
        }
        __syncthreads();  // (what the run before the last left in the same place was read before the last run's barrier)
        if (t < 4) {
            uint64_t lo = 0, hi = 0;
#pragma unroll
            for (int wv = 0; wv < 8; wv++) { lo += red[side][t][0][wv]; hi += red[side][t][1][wv]; }
            out[4 * item + t] = m31_reduce64(lo + (hi << 16));
        }
    }
}

// Columns of at most 2^10 coefficients: out[col] = sum_i cols[col][i] w_i with the weights in shared memory (made there, level by level:
// ten products deep), a warp a column, CTAs over the columns until none are left. Bound by HBM where there are many columns; folding
// a column as a tree of QM31 values in shared memory instead took ten times the arithmetic (65,000 columns of 2^8 to 2^10: 500 us).
constexpr int EVAL_SHORT_LOG = 10;
__global__ void __launch_bounds__(256) eval_short_kernel(const uint32_t* const* __restrict__ cols, int ncols, int log_n, const __grid_constant__ EvalFactors f,
                                                         uint32_t* __restrict__ out) {
    __shared__ uint4 w[1 << EVAL_SHORT_LOG];
    const uint32_t n = 1u << log_n, lane = threadIdx.x & 31u;
    if (threadIdx.x == 0) w[0] = make_uint4(1u, 0u, 0u, 0u);
    for (int k = 0; k < log_n; k++) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < (1u << k); i += 256u) {
            const uint4 x = w[i];
            const qm31 r = qm31_mul(qm31{{x.x, x.y, x.z, x.w}}, f.m[k]);
            w[(1u << k) + i] = make_uint4(r.c[0], r.c[1], r.c[2], r.c[3]);
        }
    }
    __syncthreads();
    for (int col = (int)(blockIdx.x * 8u + (threadIdx.x >> 5)); col < ncols; col += (int)(gridDim.x * 8u)) {
        const uint32_t* __restrict__ c = cols[col];
        uint64_t a[4] = {0, 0, 0, 0};
#pragma unroll 2
        for (uint32_t e = lane; e < n; e += 128u) {
            uint32_t v[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) v[u] = e + 32u * u < n ? __ldcs(c + e + 32u * u) : 0u;
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                const uint4 x = w[e + 32u * u < n ? e + 32u * u : 0u];
                a[0] += (uint64_t)v[u] * x.x; a[1] += (uint64_t)v[u] * x.y;
                a[2] += (uint64_t)v[u] * x.z; a[3] += (uint64_t)v[u] * x.w;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) a[q] = m31_fold64(a[q]);
        }
        uint32_t r[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t x = m31_reduce64(a[q]);
            const uint32_t lo = __reduce_add_sync(0xffffffffu, x & 0xffffu), hi = __reduce_add_sync(0xffffffffu, x >> 16);
            r[q] = m31_reduce64(lo + ((uint64_t)hi << 16));
        }
        if (lane == 0) reinterpret_cast<uint4*>(out)[col] = make_uint4(r[0], r[1], r[2], r[3]);
    }
}

// in: either a table of M31 columns (IS_BASE) or a dense [ncols][2^log_in] array of QM31.
// out: dense [ncols][2^(log_in - chunk_log)] QM31.
template <bool IS_BASE>
__global__ void __launch_bounds__(256) eval_fold_kernel(const uint32_t* const* __restrict__ base_cols,
                                                        const uint32_t* __restrict__ ext_in, int log_in, int chunk_log,
                                                        int level0, EvalFactors f, uint32_t* __restrict__ out) {
    __shared__ uint32_t s[4][1 << EVAL_CHUNK_LOG];
    const uint32_t E = 1u << chunk_log;
    const size_t chunk = blockIdx.x;
    const int col = blockIdx.y;
    const size_t n_in = (size_t)1 << log_in;
    for (uint32_t e = threadIdx.x; e < E; e += blockDim.x) {
        size_t idx = chunk * E + e;
        if (IS_BASE) {
            s[0][e] = base_cols[col][idx];
            s[1][e] = 0; s[2][e] = 0; s[3][e] = 0;
        } else {
            uint4 v = reinterpret_cast<const uint4*>(ext_in)[(size_t)col * n_in + idx];
            s[0][e] = v.x; s[1][e] = v.y; s[2][e] = v.z; s[3][e] = v.w;
        }
    }
    __syncthreads();
    for (int k = 0; k < chunk_log; k++) {
        const qm31 m = f.m[level0 + k];
        for (uint32_t t = threadIdx.x; t < (E >> (k + 1)); t += blockDim.x) {
            uint32_t i0 = t << (k + 1), i1 = i0 + (1u << k);
            qm31 a{{s[0][i0], s[1][i0], s[2][i0], s[3][i0]}}, b{{s[0][i1], s[1][i1], s[2][i1], s[3][i1]}};
            qm31 r = qm31_add(a, qm31_mul(b, m));
            s[0][i0] = r.c[0]; s[1][i0] = r.c[1]; s[2][i0] = r.c[2]; s[3][i0] = r.c[3];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        size_t n_out = n_in >> chunk_log;
        reinterpret_cast<uint4*>(out)[(size_t)col * n_out + chunk] = make_uint4(s[0][0], s[1][0], s[2][0], s[3][0]);
    }
}

int eval_at_point_device(zkb_ctx* ctx, const uint32_t* const* coeffs, int ncols, int log_n, const uint32_t h_point[8], uint32_t* d_out) {
    DeviceGuard g(ctx);
    // factors m_0 = y, m_1 = x, m_{k+1} = 2 m_k^2 - 1
    EvalFactors f;
    memset(&f, 0, sizeof(f));
    qm31 x{{h_point[0], h_point[1], h_point[2], h_point[3]}}, y{{h_point[4], h_point[5], h_point[6], h_point[7]}};
    f.m[0] = y;
    for (int k = 1; k < log_n; k++) {
        f.m[k] = x;
        x = qm31_double_x(x);
    }
    constexpr int MAX_COLS = 32768;  // columns a launch
    if (log_n <= EVAL_SHORT_LOG) {
        for (int c0 = 0; c0 < ncols; c0 += MAX_COLS) {
            const int nc = ncols - c0 < MAX_COLS ? ncols - c0 : MAX_COLS;
            void** d_cols;
            if (int rc = stage_ptrs(ctx, (const void* const*)(coeffs + c0), nc, &d_cols)) return rc;
            ProfScope prof(ctx, "eval_short_kernel");
            eval_short_kernel<<<(unsigned)((nc + 7) / 8 < 6 * 148 ? (nc + 7) / 8 : 6 * 148), 256, 0, ctx->stream>>>((const uint32_t* const*)d_cols, nc, log_n, f,
                                                                                                                  d_out + 4 * (size_t)c0);
            ZKB_LAUNCH_CHECK(ctx);
        }
        return ZKB_OK;
    }
    static_assert(EVAL_SHORT_LOG + 1 == EVAL_CHUNK_LOG, "what is left has a whole chunk");
    // Scratch: [weights: 2048 and 64 QM31] [ping] [pong]; columns go in batches whose partials fit.
    bool use_dot = true;
    for (int c = 0; c < ncols; c++) use_dot = use_dot && ((uintptr_t)coeffs[c] & 15) == 0;  // 16-byte loads
    // Runs of sixteen chunks, longer as long as there are two for every SM (shorter ones cost more in products with the weights than they save). Fewer
    // than 80 of sixteen are a handful of CTAs that walk them one chunk after the other; four chunks a CTA are faster there, unless a column is one run
    // and the launch that folds the runs falls away. The whole call, four chunks -> runs, columns not in L2: 8 of 2^18 (64 runs) 39.1 -> 40.3 us, 10
    // (80) 42.0 -> 41.0, 16 (128) 45.6 -> 41.4; 33 of 2^16 (66) 42.6 -> 43.4, 40 (80) 44.5 -> 44.1, 64 (128) 51 -> 47; 1 of 2^20 (32) 38.2 -> 39.0, 4 (128)
    // 49.5 -> 40.2. One run a column, 4 of 2^15: 38.6 -> 36.7, 64: 45.7 -> 43.3.
    int run_log = log_n - EVAL_CHUNK_LOG < RUN_MAX_LOG ? log_n - EVAL_CHUNK_LOG : RUN_MAX_LOG;
    while (run_log > RUN_MIN_LOG && ((size_t)ncols << (log_n - EVAL_CHUNK_LOG - run_log)) < RUN_CTAS * 148u) run_log--;
    if (!use_dot || run_log < RUN_MIN_LOG || (log_n > EVAL_CHUNK_LOG + RUN_MIN_LOG && ((size_t)ncols << (log_n - EVAL_CHUNK_LOG - RUN_MIN_LOG)) < RUN_MIN_RUNS)) run_log = 0;
    const int chunk_log = EVAL_CHUNK_LOG + run_log;
    size_t partials_per_col = (size_t)1 << (log_n - chunk_log);
    uint32_t* weights = ctx->scratch;
    const size_t weights_words = ((size_t)4 << EVAL_CHUNK_LOG) + ((size_t)4 << RUN_MAX_LOG);
    size_t half_words = (ctx->scratch_words - weights_words) / 2;
    size_t max_cols = half_words / (4 * partials_per_col);
    ZKB_CHECK_ARG(ctx, max_cols >= 1);
    if (max_cols > MAX_COLS) max_cols = MAX_COLS;
    if (use_dot) {
        eval_weights_kernel<<<(1 << EVAL_CHUNK_LOG) / 256 + 1, 256, 0, ctx->stream>>>(f, run_log, weights);
        ZKB_LAUNCH_CHECK(ctx);
    }
    for (int c0 = 0; c0 < ncols; c0 += (int)max_cols) {
        int nc = ncols - c0 < (int)max_cols ? ncols - c0 : (int)max_cols;
        void** d_cols;
        int rc = stage_ptrs(ctx, (const void* const*)(coeffs + c0), nc, &d_cols);
        if (rc) return rc;
        uint32_t* bufA = ctx->scratch + weights_words;
        uint32_t* bufB = bufA + half_words;
        uint32_t* const out = d_out + 4 * (size_t)c0;  // what the last kernel writes to
        int log_cur = log_n, level = 0;
        if (run_log) {
            const size_t items = partials_per_col * (size_t)nc;
            ProfScope prof(ctx, "eval_runs_kernel");
            eval_runs_kernel<<<(unsigned)(items < RUN_CTAS * 148u ? items : RUN_CTAS * 148u), 256, 0, ctx->stream>>>((const uint32_t* const*)d_cols, nc, log_n, run_log, weights,
                                                                                                               log_n == chunk_log ? out : bufA);
            ZKB_LAUNCH_CHECK(ctx);
        } else if (use_dot) {
            size_t items = (partials_per_col + DOT_CHUNKS - 1) / DOT_CHUNKS * (size_t)nc;
            unsigned grid = (unsigned)(items < 2 * 148 ? items : 2 * 148);
            ProfScope prof(ctx, "eval_dot_kernel");
            eval_dot_kernel<<<grid, 256, 0, ctx->stream>>>((const uint32_t* const*)d_cols, nc, log_n, weights, log_n == EVAL_CHUNK_LOG ? out : bufA);
            ZKB_LAUNCH_CHECK(ctx);
        } else {
            dim3 grid((unsigned)partials_per_col, nc);
            eval_fold_kernel<true><<<grid, 256, 0, ctx->stream>>>((const uint32_t* const*)d_cols, nullptr, log_cur, EVAL_CHUNK_LOG, level, f,
                                                                  log_n == EVAL_CHUNK_LOG ? out : bufA);
            ZKB_LAUNCH_CHECK(ctx);
        }
        log_cur -= chunk_log;
        level += chunk_log;
        while (log_cur > 0) {
            int ch = log_cur < EVAL_CHUNK_LOG ? log_cur : EVAL_CHUNK_LOG;
            unsigned threads = ch >= 9 ? 256 : 32;
            dim3 grid(1u << (log_cur - ch), nc);
            eval_fold_kernel<false><<<grid, threads, 0, ctx->stream>>>(nullptr, bufA, log_cur, ch, level, f, log_cur == ch ? out : bufB);
            ZKB_LAUNCH_CHECK(ctx);
            log_cur -= ch;
            level += ch;
            uint32_t* t = bufA; bufA = bufB; bufB = t;
        }
    }
    return ZKB_OK;
}

}  // namespace zk

using namespace zk;

extern "C" {

int zkb_eval_at_point_cols(zkb_ctx* ctx, const uint32_t* const* coeffs, int ncols, int log_n, const uint32_t* h_point,
                           uint32_t* h_out) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, ncols >= 0 && log_n >= 0 && log_n <= 30);
    if (ncols == 0) return ZKB_OK;
    ZKB_CHECK_ARG(ctx, coeffs && h_point && h_out);
    DeviceGuard g(ctx);
    uint32_t* d_out = nullptr;
    if (int rc = zkb_malloc(ctx, (size_t)ncols * 16, (void**)&d_out)) return rc;
    int rc = eval_at_point_device(ctx, coeffs, ncols, log_n, h_point, d_out);
    cudaError_t e = cudaSuccess;
    if (rc == ZKB_OK) e = cudaMemcpyAsync(h_out, d_out, (size_t)ncols * 16, cudaMemcpyDeviceToHost, ctx->stream);
    if (rc == ZKB_OK && e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    zkb_free(ctx, d_out);
    if (rc == ZKB_OK && e != cudaSuccess) rc = set_error(ctx, ZKB_ECUDA, "eval at point: %s", cudaGetErrorString(e));
    return rc;
}

}  // extern "C"
