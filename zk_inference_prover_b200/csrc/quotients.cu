// QuotientOps and AccumulationOps.
//
// accumulate_numerators, per row: sum_j (c_j * col_{idx_j}[row] - b_j) with QM31 coefficients and
// M31 column values (nitroo/crates/stwo/src/core/pcs/quotients.rs:217-229). The b_j do not depend
// on the row, so their sum is taken once on the host; the c_j * value products are accumulated
// unreduced in 64 bits (four 62-bit products fit) and folded every four columns.
//
// compute_quotients_and_combine, per row: sum over sample points z of
//   (acc_z[lift(row)] - A_z * p.y) * ((Re z.x - p.x) * Im z.y - (Re z.y - p.y) * Im z.x)^-1
// with p the row's domain point (prover/backend/cpu/quotients.rs:47-75). p comes from the twiddle
// tower; the CM31 inverses of one row are taken with one M31 inversion (Montgomery's trick on the
// norms), which is exact because inverses are unique.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "fri_tail.hpp"
#include "quot_lines.hpp"

namespace zk {

struct Secure4 { uint32_t* c[4]; };
struct Secure4C { const uint32_t* c[4]; };

// R consecutive rows per thread (one 8- or 16-byte load per column). The column addresses and the
// coefficients of a tile of columns are resolved once per CTA into shared memory, so the inner loop
// is one independent streaming load per column and 4 R multiply-adds: the kernel is bound by HBM.
constexpr int NUM_TILE = 128;

template <int R>
__global__ void __launch_bounds__(256) quot_numerators_kernel(const uint32_t* const* __restrict__ cols,
                                                              const uint32_t* __restrict__ col_idx,
                                                              const uint4* __restrict__ coeff_c, int k, qm31 b_sum, int b_first,
                                                              size_t n, Secure4 out, int chunk = 0,
                                                              uint32_t* __restrict__ partial = nullptr) {
    // With `partial`, CTA row blockIdx.y takes the columns [y * chunk, (y + 1) * chunk) and leaves its reduced sums in
    // partial[(y * 4 + coordinate) * n + row]; quot_partial_sum_kernel adds the rows up. Short, wide groups (thousands of
    // columns of a few hundred rows) would otherwise run on one or two CTAs. b_first: b_sum is taken off row 0 only.
    const int k_begin = partial ? (int)blockIdx.y * chunk : 0;
    const int k_end = partial ? (k_begin + chunk < k ? k_begin + chunk : k) : k;
    __shared__ const uint32_t* s_col[NUM_TILE];
    __shared__ uint4 s_c[NUM_TILE];
    const size_t row0 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * R;
    const bool live = row0 < n;
    uint64_t acc[R][4];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[r][q] = 0;
    auto load = [&](const uint32_t* col, uint32_t (&v)[R]) {
        if constexpr (R == 4) {
            uint4 x = __ldcs(reinterpret_cast<const uint4*>(col + row0));
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        } else {
            uint2 x = __ldcs(reinterpret_cast<const uint2*>(col + row0));
            v[0] = x.x; v[1] = x.y;
        }
    };
    auto mac = [&](const uint4& c, const uint32_t (&v)[R]) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            acc[r][0] += (uint64_t)c.x * v[r]; acc[r][1] += (uint64_t)c.y * v[r];
            acc[r][2] += (uint64_t)c.z * v[r]; acc[r][3] += (uint64_t)c.w * v[r];
        }
    };
    for (int tile0 = k_begin; tile0 < k_end; tile0 += NUM_TILE) {
        const int tk = k_end - tile0 < NUM_TILE ? k_end - tile0 : NUM_TILE;
        __syncthreads();
        for (int t = (int)threadIdx.x; t < tk; t += (int)blockDim.x) {
            s_col[t] = cols[col_idx[tile0 + t]];
            s_c[t] = coeff_c[tile0 + t];
        }
        __syncthreads();
        if (!live) continue;
        int j = 0;
        for (; j + 4 <= tk; j += 4) {
            uint32_t v[4][R];
#pragma unroll
            for (int u = 0; u < 4; u++) load(s_col[j + u], v[u]);
#pragma unroll
            for (int u = 0; u < 4; u++) mac(s_c[j + u], v[u]);
            // four 62-bit products on top of a folded (< 2^34) accumulator fit in 64 bits
#pragma unroll
            for (int r = 0; r < R; r++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[r][q] = m31_fold64(acc[r][q]);
        }
        for (; j < tk; j++) {  // at most 3 tail products
            uint32_t v[R];
            load(s_col[j], v);
            mac(s_c[j], v);
        }
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[r][q] = m31_fold64(acc[r][q]);
    }
    if (!live) return;
    uint32_t res[R][4];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
        for (int q = 0; q < 4; q++) res[r][q] = partial ? m31_reduce64(acc[r][q]) : m31_sub(m31_reduce64(acc[r][q]), b_first && row0 + r ? 0u : b_sum.c[q]);
    if (partial) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            uint32_t* dst = partial + ((size_t)blockIdx.y * 4 + q) * n + row0;
            if constexpr (R == 4) *reinterpret_cast<uint4*>(dst) = make_uint4(res[0][q], res[1][q], res[2][q], res[3][q]);
            else *reinterpret_cast<uint2*>(dst) = make_uint2(res[0][q], res[1][q]);
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if constexpr (R == 4) *reinterpret_cast<uint4*>(out.c[q] + row0) = make_uint4(res[0][q], res[1][q], res[2][q], res[3][q]);
        else *reinterpret_cast<uint2*>(out.c[q] + row0) = make_uint2(res[0][q], res[1][q]);
    }
}

// out[q][row] = sum over the S column chunks of partial[(s * 4 + q) * n + row], minus b_sum. PARTS warps share 32 of the 4 n words, a run of
// chunks each: short groups have hundreds of chunks (one thread a word walked them for 18 us), tall ones a few and many words.
template <int PARTS>
__global__ void __launch_bounds__(256) quot_partial_sum_kernel(const uint32_t* __restrict__ partial, int S, size_t n, qm31 b_sum, int b_first, Secure4 out) {
    __shared__ uint64_t sums[8][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t i = ((size_t)blockIdx.x * (8 / PARTS) + warp / PARTS) * 32 + lane;  // over 4 * n (coordinate-major)
    uint64_t acc = 0;
    if (i < 4 * n)
        for (int s = (int)(warp % PARTS); s < S; s += PARTS) acc += partial[(size_t)s * 4 * n + i];  // 31-bit terms: the 64-bit sum cannot overflow
    if (PARTS > 1) {
        sums[warp][lane] = acc;
        __syncthreads();
        if (warp % PARTS) return;
#pragma unroll
        for (int w = 1; w < PARTS; w++) acc += sums[warp + w][lane];
    }
    if (i >= 4 * n) return;
    const int q = (int)(i / n);
    const size_t row = i - (size_t)q * n;
    out.c[q][row] = m31_sub(m31_reduce64(acc), b_first && row ? 0u : b_sum.c[q]);
}

constexpr int MAX_ACCS = 8;
struct CombineArgs {
    const uint32_t* acc[MAX_ACCS][4];
    int log_ratio[MAX_ACCS];
    qm31 first_lin[MAX_ACCS];
    cm31 prx[MAX_ACCS], pry[MAX_ACCS], pix[MAX_ACCS], piy[MAX_ACCS];
    int n_acc;
    int first;  // 1: overwrite out, 0: add to out (more than MAX_ACCS accumulations)
};

// Rows [row_begin, row_begin + n_rows) of the lifting domain; the accumulations and `out` are indexed from row_begin
// (a row shard holds only its own rows; the whole domain is row_begin = 0, n_rows = 2^lifting_log).
//
// Bound by its products, 37 of a row's 60 those of an inversion: a thread takes ROWS neighbouring rows of up to ACCS accumulations and inverts the
// product of their norms once. One accumulation over 2^23 rows, a row a thread: 230 us, four: 115.
template <int ACCS, int ROWS>
__global__ void __launch_bounds__(256) quot_combine_kernel(const __grid_constant__ CombineArgs a, int lifting_log, Secure4 out,
                                                           const uint32_t* __restrict__ tw, size_t row_begin, size_t n_rows) {
    const size_t local = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * ROWS;
    if (local >= n_rows) return;
    const size_t row0 = row_begin + local;
    cm31 den[ACCS * ROWS];
    uint32_t norm[ACCS * ROWS], pref[ACCS * ROWS], py[ROWS];
    uint32_t run = 1u, px = 0u;
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
        if (ROWS == 1 || !(r & 1)) half_coset_point(tw, lifting_log, (uint32_t)((row0 + r) >> 1), px, py[r]);
        if (ROWS > 1 && (r & 1)) py[r] = m31_neg(py[r - 1]);  // odd rows hold the conjugate point; several rows start on an even one
        if (ROWS == 1 && (row0 & 1)) py[r] = m31_neg(py[r]);
#pragma unroll
        for (int z = 0; z < ACCS; z++) {
            if (z < a.n_acc) {
                const int k = r * ACCS + z;
                cm31 dx = {m31_sub(a.prx[z].a, px), a.prx[z].b};
                cm31 dy = {m31_sub(a.pry[z].a, py[r]), a.pry[z].b};
                den[k] = cm31_sub(cm31_mul(dx, a.piy[z]), cm31_mul(dy, a.pix[z]));
                norm[k] = m31_reduce64((uint64_t)den[k].a * den[k].a + (uint64_t)den[k].b * den[k].b);
                pref[k] = run;
                run = m31_mul(run, norm[k]);
            }
        }
    }
    uint32_t inv = m31_inv(run);
#pragma unroll
    for (int r = ROWS - 1; r >= 0; r--) {
        const size_t row = row0 + r;
        qm31 q = qm31_zero();
#pragma unroll
        for (int z = ACCS - 1; z >= 0; z--) {
            if (z < a.n_acc) {
                const int k = r * ACCS + z;
                uint32_t ninv = m31_mul(inv, pref[k]);
                inv = m31_mul(inv, norm[k]);
                cm31 dinv = {m31_mul(den[k].a, ninv), m31_mul(m31_neg(den[k].b), ninv)};
                const size_t li = ((row >> (a.log_ratio[z] + 1)) << 1) + (row & 1) - (((row_begin >> (a.log_ratio[z] + 1)) << 1));
                qm31 num{{a.acc[z][0][li], a.acc[z][1][li], a.acc[z][2][li], a.acc[z][3][li]}};
                num = qm31_sub(num, qm31_mul_m31(a.first_lin[z], py[r]));
                q = qm31_add(q, qm31_mul_cm31(num, dinv));
            }
        }
        if (!a.first) {
            qm31 o{{out.c[0][local + r], out.c[1][local + r], out.c[2][local + r], out.c[3][local + r]}};
            q = qm31_add(q, o);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) out.c[k][local + r] = q.c[k];
    }
}

// Slow path for lifting domains of log size 1 and 2, whose points are not in the tower.
__global__ void quot_combine_small_kernel(CombineArgs a, int lifting_log, Secure4 out, uint32_t x0, uint32_t y0,
                                          uint32_t x1, uint32_t y1) {
    int row = threadIdx.x;
    if (row >= (1 << lifting_log)) return;
    uint32_t px = (row >> 1) ? x1 : x0, py = (row >> 1) ? y1 : y0;
    if (row & 1) py = m31_neg(py);
    qm31 q = qm31_zero();
    for (int z = 0; z < a.n_acc; z++) {
        cm31 dx = {m31_sub(a.prx[z].a, px), a.prx[z].b};
        cm31 dy = {m31_sub(a.pry[z].a, py), a.pry[z].b};
        cm31 dinv = cm31_inv(cm31_sub(cm31_mul(dx, a.piy[z]), cm31_mul(dy, a.pix[z])));
        int li = ((row >> (a.log_ratio[z] + 1)) << 1) + (row & 1);
        qm31 num{{a.acc[z][0][li], a.acc[z][1][li], a.acc[z][2][li], a.acc[z][3][li]}};
        num = qm31_sub(num, qm31_mul_m31(a.first_lin[z], py));
        q = qm31_add(q, qm31_mul_cm31(num, dinv));
    }
    if (!a.first) {
        qm31 o{{out.c[0][row], out.c[1][row], out.c[2][row], out.c[3][row]}};
        q = qm31_add(q, o);
    }
    for (int k = 0; k < 4; k++) out.c[k][row] = q.c[k];
}

__global__ void __launch_bounds__(256) accumulate_kernel(Secure4 col, Secure4C other, size_t n) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
#pragma unroll
    for (int k = 0; k < 4; k++) col.c[k][i] = m31_add(col.c[k][i], other.c[k][i]);
}

__global__ void __launch_bounds__(256) lift_accumulate_kernel(Secure4 dst, int log_dst, Secure4C src, int log_ratio) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ((size_t)1 << log_dst)) return;
    size_t li = ((i >> (log_ratio + 1)) << 1) + (i & 1);
#pragma unroll
    for (int k = 0; k < 4; k++) dst.c[k][i] = m31_add(dst.c[k][i], src.c[k][li]);
}

}  // namespace zk

using namespace zk;

static cpoint host_point_q(uint32_t index) {
    cpoint g{2u, 1268011823u}, r{1u, 0u};
    for (int b = 0; b < 31; b++) {
        if ((index >> b) & 1u) r = cpoint_add(r, g);
        g = cpoint_add(g, g);
    }
    return r;
}

namespace zk {

// ---- the entries' line coefficients (core/pcs/quotients.rs:58-104, core/constraints.rs:119-134)
//
// With v an entry's value, p its power of the random coefficient and y its sample point's ordinate: a = p (conj v - v),
// c = p (conj y - y), b = v c - a y. Only c is needed entry by entry; of a and b the sums over the batch are, and those follow from
// the sums of p v and p conj v. A proof over tens of thousands of columns has as many entries: 45 ns each on a host core
// (65,000: 3 ms, 1.2 ms on four), microseconds here, and what does not depend on the coefficient is uploaded before it is drawn.
struct LineChunk { uint32_t batch, first, count, pad; };
constexpr uint32_t LINE_CHUNK = 1024;  // entries a CTA takes: a batch's sums meet in a few atomics per warp
constexpr uint32_t LINE_POW_LOG = 8;   // alpha^e = low[e mod 2^8] high[e / 2^8]

__device__ __forceinline__ qm31 line_ld(const uint32_t* p, size_t i) {
    const uint4 v = reinterpret_cast<const uint4*>(p)[i];
    return {{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ uint32_t line_warp_sum(uint32_t v) {
    return m31_reduce64(__reduce_add_sync(0xffffffffu, v & 0xffffu) + ((uint64_t)__reduce_add_sync(0xffffffffu, v >> 16) << 16));
}
__global__ void __launch_bounds__(256) quot_lines_kernel(const LineChunk* __restrict__ chunks, const uint32_t* __restrict__ batch_c, const uint32_t* __restrict__ val,
                                                         const uint32_t* __restrict__ pow, const uint32_t* __restrict__ pow_table, const uint32_t* __restrict__ values,
                                                         uint32_t* __restrict__ out_c, unsigned long long* __restrict__ sums) {
    const LineChunk ch = chunks[blockIdx.x];
    const qm31 c = line_ld(batch_c, ch.batch);
    qm31 s = qm31_zero(), sc = qm31_zero();
    for (uint32_t i = threadIdx.x; i < ch.count; i += blockDim.x) {
        const uint32_t e = pow[ch.first + i];
        const qm31 p = qm31_mul(line_ld(pow_table, e & ((1u << LINE_POW_LOG) - 1)), line_ld(pow_table, (1u << LINE_POW_LOG) + (e >> LINE_POW_LOG)));
        const qm31 v = line_ld(values, val[ch.first + i]);
        const qm31 r = qm31_mul(p, c);
        reinterpret_cast<uint4*>(out_c)[ch.first + i] = make_uint4(r.c[0], r.c[1], r.c[2], r.c[3]);
        s = qm31_add(s, qm31_mul(p, v));
        sc = qm31_add(sc, qm31_mul(p, qm31{{v.c[0], v.c[1], m31_neg(v.c[2]), m31_neg(v.c[3])}}));
    }
    unsigned long long* const at = sums + 8 * (size_t)ch.batch;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint32_t a = line_warp_sum(s.c[q]), b = line_warp_sum(sc.c[q]);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(at + q, (unsigned long long)a);
            atomicAdd(at + 4 + q, (unsigned long long)b);
        }
    }
}

// The kernels of one accumulation. d_cols: the columns' staged table; scratch_used: words of the scratch buffer that hold its inputs.
static int launch_numerators(zkb_ctx* ctx, const uint32_t* const* cols, int ncols, int log_n, const uint32_t* const* d_cols, const uint32_t* d_idx,
                             const uint32_t* d_c, int k, qm31 b_sum, int b_first, Secure4 o, size_t scratch_used) {
    size_t n = (size_t)1 << log_n;
    bool wide = n >= 4;
    for (int q = 0; q < 4; q++) wide = wide && ((uintptr_t)o.c[q] & 15) == 0;
    for (int c = 0; c < ncols; c++) wide = wide && ((uintptr_t)cols[c] & 15) == 0;
    ProfScope prof(ctx, b_first ? "quot_numerators_kernel(coefficients)" : "quot_numerators_kernel");
    // Few rows: the columns are split over the grid's second dimension, so that some 148 x 4 CTAs' worth of threads have loads on their way, sixteen
    // columns each at least. A thread walks its columns four at a time, a trip to memory each: a hundred columns of 2^13 rows on
    // eight CTAs were 35 us, of 2^17 rows 41; split, and added up, 10 + 4 and 18 + 8. Groups of fewer than 1,024 rows take narrower CTAs.
    // The pieces' sums are a launch more and as many bytes as eight columns a piece: whole -> split, 32 columns of 2^9 rows 13.2 -> 14.1 us, 2^13
    // 10.8 -> 13.2, 40 columns 13.5 -> 13.6 and 18.5 -> 16.0. Where the rows leave room for four pieces (2^17): 40 columns 20.0 -> 21.6, 48 22.7 -> 21.8; for two
    // (2^18): 80 35.1 -> 36.5, 100 41.4 -> 41.3, 112 45.6 -> 44.0, 200 75.4 -> 62.7.
    const size_t per = wide ? 4 : 2;
    const unsigned threads = n / per >= 256 ? 256u : n / per >= 32 ? (unsigned)(n / per) : 32u;
    const unsigned row_blocks = (unsigned)((n / per + threads - 1) / threads);
    const size_t scratch_free = ctx->scratch_words - scratch_used;
    const int room = (int)(148u * 1024u / (row_blocks * threads));
    int S = std::min((k + 15) / 16, room);
    S = std::min<size_t>(S, (scratch_free - 4) / (4 * n));
    if (S >= 2 && k >= (room == 2 ? 112 : room <= 4 ? 48 : 40)) {
        const int chunk = ((k + S - 1) / S + 3) / 4 * 4;
        S = (k + chunk - 1) / chunk;
        uint32_t* partial = ctx->scratch + scratch_used + ((4 - (scratch_used & 3)) & 3);  // 16-byte aligned
        dim3 grid(row_blocks, (unsigned)S);
        if (wide)
            quot_numerators_kernel<4><<<grid, threads, 0, ctx->stream>>>(d_cols, d_idx, reinterpret_cast<const uint4*>(d_c), k,
                                                                         b_sum, b_first, n, o, chunk, partial);
        else
            quot_numerators_kernel<2><<<grid, threads, 0, ctx->stream>>>(d_cols, d_idx, reinterpret_cast<const uint4*>(d_c), k,
                                                                         b_sum, b_first, n, o, chunk, partial);
        ZKB_LAUNCH_CHECK(ctx);
        if (S >= 24) quot_partial_sum_kernel<8><<<(unsigned)((4 * n + 31) / 32), 256, 0, ctx->stream>>>(partial, S, n, b_sum, b_first, o);
        else quot_partial_sum_kernel<1><<<(unsigned)((4 * n + 255) / 256), 256, 0, ctx->stream>>>(partial, S, n, b_sum, b_first, o);
        ZKB_LAUNCH_CHECK(ctx);
        return ZKB_OK;
    }
    if (wide)
        quot_numerators_kernel<4><<<(unsigned)((n / 4 + 255) / 256), 256, 0, ctx->stream>>>(
            d_cols, d_idx, reinterpret_cast<const uint4*>(d_c), k, b_sum, b_first, n, o);
    else
        quot_numerators_kernel<2><<<(unsigned)((n / 2 + 255) / 256), 256, 0, ctx->stream>>>(
            d_cols, d_idx, reinterpret_cast<const uint4*>(d_c), k, b_sum, b_first, n, o);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

static qm31 conj_q(qm31 v) { return {{v.c[0], v.c[1], m31_neg(v.c[2]), m31_neg(v.c[3])}}; }

// Below so many entries the host is done with the coefficients before a launch and its read-back would be (some 20 us).
constexpr size_t LINES_ON_DEVICE_MIN = 512;
static size_t words16(size_t n) { return (n + 3) & ~(size_t)3; }

// Uploads `n` words, through the staging ring where they fit a quarter of it.
static int upload_words(zkb_ctx* ctx, uint32_t* dst, const std::vector<uint32_t>& h) {
    if (h.empty()) return ZKB_OK;
    if (h.size() * 4 <= sizeof(void*) * (ctx->ring_cap / 4)) return upload_small(ctx, dst, h.data(), h.size());
    ZKB_CUDA(ctx, cudaMemcpyAsync(dst, h.data(), h.size() * 4, cudaMemcpyHostToDevice, ctx->stream));
    return ZKB_OK;
}

// The block: [c: 4 n][col: n][val: n][pow: n][chunks][sums: 16 words a batch]
int numerator_stage(zkb_ctx* ctx, const NumeratorEntries& e, const std::vector<NumeratorBatch>& batches, NumeratorLines& lines) {
    DeviceGuard g(ctx);
    const size_t n = e.col.size();
    const bool device = n >= LINES_ON_DEVICE_MIN;
    size_t n_chunks = 0;
    for (auto& b : batches) n_chunks += (b.count + LINE_CHUNK - 1) / LINE_CHUNK;
    const size_t o_col = 4 * n, words = o_col + 3 * words16(n) + 4 * n_chunks + 16 * batches.size();
    if (int rc = zkb_malloc(ctx, words * 4 + 16, (void**)&lines.block)) return rc;
    lines.d_c = lines.block;
    lines.d_col = lines.block + o_col;
    if (!device) return ZKB_OK;
    std::vector<uint32_t> h(3 * words16(n) + 4 * n_chunks);
    memcpy(h.data(), e.col.data(), 4 * n);
    memcpy(h.data() + words16(n), e.val.data(), 4 * n);
    memcpy(h.data() + 2 * words16(n), e.pow.data(), 4 * n);
    LineChunk* ch = reinterpret_cast<LineChunk*>(h.data() + 3 * words16(n));
    for (size_t b = 0; b < batches.size(); b++)
        for (size_t at = 0; at < batches[b].count; at += LINE_CHUNK)
            *ch++ = {(uint32_t)b, (uint32_t)(batches[b].first + at), (uint32_t)(batches[b].count - at < LINE_CHUNK ? batches[b].count - at : LINE_CHUNK), 0u};
    return upload_words(ctx, lines.d_col, h);
}

int numerator_lines(zkb_ctx* ctx, const NumeratorEntries& e, std::vector<NumeratorBatch>& batches, NumeratorLines& lines, qm31 random_coeff,
                    const qm31* h_values, const uint32_t* d_values) {
    DeviceGuard g(ctx);
    const size_t n = e.col.size(), nb = batches.size();
    if (!n) return ZKB_OK;
    std::vector<qm31> c(nb);
    for (size_t b = 0; b < nb; b++) {
        c[b] = qm31_sub(conj_q(batches[b].point_y), batches[b].point_y);
        if (batches[b].count && qm31_is_zero(c[b])) return set_error(ctx, ZKB_EINVAL, "sample point lies on the base-field circle");
    }
    std::vector<qm31> sums(2 * nb, qm31_zero());  // of p v and p conj v
    if (n < LINES_ON_DEVICE_MIN) {
        std::vector<qm31> pows(n);
        size_t top = 0;
        for (uint32_t p : e.pow) top = p > top ? p : top;
        pows.resize(top + 1);
        for (size_t k = 0; k <= top; k++) pows[k] = k ? qm31_mul(pows[k - 1], random_coeff) : qm31_one();
        std::vector<uint32_t> h(5 * n);
        for (size_t b = 0; b < nb; b++)
            for (size_t j = batches[b].first; j < batches[b].first + batches[b].count; j++) {
                const qm31 p = pows[e.pow[j]], v = h_values[e.val[j]], r = qm31_mul(p, c[b]);
                memcpy(&h[4 * j], r.c, 16);
                sums[2 * b] = qm31_add(sums[2 * b], qm31_mul(p, v));
                sums[2 * b + 1] = qm31_add(sums[2 * b + 1], qm31_mul(p, conj_q(v)));
            }
        memcpy(&h[4 * n], e.col.data(), 4 * n);
        if (int rc = upload_words(ctx, lines.d_c, h)) return rc;  // [c: 4 n][col: n], where the accumulations that follow read it
    } else {
        size_t n_chunks = 0;
        for (auto& b : batches) n_chunks += (b.count + LINE_CHUNK - 1) / LINE_CHUNK;
        uint32_t *d_val = lines.d_col + words16(n), *d_pow = d_val + words16(n), *d_chunks = d_pow + words16(n), *d_sums = d_chunks + 4 * n_chunks;
        // [the batches' c][alpha^0 ... alpha^255][alpha^(256 k)]
        const size_t n_low = (size_t)1 << LINE_POW_LOG;
        uint32_t top = 0;
        for (uint32_t p : e.pow) top = p > top ? p : top;
        const size_t n_high = (top >> LINE_POW_LOG) + 1;
        std::vector<qm31> h(nb + n_low + n_high);
        for (size_t b = 0; b < nb; b++) h[b] = c[b];
        qm31* low = h.data() + nb;
        for (size_t k = 0; k < n_low; k++) low[k] = k ? qm31_mul(low[k - 1], random_coeff) : qm31_one();
        const qm31 step = qm31_mul(low[n_low - 1], random_coeff);
        for (size_t k = 0; k < n_high; k++) low[n_low + k] = k ? qm31_mul(low[n_low + k - 1], step) : qm31_one();
        uint32_t* d_tab = nullptr;
        if (int rc = zkb_malloc(ctx, h.size() * 16, (void**)&d_tab)) return rc;
        std::vector<uint32_t> hw(4 * h.size());
        memcpy(hw.data(), h.data(), h.size() * 16);
        int rc = upload_words(ctx, d_tab, hw);
        cudaError_t err = cudaSuccess;
        if (rc == ZKB_OK) err = cudaMemsetAsync(d_sums, 0, 64 * nb, ctx->stream);
        if (rc == ZKB_OK && err == cudaSuccess) {
            ProfScope prof(ctx, "quot_lines_kernel");
            quot_lines_kernel<<<(unsigned)n_chunks, 256, 0, ctx->stream>>>(reinterpret_cast<const LineChunk*>(d_chunks), d_tab, d_val, d_pow, d_tab + 4 * nb, d_values,
                                                                           lines.d_c, reinterpret_cast<unsigned long long*>(d_sums));
            err = cudaGetLastError();
        }
        std::vector<unsigned long long> w(8 * nb);
        if (rc == ZKB_OK && err == cudaSuccess) err = cudaMemcpyAsync(w.data(), d_sums, 64 * nb, cudaMemcpyDeviceToHost, ctx->stream);
        if (rc == ZKB_OK && err == cudaSuccess) err = cudaStreamSynchronize(ctx->stream);
        zkb_free(ctx, d_tab);
        if (rc) return rc;
        if (err != cudaSuccess) return set_error(ctx, ZKB_ECUDA, "quotient lines: %s", cudaGetErrorString(err));
        for (size_t b = 0; b < nb; b++)
            for (int q = 0; q < 4; q++) {
                sums[2 * b].c[q] = (uint32_t)(w[8 * b + q] % P);
                sums[2 * b + 1].c[q] = (uint32_t)(w[8 * b + 4 + q] % P);
            }
    }
    for (size_t b = 0; b < nb; b++) {
        batches[b].first_linear = qm31_sub(sums[2 * b + 1], sums[2 * b]);
        batches[b].b_sum = qm31_sub(qm31_mul(c[b], sums[2 * b]), qm31_mul(batches[b].point_y, batches[b].first_linear));
    }
    return ZKB_OK;
}

// The combination of the columns' polynomials is itself a polynomial of their degree, so it can be taken of the coefficients, a
// blow-up fewer of them, and extended: four columns' worth of transform in the place of most of the reading. (The constant comes off
// coefficient 0, whose basis element is 1.) 256 columns of 2^20 at blow-up 4: 810 us from the evaluations, 206 + 86 from the coefficients.
// The transform of four columns costs some 17 us and as much as reading 21 columns' evaluations; the line lies a quarter above that, at 24 M words and 28
// columns saved, where nothing measured is slower. Numerators and transforms of a proof from the evaluations -> from the coefficients, blow-up 2: 64 columns of
// 2^19 498 -> 505 us, of 2^20 945 -> 943, 150 of 2^18 560 -> 565 (all left as they were), 256 of 2^17 483 -> 475, 4,500 of 2^13 476 -> 467; blow-up 4: 64 of 2^18
// 417 -> 422 and 100 of 2^17 326 -> 327 (left), 256 of 2^16 406 -> 383, 200 of 2^17 611 -> 581; blow-up 16: 100 of 2^20 2,380 -> 2,231. Coefficients that do not
// start on 16 bytes are left too.
static bool numerators_of_coeffs(const uint32_t* const* coeffs, int ncols, int log_n, int log_coeff, size_t k) {
    if ((k << log_n) - (k << log_coeff) < ((size_t)24 << 20) + ((size_t)28 << log_n)) return false;
    for (int c = 0; c < ncols; c++) if (((uintptr_t)coeffs[c] & 15) != 0) return false;
    return true;
}

int numerator_run(zkb_ctx* ctx, const uint32_t* const* cols, const uint32_t* const* coeffs, int ncols, int log_n, int log_coeff, const NumeratorLines& lines,
                  const NumeratorBatch& batch, uint32_t* const out[4]) {
    DeviceGuard g(ctx);
    const bool of_coeffs = numerators_of_coeffs(coeffs, ncols, log_n, log_coeff, batch.count);
    if (of_coeffs) {
        cols = coeffs;
        ZKB_CHECK_ARG(ctx, log_coeff >= 2 && log_coeff < log_n && log_n <= ctx->max_log);
    }
    for (int c = 0; c < ncols; c++) ZKB_CHECK_ARG(ctx, cols[c] != nullptr && ((uintptr_t)cols[c] & 7) == 0);
    void** d_cols;
    if (int rc = stage_ptrs(ctx, (const void* const*)cols, ncols, &d_cols)) return rc;
    const size_t n = (size_t)1 << log_coeff;
    uint32_t* combined = nullptr;
    if (of_coeffs)
        if (int rc = zkb_malloc(ctx, 16 * n, (void**)&combined)) return rc;
    Secure4 o;
    for (int q = 0; q < 4; q++) o.c[q] = of_coeffs ? combined + q * n : out[q];
    int rc = launch_numerators(ctx, cols, ncols, of_coeffs ? log_coeff : log_n, (const uint32_t* const*)d_cols, lines.d_col + batch.first,
                               lines.d_c + 4 * batch.first, (int)batch.count, batch.b_sum, of_coeffs ? 1 : 0, o, 0);
    if (!of_coeffs) return rc;
    if (rc == ZKB_OK) rc = zkb_lde_cols(ctx, o.c, 4, log_coeff, out, log_n);
    zkb_free(ctx, combined);
    return rc;
}

}  // namespace zk

using namespace zk;

extern "C" {

int zkb_quot_numerators(zkb_ctx* ctx, const uint32_t* const* cols, int ncols, int log_n, const uint32_t* h_col_idx,
                        const uint32_t* h_b, const uint32_t* h_c, int k, uint32_t* const out[4]) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, cols && ncols > 0 && log_n >= 1 && log_n <= 30 && k >= 0 && out);
    ZKB_CHECK_ARG(ctx, k == 0 || (h_col_idx && h_b && h_c));
    ZKB_CHECK_ARG(ctx, (size_t)k * 5 <= ctx->scratch_words);
    Secure4 o;
    for (int q = 0; q < 4; q++) {
        ZKB_CHECK_ARG(ctx, out[q] != nullptr && ((uintptr_t)out[q] & 7) == 0);
        o.c[q] = out[q];
    }
    for (int j = 0; j < k; j++) ZKB_CHECK_ARG(ctx, h_col_idx[j] < (uint32_t)ncols);
    for (int c = 0; c < ncols; c++) ZKB_CHECK_ARG(ctx, cols[c] != nullptr && ((uintptr_t)cols[c] & 7) == 0);
    qm31 b_sum = qm31_zero();
    for (int j = 0; j < k; j++) b_sum = qm31_add(b_sum, qm31{{h_b[4 * j], h_b[4 * j + 1], h_b[4 * j + 2], h_b[4 * j + 3]}});
    DeviceGuard g(ctx);
    void** d_cols;
    int rc = stage_ptrs(ctx, (const void* const*)cols, ncols, &d_cols);
    if (rc) return rc;
    // coefficient table and column indices go through the scratch buffer
    uint32_t* d_c = ctx->scratch;
    uint32_t* d_idx = ctx->scratch + (size_t)4 * k;
    if (k) {
        ZKB_CUDA(ctx, cudaMemcpyAsync(d_c, h_c, (size_t)k * 16, cudaMemcpyHostToDevice, ctx->stream));
        ZKB_CUDA(ctx, cudaMemcpyAsync(d_idx, h_col_idx, (size_t)k * 4, cudaMemcpyHostToDevice, ctx->stream));
    }
    return launch_numerators(ctx, cols, ncols, log_n, (const uint32_t* const*)d_cols, d_idx, d_c, k, b_sum, 0, o, (size_t)5 * k);
}

int zkb_quot_combine(zkb_ctx* ctx, int n_acc, const uint32_t* const* acc_cols, const int* h_acc_log,
                     const uint32_t* h_first_lin, const uint32_t* h_points, int lifting_log, uint32_t* const out[4]) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, lifting_log >= 1 && lifting_log <= ctx->max_log);
    return zkb_quot_combine_rows(ctx, n_acc, acc_cols, h_acc_log, h_first_lin, h_points, lifting_log, 0, (size_t)1 << lifting_log, out);
}

int zkb_quot_combine_rows(zkb_ctx* ctx, int n_acc, const uint32_t* const* acc_cols, const int* h_acc_log, const uint32_t* h_first_lin,
                          const uint32_t* h_points, int lifting_log, size_t row_begin, size_t n_rows, uint32_t* const out[4]) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, n_acc >= 1 && acc_cols && h_acc_log && h_first_lin && h_points && out);
    ZKB_CHECK_ARG(ctx, lifting_log >= 1 && lifting_log <= ctx->max_log);
    ZKB_CHECK_ARG(ctx, n_rows >= 1 && row_begin + n_rows <= ((size_t)1 << lifting_log));
    const bool whole = row_begin == 0 && n_rows == ((size_t)1 << lifting_log);
    // a shard starts on a row that every lifted accumulation starts a pair on, and small domains are not sharded
    ZKB_CHECK_ARG(ctx, whole || (lifting_log > 2 && (row_begin & 1) == 0 && (n_rows & 1) == 0));
    Secure4 o;
    for (int q = 0; q < 4; q++) {
        ZKB_CHECK_ARG(ctx, out[q] != nullptr);
        o.c[q] = out[q];
    }
    for (int a = 0; a < n_acc; a++) ZKB_CHECK_ARG(ctx, h_acc_log[a] >= 1 && h_acc_log[a] <= lifting_log);
    for (int a = 0; a < n_acc; a++)
        ZKB_CHECK_ARG(ctx, whole || (row_begin & (((size_t)2 << (lifting_log - h_acc_log[a])) - 1)) == 0);
    DeviceGuard g(ctx);
    size_t n = n_rows;
    for (int base = 0; base < n_acc; base += MAX_ACCS) {
        CombineArgs args;
        memset(&args, 0, sizeof(args));
        args.n_acc = n_acc - base < MAX_ACCS ? n_acc - base : MAX_ACCS;
        args.first = base == 0;
        for (int z = 0; z < args.n_acc; z++) {
            int a = base + z;
            for (int q = 0; q < 4; q++) {
                ZKB_CHECK_ARG(ctx, acc_cols[4 * a + q] != nullptr);
                args.acc[z][q] = acc_cols[4 * a + q];
            }
            args.log_ratio[z] = lifting_log - h_acc_log[a];
            for (int q = 0; q < 4; q++) args.first_lin[z].c[q] = h_first_lin[4 * a + q];
            const uint32_t* pt = h_points + 8 * a;  // x[4], y[4]
            args.prx[z] = {pt[0], pt[1]};
            args.pix[z] = {pt[2], pt[3]};
            args.pry[z] = {pt[4], pt[5]};
            args.piy[z] = {pt[6], pt[7]};
        }
        if (lifting_log <= 2) {
            int hl = lifting_log - 1;
            cpoint p0 = host_point_q((1u << (29 - hl)) & 0x7fffffffu);
            cpoint p1 = hl ? host_point_q(((1u << (29 - hl)) + (1u << (31 - hl))) & 0x7fffffffu) : p0;
            quot_combine_small_kernel<<<1, 32, 0, ctx->stream>>>(args, lifting_log, o, p0.x, p0.y, p1.x, p1.y);
        } else {
            ProfScope prof(ctx, "quot_combine_kernel");
            auto launch = [&](auto kernel, int rows) { kernel<<<(unsigned)((n / rows + 255) / 256), 256, 0, ctx->stream>>>(args, lifting_log, o, ctx->tw, row_begin, n_rows); };
            // Several rows a thread from 2^17 rows on: below, where a row a thread does not fill the GPU, they only make the chain longer. One accumulation
            // over 2^16 rows: 8.2 us a row a thread, 8.8 four; two 8.8 and 10.6, four 10.7 and 10.8 (over 2^10 7.1 and 8.8, 7.8 and 10.5, 8.7 and 10.8); over 2^17
            // 10.4 and 8.8, 10.7 and 10.6, 14.6 and 12.7.
            if (n < ((size_t)1 << 17) || n % 4 || args.n_acc > 4) launch(quot_combine_kernel<MAX_ACCS, 1>, 1);
            else if (args.n_acc == 1) launch(quot_combine_kernel<1, 4>, 4);
            else if (args.n_acc == 2) launch(quot_combine_kernel<2, 4>, 4);
            else launch(quot_combine_kernel<4, 2>, 2);
        }
        ZKB_LAUNCH_CHECK(ctx);
    }
    return ZKB_OK;
}

int zkb_accumulate(zkb_ctx* ctx, uint32_t* const col[4], const uint32_t* const other[4], size_t n) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, col && other);
    if (n == 0) return ZKB_OK;
    Secure4 a;
    Secure4C b;
    for (int q = 0; q < 4; q++) {
        ZKB_CHECK_ARG(ctx, col[q] != nullptr && other[q] != nullptr);
        a.c[q] = col[q];
        b.c[q] = other[q];
    }
    DeviceGuard g(ctx);
    accumulate_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(a, b, n);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

int zkb_lift_accumulate(zkb_ctx* ctx, uint32_t* const dst[4], int log_dst, const uint32_t* const src[4], int log_src) {
    if (!ctx) return ZKB_EINVAL;
    ZKB_CHECK_ARG(ctx, dst && src && log_src >= 1 && log_src <= log_dst && log_dst <= 30);
    Secure4 a;
    Secure4C b;
    for (int q = 0; q < 4; q++) {
        ZKB_CHECK_ARG(ctx, dst[q] != nullptr && src[q] != nullptr);
        a.c[q] = dst[q];
        b.c[q] = src[q];
    }
    DeviceGuard g(ctx);
    size_t n = (size_t)1 << log_dst;
    ProfScope prof(ctx, "lift_accumulate_kernel");
    lift_accumulate_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(a, log_dst, b, log_dst - log_src);
    ZKB_LAUNCH_CHECK(ctx);
    return ZKB_OK;
}

}  // extern "C"
