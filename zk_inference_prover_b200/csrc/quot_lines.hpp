// The prover's quotient numerators from values that are on the device (quotients.cu, poly_eval.cu); internal to the library.
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>

#include "m31.cuh"

struct zkb_ctx;

namespace zk {

// zkb_eval_at_point_cols with the values left on the device (4 words a column), stream-ordered.
int eval_at_point_device(zkb_ctx* ctx, const uint32_t* const* coeffs, int ncols, int log_n, const uint32_t h_point[8], uint32_t* d_out);

// One accumulation: the columns of one size sampled at one point. Its entries are [first, first + count) of the entry arrays.
struct NumeratorBatch {
    qm31 point_y;
    size_t first, count;
    qm31 first_linear, b_sum;  // results: the sums of the line coefficients a and b
};

// Entry j: the column (its place in its size's table), the place of its value in the value array, its power of the random coefficient.
struct NumeratorEntries { std::vector<uint32_t> col, val, pow; };

// The entries' columns and coefficients c on the device. stage uploads what does not depend on the random coefficient; lines fills in
// the coefficients and the batches' sums (one round trip). values: n_values on the host and, the same, on the device.
struct NumeratorLines {
    uint32_t *d_col = nullptr, *d_c = nullptr;
    uint32_t* block = nullptr;  // the allocation behind them; zkb_free it
};
int numerator_stage(zkb_ctx* ctx, const NumeratorEntries& e, const std::vector<NumeratorBatch>& batches, NumeratorLines& lines);
int numerator_lines(zkb_ctx* ctx, const NumeratorEntries& e, std::vector<NumeratorBatch>& batches, NumeratorLines& lines, qm31 random_coeff,
                    const qm31* h_values, const uint32_t* d_values);
// cols: the columns' 2^log_n evaluations; coeffs: the 2^log_coeff coefficients they are the extension of.
int numerator_run(zkb_ctx* ctx, const uint32_t* const* cols, const uint32_t* const* coeffs, int ncols, int log_n, int log_coeff, const NumeratorLines& lines,
                  const NumeratorBatch& batch, uint32_t* const out[4]);

}  // namespace zk
