// Row-wise steps that run behind a contraction in its own launch.
#pragma once
#include "gemm.cuh"

namespace ts2 {

// What becomes of the product, 128 columns of a row at a time (widths are multiples of 128 in all forms but the first and the
// last).  The row kernel (gemm_row.cu) has the third, pairs of CTAs (Epilogue::row) all but the first.
enum RowForm {
    ROW_PLAIN = 0, // Epilogue::out_kind, as any contraction
    ROW_NORM,      // C = c_in + product (fp32); n_fast = tile normalisation of C, n16 optionally (tilenorm_forward)
    ROW_NORM_BWD,  // product = gradient of the normalised x: g = (add ? g : 0) + its tile-norm backward (tilenorm_backward)
    ROW_LSE,       // product = logits, base 2: per row and 64 columns {maximum, sum of 2^(x - maximum)}, the target's logit
};
struct RowOp {
    int form = ROW_PLAIN;
    // ROW_NORM
    float s_act = 1.f;
    void *n_fast = nullptr; // in the format of the contraction's operands
    __half *n16 = nullptr;
    // ROW_NORM_BWD; the product is multiplied with dyn first
    const float *x = nullptr, *dyn = nullptr;
    float *g = nullptr;
    int add = 0;
    unsigned *absmax = nullptr, *health = nullptr;
    unsigned step_no = 0;
    // ROW_LSE: bias [N] or null, target [M] (negative: none); partial [4 x ceil(N / 256)][M], target_logit [M]
    const float *bias = nullptr;
    const int *target = nullptr;
    float2 *partial = nullptr;
    float *target_logit = nullptr;
};

// First contraction (K contiguous in both operands) with ROW_NORM_BWD behind it, and optionally a second one beside it in the same
// launch: token-major operands, fp32 output or added to it, independent of the first.
struct RowGemm {
    GemmArgs a;
    RowOp op;
    const GemmArgs *second = nullptr;
};
// K split and estimated time (us) of one contraction in this kernel
double gemm_row_plan(int device, int kind, int64_t M, int64_t N, int64_t K, int *splits);
// whether gemm_row() is the faster way for this shape and the backward of a normalisation behind it
bool gemm_row_takes(int device, int kind, int64_t M, int64_t N, int64_t K);
// whether the second contraction fits beside the first
bool gemm_row_takes_pair(int device, const GemmArgs &a, const GemmArgs &second);
int gemm_row(const RowGemm &r);

} // namespace ts2
