// Row-wise steps that run behind a contraction in its own launch.
#pragma once
#include "gemm.cuh"

namespace ts2 {

// What pairs of CTAs make of their product (Epilogue::row; widths are multiples of 128 but in the last form)
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

} // namespace ts2
