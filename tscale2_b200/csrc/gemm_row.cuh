// Row-wise steps that run behind a contraction in its own launch.
#pragma once
#include "gemm.cuh"

namespace ts2 {

// What becomes of a product, 128 columns of a row at a time
enum RowForm {
    ROW_PLAIN = 0, // Epilogue::out_kind, as any contraction
    ROW_NORM,      // C = c_in + product (fp32); n_fast = tile normalisation of C, n16 optionally (tilenorm_forward)
    ROW_NORM_BWD,  // product = gradient of the normalised x: g = (add ? g : 0) + its tile-norm backward (tilenorm_backward)
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
};

} // namespace ts2
