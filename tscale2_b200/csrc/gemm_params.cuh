// What the contraction kernels of gemm.cu (one CTA per tile) and gemm_pair.cu (two CTAs per tile) share.
#pragma once
#include "gemm.cuh"
#include <cuda.h>

namespace ts2 {

static constexpr int BM = 128;
static constexpr int STAGE_ROW_BYTES = 128; // one swizzle row

struct GemmParams {
    int M, N;
    int m_tiles, n_tiles, splits;
    int n_fast;        // tile order: consecutive tiles walk N first (the CTAs of a wave share A rows) or M first (share B rows)
    int k_blocks;      // total K blocks (one block = one pipeline stage)
    int kb_per_split;
    uint32_t idesc;
    void *C;
    long long ldc;
    float alpha;
    const float *dyn_scale, *dyn_scale2, *row_scale, *col_scale, *c_in;
    int out_kind;
    float *workspace;
    int32_t *status;
    // dynamic unit scheduler: {next unit, finished CTAs}, both zero between launches (the last CTA to finish resets
    // them); null: unit i of CTA b is b + i * gridDim.x
    int *sched = nullptr;
    // grouped forms (mixture-of-experts): 0 none; 1 every 128-row M tile belongs to one group (tile_group[m_tile],
    // negative: skip) and reads B rows [group * group_rows_b + n]; 2 the K range of a unit is the row segment of
    // its group (group_kptr[g] .. group_kptr[g+1], multiples of the K block) and C moves by c_group_stride per group
    int group_mode, groups;
    const int *tile_group;
    int group_rows_b;
    const int *group_kptr;
    long long c_group_stride;
    int bk;
    int tma_store; // the epilogue stages 32-row blocks in shared memory and writes them with TMA (tmC)
    // gated-activation form (see Epilogue in gemm.cuh): a tile is 128 "wide" columns [nt * 128, +128) and the 128
    // "gate" columns pair_stride further on
    int pair_stride = 0;
    void *act_out = nullptr;
    long long act_ld = 0;
    float *act_scale = nullptr;
    float act_mult = 1.f;
    int act_kind = 0; // format of act_out: 0 e4m3, 1 fp16, 2 int8
    float *bwd_dscale = nullptr; // backward of the attention gate (see Epilogue)
    // tile normalisation behind the product, or its backward (see Epilogue)
    int norm16 = 0, norm_add = 0;
    const float *norm_dyn = nullptr;
    unsigned *norm_absmax = nullptr, *norm_health = nullptr;
    unsigned norm_step = 0;
    // log-sum-exp of the row
    const float *lse_bias = nullptr;
    const int *lse_target = nullptr;
    float2 *lse_partial = nullptr;
    float *lse_logit = nullptr;
};

// Forms of the epilogue of gemm_pair.cu: fp32 output, accumulate form and partial tiles; fp16 / bf16 output; gated
// activation; its backward; backward of the attention gate; residual input + tile normalisation; backward of the latter;
// log-sum-exp of the row
enum PairForm { P_F32, P_16, P_GATED, P_ACT_BWD, P_GATE_BWD, P_NORM, P_NORM_BWD, P_LSE };
// gemm_pair.cu: the contraction on pairs of CTAs (tiles of 256 x 256).  tmB's box is 128 rows (K-major) or one K block
// (token-major); tmC's and tmCin's are 32 rows x 128 bytes (P_GATED: tmC 32 x 64 bytes).  grid: CTAs, an even number.
// P_ACT_BWD: tmC 32 rows x 64 bytes, tmCin [wide | gate] in 32 rows x 128; P_GATE_BWD: the same, and tmX: o, tmY: dout, both
// 32 rows x 128; P_NORM: tmX: n_fast, tmY: n16; P_NORM_BWD: tmX: x, tmCin and tmC: g; tmX, tmY otherwise unused
int gemm_pair_launch(int device, cudaStream_t stream, int es, int mma, bool mn, PairForm form, int grid, const CUtensorMap &tmA,
                     const CUtensorMap &tmB, const CUtensorMap &tmC, const CUtensorMap &tmCin, const CUtensorMap &tmX, const CUtensorMap &tmY,
                     const GemmParams &p);

// instruction descriptor of a contraction on bm x bn tiles
uint32_t gemm_instr_desc(int kind, bool mn, int bm, int bn);
// timing statistics (gemm_timing_enable): events around a launch, null where they are off
struct GemmTimed {
    cudaEvent_t a = nullptr, b = nullptr;
};
GemmTimed gemm_timed_begin(cudaStream_t stream);
void gemm_timed_end(const GemmTimed &t, cudaStream_t stream, double flops, double bytes, int tag);

} // namespace ts2
