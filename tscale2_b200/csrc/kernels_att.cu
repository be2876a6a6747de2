// Attention part of the training step: per-head normalisation + RoPE of Q/K/V and
// their backward, and the attention core over one inclusive key span per node
// (ComputeValLookup / GradQ / GradK, src/gpt/compute/layer_att_reference.h:41-212):
//   dp(from,to) = q_from . k_to * sqrt(1/128) * 0.5/ln2 - slope * (from - to)
//   weights 2^(dp - maxDP) with maxDP >= 0 and an extra zero vector of weight 2^-maxDP.
// This file holds the warp-per-row formulation (fp32 math, coalesced 8-byte loads), kept as an
// independent second formulation for the tests; the engine runs the tcgen05 kernels of
// kernels_att_tc.cu (kernels_att_mma.cu holds an mma.sync formulation, also kept for the tests).
#include "kernels.cuh"
#include "row_math.cuh"

namespace ts2 {

static constexpr int WARPS = 8;
static constexpr int THREADS = WARPS * 32;

static int grid_for(const Ctx &c, long long warp_items)
{
    long long blocks = ceil_div(warp_items, WARPS);
    long long cap = (long long)sm_count(c.device) * 8;
    return (int)std::max<long long>(1, std::min(blocks, cap));
}

// for the grid-stride kernels that carry most of the bytes: exactly the blocks that are resident at once.  With a
// fixed 8 blocks per SM a kernel that fits 5 (48 registers) ran a second, partly filled wave at a fraction of the
// bandwidth.
template <typename K>
static int grid_for(const Ctx &c, K kernel, long long warp_items)
{
    long long blocks = ceil_div(warp_items, WARPS);
    long long cap = (long long)sm_count(c.device) * resident_blocks(c.device, (const void *)kernel, THREADS);
    return (int)std::max<long long>(1, std::min(blocks, cap));
}

#define WARP_ITEM_LOOP(total) \
    const int lane = threadIdx.x & 31; \
    for (unsigned item = blockIdx.x * WARPS + (threadIdx.x >> 5), total_items = (unsigned)(total); item < total_items; \
         item += gridDim.x * WARPS)

// AttDotScale = CalcDotScale(128) * ATT_DOTPRODUCT_SCALE / LOG2 (layer_att_reference.h:30-33)
__host__ __device__ inline float att_dot_scale() { return sqrtf(1.0f / 128) * (0.5f / 0.693147f) * 1.0f; }

// rope[t][2i] = cos(t * theta^(-2i/128)), rope[t][2i+1] = sin(...)   (TRopeComputer, src/gpt/att/rope.cpp:4-24)
__global__ void fill_rope_kernel(float *__restrict__ rope, int T)
{
    grid_dep_wait();
    const long long total = (long long)T * 64;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int t = (int)(i / 64), k = (int)(i % 64);
        const float freq = (float)exp(-log(500000.0) * (k * 2. / 128));
        const float angle = (float)t * freq;
        rope[(size_t)t * 128 + 2 * k] = (float)cos((double)angle);
        rope[(size_t)t * 128 + 2 * k + 1] = (float)sin((double)angle);
    }
}

int fill_rope(const Ctx &c, float *rope, int T)
{
    TS2_LAUNCH((fill_rope_kernel), std::max(1, std::min(T, 1024)), 64, 0, c.stream, rope, T);
    return TS2_OK;
}

// The two kernels below give half a warp to a (node, head): lane = 8 consecutive elements, 16-byte accesses to the fp16
// arrays, and one set of addresses, tests and shuffles for two items.  With a warp per item and 8-byte accesses they were
// bound by instruction issue; 65536 nodes x 12 heads, e4m3: forward 233 -> 193 us (1.2 GB), backward 272 -> 208 us (1.3 GB).

__global__ void att_post_forward_kernel(const __half *__restrict__ qkvg, const float *__restrict__ rope, int T, int H,
                                        __half *__restrict__ q, __half *__restrict__ k, __half *__restrict__ v,
                                        float *__restrict__ qscale, float *__restrict__ vscale)
{
    grid_dep_wait();
    const int Q = H * TILE;
    const unsigned items = (unsigned)((long long)T * H);
    WARP_ITEM_LOOP(((long long)T * H + 1) / 2)
    {
        const unsigned it = 2 * item + (lane >> 4);
        const bool ok = it < items;
        const size_t t = ok ? it / H : 0;
        const int h = ok ? (int)(it % H) : 0, e = (lane & 15) * 8;
        const __half *src = qkvg + t * 4 * Q + h * TILE + e;
        const uint4 rq = *(const uint4 *)src, rk = *(const uint4 *)(src + Q), rv = *(const uint4 *)(src + 2 * Q);
        const float4 c0 = *(const float4 *)(rope + t * 128 + e), c1 = *(const float4 *)(rope + t * 128 + e + 4);
        float x[8], y[8];
        half8_to_float(rq, x);
        half8_to_float(rv, y);
        const float sq = tile_scale(half_warp_sum(dot8(x, x))), sv = tile_scale(half_warp_sum(dot8(y, y)));
        if (!ok)
            continue;
        const size_t off = t * Q + h * TILE + e;
        scale8(x, sq);
        rope8(x, c0, c1, 1.f);
        *(uint4 *)(q + off) = float_to_half8(x);
        scale8(y, sv);
        *(uint4 *)(v + off) = float_to_half8(y);
        half8_to_float(rk, x);
        rope8(x, c0, c1, 1.f);
        *(uint4 *)(k + off) = float_to_half8(x);
        if ((lane & 15) == 0) {
            qscale[t * H + h] = sq;
            vscale[t * H + h] = sv;
        }
    }
}

int att_post_forward(const Ctx &c, const __half *qkvg, const float *rope, int T, int H, __half *q, __half *k, __half *v, float *qscale,
                     float *vscale)
{
    TS2_LAUNCH((att_post_forward_kernel), grid_for(c, att_post_forward_kernel, ((long long)T * H + 1) / 2), THREADS, 0, c.stream, qkvg, rope, T, H,
               q, k, v, qscale, vscale);
    return TS2_OK;
}

// GT: type of the incoming gradients (float or __half)
template <int FT>
__device__ __forceinline__ void store_operand8(void *d, size_t idx, const float (&v)[8])
{
    if constexpr (FT == 0) {
        __nv_fp8x4_e4m3 lo(make_float4(v[0], v[1], v[2], v[3])), hi(make_float4(v[4], v[5], v[6], v[7]));
        *(uint2 *)((uint8_t *)d + idx) = make_uint2(lo.__x, hi.__x);
    } else {
        *(uint4 *)((__half *)d + idx) = float_to_half8(v);
    }
}
template <typename GT>
struct Grad8 { // eight values as they are in memory
    uint4 w[sizeof(GT) / 2];
    __device__ __forceinline__ void load(const GT *p)
    {
#pragma unroll
        for (int i = 0; i < (int)sizeof(GT) / 2; ++i)
            w[i] = ((const uint4 *)p)[i];
    }
    __device__ __forceinline__ void get(float (&f)[8]) const
    {
        if constexpr (sizeof(GT) == 2) {
            half8_to_float(w[0], f);
        } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                f[4 * i] = __uint_as_float(w[i].x), f[4 * i + 1] = __uint_as_float(w[i].y);
                f[4 * i + 2] = __uint_as_float(w[i].z), f[4 * i + 3] = __uint_as_float(w[i].w);
            }
        }
    }
};

template <int FT, typename GT>
__global__ void att_post_backward_kernel(const GT *__restrict__ dq, const GT *__restrict__ dk, const GT *__restrict__ dv,
                                         const __half *__restrict__ q, const __half *__restrict__ v, const float *__restrict__ qscale,
                                         const float *__restrict__ vscale, const float *__restrict__ rope,
                                         const float *__restrict__ sko_k, int T, int H, void *__restrict__ d4)
{
    grid_dep_wait();
    const int Q = H * TILE;
    const float kfold = __ldg(sko_k);
    const unsigned items = (unsigned)((long long)T * H);
    WARP_ITEM_LOOP(((long long)T * H + 1) / 2)
    {
        const unsigned it = 2 * item + (lane >> 4);
        const bool ok = it < items;
        const size_t t = ok ? it / H : 0;
        const int h = ok ? (int)(it % H) : 0, e = (lane & 15) * 8;
        const size_t off = t * Q + h * TILE + e;
        Grad8<GT> gq, gk, gv;
        gq.load(dq + off);
        gk.load(dk + off);
        gv.load(dv + off);
        const uint4 rq = *(const uint4 *)(q + off), rv = *(const uint4 *)(v + off);
        const float4 c0 = *(const float4 *)(rope + t * 128 + e), c1 = *(const float4 *)(rope + t * 128 + e + 4);
        const float sq = qscale[t * H + h], sv = vscale[t * H + h];
        float x[8], g[8], y[8], u[8];
        half8_to_float(rq, x);
        gq.get(g);
        half8_to_float(rv, y);
        gv.get(u);
        const float pq = half_warp_sum(dot8(x, g)) * (1.f / 128), pv = half_warp_sum(dot8(y, u)) * (1.f / 128);
        if (!ok)
            continue;
        const size_t out = t * 4 * Q + h * TILE + e;
        // q: tile-norm backward in the rotated frame (the rotation is orthogonal), then rotate back
#pragma unroll
        for (int i = 0; i < 8; ++i)
            g[i] -= x[i] * pq;
        rope8(g, c0, c1, -1.f);
        scale8(g, sq);
        store_operand8<FT>(d4, out, g);
        // v: tile-norm backward
#pragma unroll
        for (int i = 0; i < 8; ++i)
            u[i] = sv * (u[i] - y[i] * pv);
        store_operand8<FT>(d4, out + 2 * Q, u);
        // k: rotate back; the matrix scale of K is folded in here so that the 4-way dX contraction
        // can use scale-free weights for every block
        gk.get(g);
        rope8(g, c0, c1, -1.f);
        scale8(g, kfold);
        store_operand8<FT>(d4, out + Q, g);
    }
}

int att_post_backward(const Ctx &c, const void *dq, const void *dk, const void *dv, bool grads16, const __half *q, const __half *v,
                      const float *qscale, const float *vscale, const float *rope, const float *sko_k, int T, int H, void *d4)
{
#define TS2_POST_BWD(FT_, GT_)                                                                                          \
    TS2_LAUNCH((att_post_backward_kernel<FT_, GT_>), grid_for(c, att_post_backward_kernel<FT_, GT_>, ((long long)T * H + 1) / 2), THREADS, 0, c.stream, \
               (const GT_ *)dq, (const GT_ *)dk, (const GT_ *)dv, q, v, qscale, vscale, rope, sko_k, T, H, d4)
    if (c.ft == 0 && grads16)
        TS2_POST_BWD(0, __half);
    else if (c.ft == 0)
        TS2_POST_BWD(0, float);
    else if (grads16)
        TS2_POST_BWD(1, __half);
    else
        TS2_POST_BWD(1, float);
#undef TS2_POST_BWD
    return TS2_OK;
}

// ---------------------------------------------------------------------------------
// attention core, one warp per (node, head)

__global__ void attention_forward_kernel(const __half *__restrict__ q, const __half *__restrict__ k, const __half *__restrict__ v,
                                         const int *__restrict__ span_start, const int *__restrict__ span_finish, int T, int H,
                                         float slope, __half *__restrict__ o, float *__restrict__ lse)
{
    grid_dep_wait();
    const int Q = H * TILE;
    const float ds = att_dot_scale();
    WARP_ITEM_LOOP((long long)T * H)
    {
        const int t = (int)(item / H), h = (int)(item % H), off = h * TILE + lane * 4;
        const float4 qv = load_half4(q + (size_t)t * Q + off);
        float m = 0.f, S = 1.f; // running maximum (never below 0) and sum, including the zero vector of weight 2^-m
        float4 acc = make_float4(0, 0, 0, 0);
        const int s0 = span_start[t], s1 = span_finish[t];
        for (int to = s0; to <= s1; ++to) {
            const float4 kv = load_half4(k + (size_t)to * Q + off);
            const float dp = warp_sum(dot4(qv, kv)) * ds - slope * (float)(t - to);
            if (dp > m) {
                const float r = exp2f(m - dp);
                S *= r;
                acc = scale4(acc, r);
                m = dp;
            }
            const float w = exp2f(dp - m);
            S += w;
            acc = axpy4(w, load_half4(v + (size_t)to * Q + off), acc);
        }
        store_half4(o + (size_t)t * Q + off, scale4(acc, 1.f / S));
        if (lane == 0)
            lse[(size_t)t * H + h] = m + log2f(S);
    }
}

int attention_forward_rowwise(const Ctx &c, const __half *q, const __half *k, const __half *v, const int *span_start,
                              const int *span_finish, int T, int H, float slope, __half *o, float *lse)
{
    TS2_LAUNCH((attention_forward_kernel), grid_for(c, (long long)T * H), THREADS, 0, c.stream, q, k, v, span_start, span_finish, T, H,
               slope, o, lse);
    return TS2_OK;
}

__global__ void attention_dq_kernel(const __half *__restrict__ q, const __half *__restrict__ k, const __half *__restrict__ v,
                                    const __half *__restrict__ dout, const float *__restrict__ lse, const float *__restrict__ dscale,
                                    const int *__restrict__ span_start, const int *__restrict__ span_finish, int T, int H, float slope,
                                    float *__restrict__ dq)
{
    grid_dep_wait();
    const int Q = H * TILE;
    const float ds = att_dot_scale(), c2 = ds * 0.693147f;
    WARP_ITEM_LOOP((long long)T * H)
    {
        const int t = (int)(item / H), h = (int)(item % H), off = h * TILE + lane * 4;
        const float4 qv = load_half4(q + (size_t)t * Q + off), dov = load_half4(dout + (size_t)t * Q + off);
        const float l = lse[(size_t)t * H + h], dsc = dscale[(size_t)t * H + h];
        float4 acc = make_float4(0, 0, 0, 0);
        const int s0 = span_start[t], s1 = span_finish[t];
        for (int to = s0; to <= s1; ++to) {
            const float4 kv = load_half4(k + (size_t)to * Q + off), vv = load_half4(v + (size_t)to * Q + off);
            const float dp = warp_sum(dot4(qv, kv)) * ds - slope * (float)(t - to);
            const float w = exp2f(dp - l);
            const float dW = warp_sum(dot4(dov, vv));
            acc = axpy4(w * (dW - dsc) * c2, kv, acc);
        }
        *(float4 *)(dq + (size_t)t * Q + off) = acc;
    }
}

__global__ void attention_dkv_kernel(const __half *__restrict__ q, const __half *__restrict__ k, const __half *__restrict__ v,
                                     const __half *__restrict__ dout, const float *__restrict__ lse, const float *__restrict__ dscale,
                                     const int *__restrict__ span_start, const int *__restrict__ span_finish,
                                     const int *__restrict__ rev_first, const int *__restrict__ rev_last, int T, int H, float slope,
                                     float *__restrict__ dk, float *__restrict__ dv)
{
    grid_dep_wait();
    const int Q = H * TILE;
    const float ds = att_dot_scale(), c2 = ds * 0.693147f;
    WARP_ITEM_LOOP((long long)T * H)
    {
        const int to = (int)(item / H), h = (int)(item % H), off = h * TILE + lane * 4;
        const float4 kv = load_half4(k + (size_t)to * Q + off), vv = load_half4(v + (size_t)to * Q + off);
        float4 ak = make_float4(0, 0, 0, 0), av = make_float4(0, 0, 0, 0);
        const int f0 = rev_first[to], f1 = rev_last[to];
        for (int t = f0; t <= f1; ++t) {
            if (span_start[t] > to || span_finish[t] < to)
                continue;
            const float4 qv = load_half4(q + (size_t)t * Q + off), dov = load_half4(dout + (size_t)t * Q + off);
            const float dp = warp_sum(dot4(qv, kv)) * ds - slope * (float)(t - to);
            const float w = exp2f(dp - lse[(size_t)t * H + h]);
            const float dW = warp_sum(dot4(dov, vv));
            ak = axpy4(w * (dW - dscale[(size_t)t * H + h]) * c2, qv, ak);
            av = axpy4(w, dov, av);
        }
        *(float4 *)(dk + (size_t)to * Q + off) = ak;
        *(float4 *)(dv + (size_t)to * Q + off) = av;
    }
}

int attention_backward_rowwise(const Ctx &c, const __half *q, const __half *k, const __half *v, const __half *dout, const float *lse,
                               const float *dscale, const int *span_start, const int *span_finish, const int *rev_first,
                               const int *rev_last, int T, int H, float slope, float *dq, float *dk, float *dv)
{
    const int grid = grid_for(c, (long long)T * H);
    TS2_LAUNCH((attention_dq_kernel), grid, THREADS, 0, c.stream, q, k, v, dout, lse, dscale, span_start, span_finish, T, H, slope, dq);
    TS2_LAUNCH((attention_dkv_kernel), grid, THREADS, 0, c.stream, q, k, v, dout, lse, dscale, span_start, span_finish, rev_first,
               rev_last, T, H, slope, dk, dv);
    return TS2_OK;
}

int attention_forward(const Ctx &c, const __half *q, const __half *k, const __half *v, const int *span_start, const int *span_finish,
                      int T, int H, float slope, __half *o, float *lse, const AttGate &gate)
{
    return attention_forward_tc(c, q, k, v, span_start, span_finish, T, H, slope, o, lse, &gate);
}

} // namespace ts2
