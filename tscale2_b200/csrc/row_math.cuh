// Arithmetic of the row-wise kernels, on values in registers: the kernels that run it on tensors in memory
// (kernels_elem.cu, kernels_att.cu) and the contractions whose epilogue runs it on their own product (gemm_row.cu, gemm_pair.cu)
// share it.  A warp holds 128 consecutive columns of a row, four to a lane; in the functions on
// eight values half a warp does.
#pragma once
#include "fast_types.cuh"

namespace ts2 {

// ---- tile normalisation ---------------------------------------------------------
// gradient of the raw values x from the gradient d of the normalised ones (whole warp); xd: the lane's part of x . d
__device__ __forceinline__ float4 tilenorm_backward4(float4 x, float4 d, float xd)
{
    const float sum2 = warp_sum(dot4(x, x));
    const float dp = warp_sum(xd);
    if (sum2 == 0.f)
        return make_float4(0, 0, 0, 0);
    const float sigma = dp / sum2, scale = sqrtf(128.f / sum2);
    return make_float4(scale * (d.x - x.x * sigma), scale * (d.y - x.y * sigma), scale * (d.z - x.z * sigma), scale * (d.w - x.w * sigma));
}
__device__ __forceinline__ float4 tilenorm_backward4(float4 x, float4 d) { return tilenorm_backward4(x, d, dot4(x, d)); }
// running |maximum| of a gradient; fmaxf drops a NaN operand: a NaN turns it into inf instead
__device__ __forceinline__ float absmax4(float m, float4 r)
{
    m = fmaxf(m, fmaxf(fmaxf(fabsf(r.x), fabsf(r.y)), fmaxf(fabsf(r.z), fabsf(r.w))));
    return r.x == r.x && r.y == r.y && r.z == r.z && r.w == r.w ? m : INFINITY;
}
// a block's maximum into the running one; NaN and inf never become the scale reference, health keeps the first step they came up in
__device__ __forceinline__ void absmax_report(float m, unsigned *absmax, unsigned *health, unsigned step_no)
{
    if (m == m && m < 3.0e38f)
        atomicMax(absmax, __float_as_uint(m));
    else if (health)
        atomicCAS(health, 0u, step_no);
}

// ---- eight values a lane, half a warp a row: heads of the attention ----------------
__device__ __forceinline__ void half8_to_float(uint4 raw, float (&f)[8])
{
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 p = __half22float2(h2_from_bits(w[i]));
        f[2 * i] = p.x;
        f[2 * i + 1] = p.y;
    }
}
__device__ __forceinline__ uint4 float_to_half8(const float (&f)[8])
{
    return make_uint4(bits_from_h2(sat_half2(f[0], f[1])), bits_from_h2(sat_half2(f[2], f[3])), bits_from_h2(sat_half2(f[4], f[5])),
                      bits_from_h2(sat_half2(f[6], f[7])));
}
__device__ __forceinline__ float half_warp_sum(float v)
{
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float dot8(const float (&a)[8], const float (&b)[8])
{
    return (a[0] * b[0] + a[1] * b[1] + a[2] * b[2] + a[3] * b[3]) + (a[4] * b[4] + a[5] * b[5] + a[6] * b[6] + a[7] * b[7]);
}
// pairs (0,1) and (2,3) of four elements; cs = (cos0, sin0, cos1, sin1)
__device__ __forceinline__ float4 rope_apply(float4 v, float4 cs, float dir)
{
    const float s0 = cs.y * dir, s1 = cs.w * dir;
    return make_float4(v.x * cs.x - v.y * s0, v.x * s0 + v.y * cs.x, v.z * cs.z - v.w * s1, v.z * s1 + v.w * cs.z);
}
// rotates the lane's four pairs; c0, c1: (cos, sin) of two pairs each
__device__ __forceinline__ void rope8(float (&v)[8], float4 c0, float4 c1, float dir)
{
    const float4 a = rope_apply(make_float4(v[0], v[1], v[2], v[3]), c0, dir), b = rope_apply(make_float4(v[4], v[5], v[6], v[7]), c1, dir);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
__device__ __forceinline__ void scale8(float (&v)[8], float s)
{
#pragma unroll
    for (int i = 0; i < 8; ++i)
        v[i] *= s;
}

} // namespace ts2
