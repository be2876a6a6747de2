// Gradient apply and weight requantisation: the arithmetic of the reference's MatrixRowSum2Kernel,
// UpdateGlobalRowDisp, AddGradientKernel (src/gpt/matrix/agpu_cuda.cu:32-134) and ConvertMatrixKernel
// (src/gpt/matrix/agpu_cuda.cuh:63-101), restructured from one chain of launches per matrix into a few launches
// over flat buffers that hold every matrix, so that a data-parallel rank can own any contiguous part of them.
// The requantiser's output is also copied transposed for the dX contractions, so no per-step transpose remains.
#include "kernels.cuh"
#include "fast_types.cuh"

namespace ts2 {

static constexpr int WARPS = 8;
static constexpr int THREADS = WARPS * 32;

// ---------------------------------------------------------------------------------
// Flat, sharded form of the optimizer and the requantiser.  All matrices live in flat buffers (weights, momentum,
// gradient) in matrix order, grouped into buckets (embedding, final layer, one per layer).  A rank owns one
// contiguous element range of every bucket (the whole bucket without data parallelism); OptSeg describes the part
// of one matrix that falls into such a range.  Work items are (segment, row) pairs: one warp per row part, so every
// per-row sum has a fixed order and nothing needs atomics.  Per-row results go to vectors indexed by a global row
// number (rows of all matrices in matrix order); rows cut by a range boundary are completed by the data-parallel
// sum of those vectors.  This replaces the per-matrix chains MatrixRowSum2Kernel -> UpdateGlobalRowDisp ->
// AddGradientKernel -> ConvertMatrixKernel of the reference (agpu_cuda.cu:32-134, agpu_cuda.cuh:63-101) by five
// launches per step over everything a rank owns.

// The launches below take a run of segments and the work items [item0, item0 + nitems) they hold.
// binary search: the segment that holds work item `item`
__device__ __forceinline__ int find_seg(const OptSeg *__restrict__ segs, int nseg, int item)
{
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (segs[mid].item0 <= item)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// columns [c0, c1) of row r of the segment's matrix that belong to the range
__device__ __forceinline__ void seg_row_cols(const OptSeg &sg, int r, long long &base, int &c0, int &c1)
{
    const long long row_begin = (long long)r * sg.x;
    c0 = (int)(max(row_begin, sg.a) - row_begin);
    c1 = (int)(min(row_begin + sg.x, sg.b) - row_begin);
    base = sg.flat_off + row_begin;
}

__global__ void opt_row_sum2_kernel(const OptSeg *__restrict__ segs, int nseg, int item0, int nitems, const float *__restrict__ grad,
                                    float *__restrict__ rowsum)
{
    grid_dep_wait();
    const int lane = threadIdx.x & 31;
    for (int item = item0 + blockIdx.x * WARPS + (threadIdx.x >> 5); item < item0 + nitems; item += gridDim.x * WARPS) {
        const OptSeg sg = segs[find_seg(segs, nseg, item)];
        const int r = sg.row0 + (item - sg.item0);
        long long base;
        int c0, c1;
        seg_row_cols(sg, r, base, c0, c1);
        const float4 *src = (const float4 *)(grad + base);
        float s = 0.f;
        for (int i = c0 / 4 + lane; i < c1 / 4; i += 32) {
            const float4 v = src[i];
            s += dot4(v, v);
        }
        s = warp_sum(s);
        if (lane == 0)
            rowsum[sg.grow0 + r] = s;
    }
}

// dispersion EMA -> row scale for every row of a matrix (UpdateGlobalRowDisp).  blockIdx.x = matrix; rows with a dispersion
// of their own are divided over blockIdx.y (one block took 43 us for a 50 k-row embedding, these 5), a matrix with one is
// the first block's.  The weight of the average is advanced by opt_sko_kernel, when no block reads the old one any more.
__global__ void opt_disp_kernel(const OptMat *__restrict__ mats, const float *__restrict__ rowsum, float disp_decay,
                                float *__restrict__ row_scale)
{
    grid_dep_wait();
    __shared__ float red[32];
    __shared__ float bcast;
    const OptMat mt = mats[blockIdx.x];
    const float *sum2 = rowsum + mt.grow0;
    float *rs_out = row_scale + mt.grow0;
    const long long step = mt.y / mt.row_disp_size;
    const float sw = *mt.sum_weight * disp_decay + 1.f;
    const float norm = 1.f / sw;
    if (step == 1) {
        for (long long r = blockIdx.y * blockDim.x + threadIdx.x; r < mt.y; r += gridDim.y * blockDim.x) {
            const float rd = mt.row_disp[r] * disp_decay + sum2[r] / (float)mt.x;
            mt.row_disp[r] = rd;
            const float d = rd * norm;
            rs_out[r] = d > 0.f ? 1.f / sqrtf(d) : 0.f;
        }
    } else if (blockIdx.y == 0) {
        for (int b = 0; b < mt.row_disp_size; ++b) {
            float s = 0.f;
            for (long long k = threadIdx.x; k < step; k += blockDim.x)
                s += sum2[b * step + k];
            s = warp_sum(s);
            if ((threadIdx.x & 31) == 0)
                red[threadIdx.x >> 5] = s;
            __syncthreads();
            if (threadIdx.x == 0) {
                float tot = 0.f;
                for (int i = 0; i < (int)blockDim.x / 32; ++i)
                    tot += red[i];
                const float rd = mt.row_disp[b] * disp_decay + tot / ((float)mt.x * (float)step);
                mt.row_disp[b] = rd;
                const float d = rd * norm;
                bcast = d > 0.f ? 1.f / sqrtf(d) : 0.f;
            }
            __syncthreads();
            const float rs = bcast;
            for (long long k = threadIdx.x; k < step; k += blockDim.x)
                rs_out[b * step + k] = rs;
            __syncthreads();
        }
    }
}

// AddGradientKernel on the rows of the range (UPDATE) and the sum of squares of the (new) weights per row part
template <bool UPDATE>
__global__ void opt_update_kernel(const OptSeg *__restrict__ segs, int nseg, int item0, int nitems, const float *__restrict__ grad,
                                  const float *__restrict__ row_scale, ts2_training_step step, float *__restrict__ avg,
                                  float *__restrict__ w, double *__restrict__ roww2)
{
    grid_dep_wait();
    const int lane = threadIdx.x & 31;
    for (int item = item0 + blockIdx.x * WARPS + (threadIdx.x >> 5); item < item0 + nitems; item += gridDim.x * WARPS) {
        const OptSeg sg = segs[find_seg(segs, nseg, item)];
        const int r = sg.row0 + (item - sg.item0);
        long long base;
        int c0, c1;
        seg_row_cols(sg, r, base, c0, c1);
        float4 *ww = (float4 *)(w + base);
        double s = 0.0;
        if (UPDATE) {
            const float rs = row_scale[sg.grow0 + r];
            const float step_mult = step.rate * sqrtf(sg.sparsity);
            const float shrink = 1.f - step_mult * step.l2reg;
            const float beta1 = step.beta1, w0 = step.weight0, w1 = step.weight1;
            const float4 *g = (const float4 *)(grad + base);
            float4 *a = (float4 *)(avg + base);
            for (int i = c0 / 4 + lane; i < c1 / 4; i += 32) {
                const float4 d = scale4(g[i], rs);
                const float4 oa = a[i], ow = ww[i];
                float4 na, nw;
#define TS2_UPD(f)                                         \
    na.f = oa.f * beta1 + d.f * (1.f - beta1);             \
    nw.f = ow.f * shrink + (na.f * w1 + d.f * w0) * step_mult;
                TS2_UPD(x)
                TS2_UPD(y)
                TS2_UPD(z)
                TS2_UPD(w)
#undef TS2_UPD
                a[i] = na;
                ww[i] = nw;
                s += (double)nw.x * nw.x + (double)nw.y * nw.y + (double)nw.z * nw.z + (double)nw.w * nw.w;
            }
        } else {
            for (int i = c0 / 4 + lane; i < c1 / 4; i += 32) {
                const float4 v = ww[i];
                s += (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w;
            }
        }
        for (int o = 16; o > 0; o >>= 1)
            s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0)
            roww2[sg.grow0 + r] = s;
    }
}

// one block per matrix: sko = sqrt(sum of squares / (x y)), rows summed in a fixed order
// (disp_decay >= 0: a step was applied, the weight of the dispersion average moves on)
__global__ void opt_sko_kernel(const OptMat *__restrict__ mats, const double *__restrict__ roww2, float *__restrict__ skos, float disp_decay,
                               const WrongSoFar wrong)
{
    grid_dep_wait();
    if (wrong.out && blockIdx.x == 0 && threadIdx.x == 0)
        *wrong.out = (wrong.device_status ? *wrong.device_status : 0) | (wrong.static_status ? *wrong.static_status : 0) |
                     wrong.batch_status[0] | wrong.batch_status[4];
    __shared__ double red[32];
    const OptMat mt = mats[blockIdx.x];
    double s = 0.0;
    for (long long r = threadIdx.x; r < mt.y; r += blockDim.x)
        s += roww2[mt.grow0 + r];
    for (int o = 16; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int i = 0; i < (int)blockDim.x / 32; ++i)
            tot += red[i];
        skos[blockIdx.x] = sqrtf((float)tot / (float)(mt.x * mt.y));
        if (disp_decay >= 0.f)
            *mt.sum_weight = *mt.sum_weight * disp_decay + 1.f;
    }
}

// four weights in operand format KIND (OptSeg::qkind), as one word, or two for fp16 (first: the lower pair)
__device__ __forceinline__ uint2 quantize4(float4 v, int kind)
{
    if (kind == 2) // int8: nearest even, saturating (PackFloatToInt8, src/gpt/model_params/sse_utils.h:56-78)
        return make_uint2(sat_i8(v.x) | (sat_i8(v.y) << 8) | (sat_i8(v.z) << 16) | (sat_i8(v.w) << 24), 0u);
    if (kind == 0)
        return make_uint2(encode_e4m3_weight(v.x) | (encode_e4m3_weight(v.y) << 8) | (encode_e4m3_weight(v.z) << 16) | (encode_e4m3_weight(v.w) << 24), 0u);
    const __half h0 = __float2half_rn(v.x), h1 = __float2half_rn(v.y), h2 = __float2half_rn(v.z), h3 = __float2half_rn(v.w);
    return make_uint2((uint32_t)__half_as_ushort(h0) | ((uint32_t)__half_as_ushort(h1) << 16),
                      (uint32_t)__half_as_ushort(h2) | ((uint32_t)__half_as_ushort(h3) << 16));
}
__device__ __forceinline__ float quant_mult(float sko) { return sko == 0.f ? 0.f : 1.f / (sko * (1.f / 32)); }

// ConvertMatrixKernel on the rows of the range: q = enc(w * 32 / sko) into the matrix's row-major quantized copy
__global__ void opt_quant_kernel(const OptSeg *__restrict__ segs, int nseg, int nitems, const float *__restrict__ w,
                                 const float *__restrict__ skos)
{
    grid_dep_wait();
    const int lane = threadIdx.x & 31;
    for (int item = blockIdx.x * WARPS + (threadIdx.x >> 5); item < nitems; item += gridDim.x * WARPS) {
        const OptSeg sg = segs[find_seg(segs, nseg, item)];
        const int r = sg.row0 + (item - sg.item0);
        long long base;
        int c0, c1;
        seg_row_cols(sg, r, base, c0, c1);
        const float mult = quant_mult(skos[sg.mat]);
        const float4 *src = (const float4 *)(w + base);
        uint8_t *dst = sg.qbase + (size_t)r * sg.x * sg.qsize;
        for (int i = c0 / 4 + lane; i < c1 / 4; i += 32) {
            const uint2 q = quantize4(scale4(src[i], mult), sg.qkind);
            if (sg.qkind == 1)
                *(uint2 *)(dst + 8 * (size_t)i) = q;
            else
                *(uint32_t *)(dst + 4 * (size_t)i) = q.x;
        }
    }
}

static int opt_grid(const Ctx &c, int nitems)
{
    return (int)std::max<long long>(1, std::min<long long>(ceil_div(nitems, WARPS), (long long)sm_count(c.device) * 8));
}

int opt_row_sum2(const Ctx &c, const OptSeg *segs, int nseg, int item0, int nitems, const float *grad, float *rowsum)
{
    if (nitems <= 0)
        return TS2_OK;
    TS2_LAUNCH((opt_row_sum2_kernel), opt_grid(c, nitems), THREADS, 0, c.stream, segs, nseg, item0, nitems, grad, rowsum);
    return TS2_OK;
}

int opt_disp(const Ctx &c, const OptMat *mats, int n_mats, const float *rowsum, float disp_decay, float *row_scale)
{
    TS2_LAUNCH((opt_disp_kernel), dim3(n_mats, 8), 1024, 0, c.stream, mats, rowsum, disp_decay, row_scale);
    return TS2_OK;
}

int opt_update(const Ctx &c, const OptSeg *segs, int nseg, int item0, int nitems, const float *grad, const float *row_scale,
               const ts2_training_step *step, float *avg, float *w, double *roww2)
{
    if (nitems <= 0)
        return TS2_OK;
    if (step)
        TS2_LAUNCH((opt_update_kernel<true>), opt_grid(c, nitems), THREADS, 0, c.stream, segs, nseg, item0, nitems, grad, row_scale, *step, avg,
                   w, roww2);
    else
        TS2_LAUNCH((opt_update_kernel<false>), opt_grid(c, nitems), THREADS, 0, c.stream, segs, nseg, item0, nitems, nullptr, nullptr,
                   ts2_training_step(), nullptr, w, roww2);
    return TS2_OK;
}

int opt_sko(const Ctx &c, const OptMat *mats, int n_mats, const double *roww2, float *skos, float disp_decay, const int *batch_status, int *wrong)
{
    WrongSoFar w;
    if (wrong) {
        w.device_status = device_status_word(c.device), w.static_status = static_status_word_if_ready(c.device);
        w.batch_status = batch_status, w.out = wrong;
    }
    TS2_LAUNCH((opt_sko_kernel), n_mats, 1024, 0, c.stream, mats, roww2, skos, disp_decay, w);
    return TS2_OK;
}

int opt_quantize(const Ctx &c, const OptSeg *segs, int nseg, int nitems, const float *w, const float *skos)
{
    if (nitems <= 0)
        return TS2_OK;
    TS2_LAUNCH((opt_quant_kernel), opt_grid(c, nitems), THREADS, 0, c.stream, segs, nseg, nitems, w, skos);
    return TS2_OK;
}

// Copies of quantized blocks into another row-major place and / or their transpose, all of a model's in one launch, from
// the quantized values, or (CopyJob::w) from the weights themselves, which are quantized on the way: one launch and one pass
// less where this rank holds whole matrices (124 M parameters 350 + 155 -> 494 us, 437 M 642 + 350 -> 947).  A tile is 128
// bytes of 128 rows (64 rows of 2-byte values): it comes in as 16-byte vectors, lies in shared
// memory with its 16-byte pieces rotated by the row group (so that both the vector writes and the word reads of eight
// row groups are free of bank conflicts), is transposed in registers by byte permutes and leaves in 16-byte vectors.
// A small model's launch is one tile per CTA, a chain of latencies: the search for the tile's job is one load per 32 jobs.
// Four rows a thread are in flight; eight cost a third of the resident blocks and gain nothing (3272 against 3257 us for eight
// steps of a 4 M parameter model, 67.3 against 67.5 ms for one of 437 M).
// Bound by its bytes (read once, written once or twice): 4 transposes of [16384 x 2048] bytes and their like took 52 us
// each with 32 x 32 byte tiles (1.3 TB/s) and a launch of their own; an expert layer of 32 experts was 97 launches.
__device__ __forceinline__ void transpose4(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t (&c)[4])
{
    const uint32_t l01 = __byte_perm(a0, a1, 0x5140), h01 = __byte_perm(a0, a1, 0x7362);
    const uint32_t l23 = __byte_perm(a2, a3, 0x5140), h23 = __byte_perm(a2, a3, 0x7362);
    c[0] = __byte_perm(l01, l23, 0x5410), c[1] = __byte_perm(l01, l23, 0x7632);
    c[2] = __byte_perm(h01, h23, 0x5410), c[3] = __byte_perm(h01, h23, 0x7632);
}

// four bytes of the operand format as four halves
__device__ __forceinline__ uint2 widen4(uint32_t w, int kind)
{
    if (kind == QCOPY_I8_HALF) {
        const __half2 a = __floats2half2_rn((float)(int8_t)w, (float)(int8_t)(w >> 8)),
                      b = __floats2half2_rn((float)(int8_t)(w >> 16), (float)(int8_t)(w >> 24));
        return make_uint2(*(const uint32_t *)&a, *(const uint32_t *)&b);
    }
    const __half2_raw a = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w & 0xffff), __NV_E4M3),
                      b = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w >> 16), __NV_E4M3);
    return make_uint2((uint32_t)a.x | (uint32_t)a.y << 16, (uint32_t)b.x | (uint32_t)b.y << 16);
}

// The scale vectors of every layer from its matrices' scales (skos, in matrix order): forward column scales a (x sko_k for
// the K block of an attention layer), dW row scales 1 / sko for the matrices that are followed by a normalisation (Q, K,
// V; Expand), 1 elsewhere.  An expert layer has no K block and one row vector, for Expand.
constexpr int SCALE_BLOCKS = 8; // per layer
__device__ __forceinline__ void layer_scales(const ScaleJob &jb, float a, int block)
{
    const bool att = jb.kind == SCALES_ATT;
    for (int i = block * blockDim.x + threadIdx.x; i < jb.ncat * jb.W; i += SCALE_BLOCKS * blockDim.x) {
        const int j = i / jb.W;
        jb.fwd_col[i] = (att && j == 1) ? a * jb.skos[1] : a;
        if (jb.kind == SCALES_MOE) {
            if (j == 0)
                jb.bwd_row[i] = 1.f / jb.skos[0];
            continue;
        }
        jb.bwd_row[i] = (att ? j < 3 : j == 0) ? 1.f / jb.skos[j] : 1.f;
    }
}

// copies, and in the blocks from `blocks` on the scale vectors
__global__ void __launch_bounds__(256) qcopy_kernel(const CopyJob *__restrict__ jobs, int n_jobs, int tiles, int blocks,
                                                    const ScaleJob *__restrict__ scales, float a)
{
    grid_dep_wait();
    __shared__ uint4 tile_s[128 * 8];
    const int tid = threadIdx.x;
    if ((int)blockIdx.x >= blocks) {
        const int i = (int)blockIdx.x - blocks;
        layer_scales(scales[i / SCALE_BLOCKS], a, i % SCALE_BLOCKS);
        return;
    }
    for (int tile = blockIdx.x; tile < tiles; tile += blocks) {
        // the last job that starts at or before the tile: a warp counts them, 32 a load
        int lo = -1;
#pragma unroll 4
        for (int j = 0; j < n_jobs; j += 32)
            lo += __popc(__ballot_sync(0xffffffffu, j + (tid & 31) < n_jobs && jobs[j + (tid & 31)].tile0 <= tile));
        const CopyJob jb = jobs[lo];
        const int two = jb.kind == QCOPY_2BYTE, rows = two ? 64 : 128, shift = two ? 3 : 4;
        const int t = tile - jb.tile0, tx = t % jb.tiles_x, y0 = (t / jb.tiles_x) * rows;
        const long long xb = (long long)tx * 128; // byte offset of the tile in a source row
        if (jb.w) {
            // straight from the weights: a warp (two-byte values: half a warp) takes the 128 (64) columns of a row, four a lane
            const float mult = quant_mult(*jb.sko);
            const int per = two ? 16 : 32, sub = tid % per, step = 256 / per, es = two ? 2 : 1;
            constexpr int AHEAD = 4;
            for (int r0 = tid / per; r0 < rows; r0 += AHEAD * step) {
                float4 f[AHEAD];
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {
                    const int r = r0 + u * step;
                    f[u] = r < rows && y0 + r < jb.y ? *(const float4 *)(jb.w + (long long)(y0 + r) * jb.x + xb / es + sub * 4) : make_float4(0, 0, 0, 0);
                }
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {
                    const int r = r0 + u * step;
                    if (r >= rows)
                        break;
                    const uint2 q = quantize4(scale4(f[u], mult), jb.qkind);
                    uint8_t *const s = (uint8_t *)tile_s + (r * 8 + ((two ? sub >> 1 : sub >> 2) ^ ((r >> shift) & 7))) * 16;
                    const bool in = y0 + r < jb.y;
                    if (two) {
                        *(uint2 *)(s + (sub & 1) * 8) = q;
                        if (in)
                            *(uint2 *)(jb.q + (y0 + r) * jb.ld_src + xb + sub * 8) = q;
                        if (in && jb.dst)
                            *(uint2 *)(jb.dst + (y0 + r) * jb.ld + xb + sub * 8) = q;
                    } else {
                        *(uint32_t *)(s + (sub & 3) * 4) = q.x;
                        if (in)
                            *(uint32_t *)(jb.q + (y0 + r) * jb.ld_src + xb + sub * 4) = q.x;
                        if (in && jb.dst)
                            *(uint32_t *)(jb.dst + (y0 + r) * jb.ld + xb + sub * 4) = q.x;
                    }
                }
            }
        } else {
            for (int v = tid; v < rows * 8; v += 256) {
                const int r = v >> 3, c = v & 7;
                uint4 q = make_uint4(0, 0, 0, 0);
                if (y0 + r < jb.y) {
                    q = *(const uint4 *)(jb.src + (y0 + r) * jb.ld_src + xb + c * 16);
                    if (jb.dst)
                        *(uint4 *)(jb.dst + (y0 + r) * jb.ld + xb + c * 16) = q;
                }
                tile_s[r * 8 + (c ^ ((r >> shift) & 7))] = q;
            }
        }
        if (jb.dstT) { // the same for the whole block
            __syncthreads();
            const uint32_t *words = (const uint32_t *)tile_s;
            const int rg = tid & 7, cg = tid >> 3, wc = cg ^ (rg << 2);
            if (two) {
                const int row0 = y0 + rg * 8;
                uint32_t w[8], c0[4], c1[4];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    w[i] = words[(rg * 8 + i) * 32 + wc];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    c0[i] = __byte_perm(w[2 * i], w[2 * i + 1], 0x5410);
                    c1[i] = __byte_perm(w[2 * i], w[2 * i + 1], 0x7632);
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const uint32_t *c = j ? c1 : c0;
                    uint8_t *d = jb.dstT + ((long long)tx * 64 + cg * 2 + j) * jb.ldT + (long long)row0 * 2;
                    if (row0 + 8 <= jb.y)
                        *(uint4 *)d = make_uint4(c[0], c[1], c[2], c[3]);
                    else
                        for (int i = 0; row0 + i < jb.y; ++i)
                            ((uint16_t *)d)[i] = (uint16_t)(c[i >> 1] >> (16 * (i & 1)));
                }
            } else {
                const int row0 = y0 + rg * 16;
                uint32_t out[4][4]; // [column][four rows]
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    uint32_t w[4], c[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        w[i] = words[(rg * 16 + 4 * b + i) * 32 + wc];
                    transpose4(w[0], w[1], w[2], w[3], c);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        out[j][b] = c[j];
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const long long col = xb + cg * 4 + j;
                    if (jb.kind == QCOPY_1BYTE) {
                        uint8_t *d = jb.dstT + col * jb.ldT + row0;
                        if (row0 + 16 <= jb.y)
                            *(uint4 *)d = make_uint4(out[j][0], out[j][1], out[j][2], out[j][3]);
                        else
                            for (int i = 0; row0 + i < jb.y; ++i)
                                d[i] = (uint8_t)(out[j][i >> 2] >> (8 * (i & 3)));
                    } else {
                        uint8_t *d = jb.dstT + col * jb.ldT + (long long)row0 * 2;
                        uint2 h[4];
#pragma unroll
                        for (int b = 0; b < 4; ++b)
                            h[b] = widen4(out[j][b], jb.kind);
                        if (row0 + 16 <= jb.y) {
                            *(uint4 *)d = make_uint4(h[0].x, h[0].y, h[1].x, h[1].y);
                            *((uint4 *)d + 1) = make_uint4(h[2].x, h[2].y, h[3].x, h[3].y);
                        } else {
                            for (int i = 0; row0 + i < jb.y; ++i) {
                                const uint32_t w = (i & 2) ? h[i >> 2].y : h[i >> 2].x;
                                ((uint16_t *)d)[i] = (uint16_t)(w >> (16 * (i & 1)));
                            }
                        }
                    }
                }
            }
        }
        __syncthreads();
    }
}

int qcopy_tiles(CopyJob &job)
{
    const int es = job.kind == QCOPY_2BYTE ? 2 : 1;
    job.tiles_x = (int)((int64_t)job.x * es / 128);
    return job.tiles_x * (int)ceil_div(job.y, es == 2 ? 64 : 128);
}

int qcopy(const Ctx &c, const CopyJob *jobs, int n_jobs, int tiles, const ScaleJob *scales, int n_scales, float a)
{
    const int blocks = std::min(tiles, sm_count(c.device) * 8);
    if (blocks + n_scales > 0)
        TS2_LAUNCH((qcopy_kernel), blocks + n_scales * SCALE_BLOCKS, 256, 0, c.stream, jobs, n_jobs, tiles, blocks, scales, a);
    return TS2_OK;
}

} // namespace ts2
