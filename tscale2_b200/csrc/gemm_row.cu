// Contractions of few tiles: one 128 x 128 tile, or a share of its K range, per CTA, and what follows in the same launch.
//
// The backward pass of a layer ends with a product of few tiles and a long K (the gradient of the layer's input), the backward
// of the normalisation on it and, from the same operand, the layer's weight gradient.  In a step of a small model those were
// four launches of a chain (contraction, sum of its K splits, normalisation, weight gradient), each a few microseconds of
// latency.  Here
//  * a K range is shared by the CTAs of a cluster (up to 8): each leaves its fp32 partial tile in its own shared memory and
//    sums one part of the rows over all of them through distributed shared memory, in rank order (no workspace, no second
//    launch, the same bits every time);
//  * the product lies in shared memory row by row, a warp takes a whole 128-column row, four columns a lane, as the
//    normalisation's own kernel does with rows in memory, with the same arithmetic (row_math.cuh);
//  * the weight gradient, independent of both, takes further CTAs of the launch.
// Two blocks of dim 256, 8 steps of 4 x 128 tokens and an export, fp16: 3.56 -> 3.24 ms; 8 batches of 3 x 100 tokens, two steps and an
// export, e4m3: 3.22 -> 2.86 ms.
// The other row-wise steps of a layer (residual + normalisation, split of Q | K | V, backward of gate and activation) ran here
// as well and gained nothing: their products have a short K and so few CTAs that a launch over all SMs is as fast.  A launch with
// clusters takes about 2 us more than one without.
// Warp 0 copies (TMA, 3 stages of 32 KB), warp 1 issues the MMAs, then all 8 warps work on rows; two CTAs fit an SM, so that
// the next launch's set-up finds room (16 warps and one CTA per SM were 5 % slower over a step).  Every wait is bounded, as in
// gemm.cu; a CTA whose wait ran out writes nothing but still meets its cluster.
#include "gemm_row.cuh"
#include "gemm_params.cuh"
#include "row_math.cuh"

namespace ts2 {

namespace {

constexpr int R_BN = 128, R_STAGES = 3, R_STAGE_BYTES = 2 * BM * STAGE_ROW_BYTES, R_THREADS = 256, R_WARPS = R_THREADS / 32;
constexpr int R_PITCH = R_BN + 4; // floats per row of the product in shared memory: 16-byte accesses without bank conflicts
constexpr int R_BAR_OFF = R_STAGES * R_STAGE_BYTES;
constexpr int R_SMEM = R_BAR_OFF + 256 + 1024; // + alignment slack
static_assert(BM * R_PITCH * 4 <= R_BAR_OFF, "the product takes the place of the ring");
constexpr int R_MAX_SPLITS = 8; // portable cluster size
constexpr int R_ROWS = 4;       // rows a warp takes at a time

struct RowProblem {
    int M, N, n_tiles, tiles, splits, k_blocks, kb_per_split;
    uint32_t idesc;
    float alpha;
    const float *dyn_scale, *dyn_scale2, *row_scale;
    // second problem: C = (c_in or nothing) + product
    const float *c_in;
    float *C;
    long long ldc;
};
struct RowParams {
    RowProblem pr[2];
    RowOp op; // of pr[0]
    int first2; // CTAs of the first problem, a multiple of the cluster size
    int32_t *status;
};

template <int MMA>
__device__ __forceinline__ void umma_row(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    if constexpr (MMA == 0)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
                     "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                     : "memory");
    else if constexpr (MMA == 1)
        umma_f16(tmem_d, adesc, bdesc, idesc, accumulate);
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
                     "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                     : "memory");
}

__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 16 bytes of shared memory of CTA `rank` of the cluster, at this CTA's address `addr`
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr, uint32_t rank)
{
    float4 v;
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr), "r"(rank)
                 : "memory");
    return v;
}

// Main loop of one unit: the whole warps 0 and 1 come here.  Returns when this thread's part is issued; `done` completes when
// every MMA has.
template <int MMA, bool MN>
__device__ __forceinline__ void row_main_loop(const CUtensorMap *tmA, const CUtensorMap *tmB, const RowProblem &p, int m0, int n0, int kb0, int kb1,
                                              uint32_t ring, uint32_t full0, uint32_t empty0, uint32_t done, uint32_t tmem, volatile int *abort_flag)
{
    constexpr int ES = MMA == 1 ? 2 : 1;
    constexpr int ROW_ELEMS = STAGE_ROW_BYTES / ES, UMMA_K = 32 / ES, BK = ROW_ELEMS; // K elements per stage, in both layouts
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) != 0)
        return;
    if (warp == 0) {
        int issued = 0;
        bool ok = true;
        for (int kb = kb0; kb < kb1; ++kb, ++issued) {
            const int st = issued % R_STAGES;
            if (!(ok = mbar_wait(empty0 + 8 * st, ((issued / R_STAGES) & 1) ^ 1, abort_flag)))
                break;
            const uint32_t fb = full0 + 8 * st, sa = ring + st * R_STAGE_BYTES, sb = sa + BM * STAGE_ROW_BYTES;
            mbar_arrive_expect_tx(fb, R_STAGE_BYTES);
            if constexpr (!MN) {
                tma_load_2d(sa, tmA, fb, kb * BK, m0);
                tma_load_2d(sb, tmB, fb, kb * BK, n0);
            } else { // one box per 128-byte atom along M / N
#pragma unroll
                for (int j = 0; j < BM / ROW_ELEMS; ++j)
                    tma_load_2d(sa + j * BK * STAGE_ROW_BYTES, tmA, fb, m0 + j * ROW_ELEMS, kb * BK);
#pragma unroll
                for (int j = 0; j < R_BN / ROW_ELEMS; ++j)
                    tma_load_2d(sb + j * BK * STAGE_ROW_BYTES, tmB, fb, n0 + j * ROW_ELEMS, kb * BK);
            }
        }
        if (!ok) { // copies in flight must land before anything else happens to the ring (bounded)
            const long long t0 = clock64();
            for (int i = max(0, issued - R_STAGES); i < issued; ++i)
                while (!mbar_try_wait(full0 + 8 * (i % R_STAGES), (i / R_STAGES) & 1) && clock64() - t0 < 200000000ll) {
                }
        }
    } else {
        for (int kb = kb0, i = 0; kb < kb1; ++kb, ++i) {
            const int st = i % R_STAGES;
            if (!mbar_wait(full0 + 8 * st, (i / R_STAGES) & 1, abort_flag))
                break;
            tc_fence_after();
            const uint32_t sa = ring + st * R_STAGE_BYTES, sb = sa + BM * STAGE_ROW_BYTES;
            const uint32_t lbo = MN ? BK * STAGE_ROW_BYTES : 16, step = MN ? (UMMA_K * STAGE_ROW_BYTES) >> 4 : (UMMA_K * ES) >> 4;
            const uint64_t ad = umma_smem_desc(sa, lbo, 1024), bd = umma_smem_desc(sb, lbo, 1024);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                umma_row<MMA>(tmem, ad + (uint64_t)(k * step), bd + (uint64_t)(k * step), p.idesc, i > 0 || k > 0 ? 1u : 0u);
            tc_commit(empty0 + 8 * st);
        }
        tc_commit(done); // also on the abort path: completes when the MMAs issued so far have
    }
}

// rows [r0, r1) of the tile, this warp's share of them R_ROWS at a time: body(first row, how many)
template <class F>
__device__ __forceinline__ void for_rows(int r0, int r1, F body)
{
    for (int r = r0 + (int)(threadIdx.x >> 5) * R_ROWS; r < r1; r += R_WARPS * R_ROWS)
        body(r, min(R_ROWS, r1 - r));
}

// MMA1, MMA2: operand kinds (0 e4m3, 1 fp16, 2 int8) of the two problems
template <int MMA1, int MMA2>
__global__ void __launch_bounds__(R_THREADS, 2)
    gemm_row_kernel(const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ CUtensorMap tmA2,
                    const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ RowParams p)
{
    extern __shared__ uint8_t row_smem[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)row_smem + 1023) & ~(uintptr_t)1023); // the same offset in every CTA of a cluster
    uint64_t *bars = (uint64_t *)(smem + R_BAR_OFF);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + R_STAGES), done = smem_u32(bars + 2 * R_STAGES);
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * R_STAGES + 1);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    float *const tile_s = (float *)smem;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool second = (int)blockIdx.x >= p.first2;
    const RowProblem &pr = p.pr[second ? 1 : 0];
    const int unit = (int)blockIdx.x - (second ? p.first2 : 0), splits = pr.splits, tile = unit / splits, split = unit - tile * splits;
    if (tile >= pr.tiles)
        return; // filler up to a whole cluster (of a problem without splits: its CTAs meet no cluster barrier)
    const int mt = tile / pr.n_tiles, nt = tile - mt * pr.n_tiles, m0 = mt * BM, n0 = nt * R_BN;
    const int kb0 = split * pr.kb_per_split, kb1 = min(pr.k_blocks, kb0 + pr.kb_per_split);

    if (threadIdx.x == 0) {
        for (int s = 0; s < R_STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(done, 1);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(second ? &tmA2 : &tmA1);
        prefetch_tmap(second ? &tmB2 : &tmB1);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), R_BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_wait();
    const uint32_t tmem = *tmem_slot;
    if (warp < 2) {
        if (!second)
            row_main_loop<MMA1, false>(&tmA1, &tmB1, pr, m0, n0, kb0, kb1, smem_u32(smem), full0, empty0, done, tmem, abort_flag);
        else
            row_main_loop<MMA2, true>(&tmA2, &tmB2, pr, m0, n0, kb0, kb1, smem_u32(smem), full0, empty0, done, tmem, abort_flag);
        __syncwarp();
    }
    bool ok = mbar_wait(done, 0, abort_flag);
    ok = __syncthreads_and(ok && !*abort_flag);
    tc_fence_after();
    const bool integer = second ? MMA2 == 2 : MMA1 == 2;
    if (ok) { // accumulator -> rows in shared memory, over the ring (every copy and MMA is complete)
        const int quarter = warp & 3, half = warp >> 2;
        float4 *dst = (float4 *)(tile_s + (quarter * 32 + lane) * R_PITCH + half * 64);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            uint32_t r[32];
            tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + half * 64 + j * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float4 v = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
                if (integer)
                    v = make_float4((float)(int)r[4 * i], (float)(int)r[4 * i + 1], (float)(int)r[4 * i + 2], (float)(int)r[4 * i + 3]);
                dst[8 * j + i] = v;
            }
        }
    }
    tc_fence_before();
    if (splits > 1) // every CTA of the cluster passes here and at the end, whatever became of its waits
        cluster_sync_all();
    else
        __syncthreads();
    if (warp == 1)
        tmem_dealloc(tmem, R_BN);

    if (ok) {
        // this CTA's share of the rows, those past M left out
        const int r0 = split * BM / splits, r1 = (split + 1) * BM / splits, rm = min(r1, pr.M - m0);
        const uint32_t tile_addr = smem_u32(tile_s);
        float alpha = pr.alpha;
        if (pr.dyn_scale)
            alpha *= __ldg(pr.dyn_scale);
        if (pr.dyn_scale2)
            alpha *= __ldg(pr.dyn_scale2);
        auto times = [](float4 v, float f) { // rounded: no part of an fma with what it is added to
            return make_float4(__fmul_rn(v.x, f), __fmul_rn(v.y, f), __fmul_rn(v.z, f), __fmul_rn(v.w, f));
        };
        auto product = [&](int r, int c) { // columns c .. c + 3 of row r, summed over the cluster in rank order, with the scales applied
            float4 s = make_float4(0, 0, 0, 0);
            if (splits == 1)
                s = *(const float4 *)(tile_s + r * R_PITCH + c);
            else
                for (int sp = 0; sp < splits; ++sp) {
                    const float4 v = ld_cluster4(tile_addr + (uint32_t)(r * R_PITCH + c) * 4, sp);
                    s = make_float4(s.x + v.x, s.y + v.y, s.z + v.z, s.w + v.w);
                }
            return times(s, alpha * (pr.row_scale ? __ldg(pr.row_scale + m0 + r) : 1.f));
        };
        const int c = lane * 4, col = n0 + c;
        if (second) {
            if (col < pr.N)
                for_rows(r0, rm, [&](int r, int n) {
                    float4 in[R_ROWS];
                    if (pr.c_in)
#pragma unroll
                        for (int i = 0; i < R_ROWS; ++i)
                            if (i < n)
                                in[i] = *(const float4 *)(pr.c_in + (m0 + r + i) * pr.ldc + col);
#pragma unroll
                    for (int i = 0; i < R_ROWS; ++i) {
                        if (i >= n)
                            break;
                        float4 v = product(r + i, c);
                        if (pr.c_in)
                            v = make_float4(in[i].x + v.x, in[i].y + v.y, in[i].z + v.z, in[i].w + v.w);
                        *(float4 *)(pr.C + (m0 + r + i) * pr.ldc + col) = v;
                    }
                });
        } else {
            const RowOp &op = p.op;
            const float a = op.dyn ? __ldg(op.dyn) : 1.f;
            float mx = 0.f;
            for_rows(r0, rm, [&](int r, int n) {
                float4 xv[R_ROWS], gv[R_ROWS];
#pragma unroll
                for (int i = 0; i < R_ROWS; ++i) {
                    const long long at = (long long)(m0 + r + i) * pr.N + col;
                    xv[i] = i < n ? *(const float4 *)(op.x + at) : make_float4(0, 0, 0, 0);
                    gv[i] = i < n && op.add ? *(const float4 *)(op.g + at) : make_float4(0, 0, 0, 0);
                }
#pragma unroll
                for (int i = 0; i < R_ROWS; ++i) {
                    if (i >= n)
                        break;
                    const float4 x = xv[i], dn = times(product(r + i, c), a);
                    // the sum's order spelled out: the compiler's own choice follows from what stands around it
                    const float xd = fmaf(x.w, dn.w, fmaf(x.z, dn.z, fmaf(x.y, dn.y, __fmul_rn(x.x, dn.x))));
                    const float4 d = tilenorm_backward4(x, dn, xd);
                    const float4 g = make_float4(gv[i].x + d.x, gv[i].y + d.y, gv[i].z + d.z, gv[i].w + d.w);
                    *(float4 *)(op.g + (long long)(m0 + r + i) * pr.N + col) = g;
                    mx = absmax4(mx, g);
                }
            });
            mx = warp_max(mx);
            if (lane == 0 && r0 < rm)
                absmax_report(mx, op.absmax, op.health, op.step_no);
        }
    }
    __syncwarp();
    if (splits > 1)
        cluster_sync_all(); // the other CTAs have read this one's rows
    if (threadIdx.x == 0 && *abort_flag)
        atomicOr(p.status, TS2_STATUS_WAIT_TIMEOUT);
}

RowProblem row_problem(const GemmArgs &a, int splits)
{
    RowProblem p;
    const int es = a.kind == KIND_F16 ? 2 : 1;
    p.M = (int)a.M;
    p.N = (int)a.N;
    p.n_tiles = (int)ceil_div(a.N, R_BN);
    p.tiles = (int)ceil_div(a.M, BM) * p.n_tiles;
    p.k_blocks = (int)ceil_div(a.K, STAGE_ROW_BYTES / es);
    p.kb_per_split = (int)ceil_div(p.k_blocks, splits);
    p.splits = splits;
    p.idesc = gemm_instr_desc(a.kind, a.mn_major, BM, R_BN);
    p.alpha = a.epi.alpha;
    p.dyn_scale = a.epi.dyn_scale;
    p.dyn_scale2 = a.epi.dyn_scale2;
    p.row_scale = a.epi.row_scale;
    p.c_in = a.epi.out_kind != TS2_OUT_F32_ADD ? nullptr : a.epi.c_in ? a.epi.c_in : (const float *)a.C;
    p.C = (float *)a.C;
    p.ldc = a.ldc;
    return p;
}

int row_maps(const GemmArgs &a, CUtensorMap *tA, CUtensorMap *tB)
{
    const int es = a.kind == KIND_F16 ? 2 : 1, bk = STAGE_ROW_BYTES / es;
    int rc;
    if (a.mn_major) {
        if ((rc = make_tensor_map(tA, a.A, es, a.M, a.K, a.lda, bk)) != TS2_OK)
            return rc;
        return make_tensor_map(tB, a.B, es, a.N, a.K, a.ldb, bk);
    }
    if ((rc = make_tensor_map(tA, a.A, es, a.K, a.M, a.lda, BM)) != TS2_OK)
        return rc;
    return make_tensor_map(tB, a.B, es, a.K, a.N, a.ldb, R_BN);
}

template <int MMA1, int MMA2>
int launch_row(int device, cudaStream_t stream, int grid, int cluster, const CUtensorMap (&tm)[4], const RowParams &p)
{
    auto kern = gemm_row_kernel<MMA1, MMA2>;
    static bool configured[16] = {};
    if (!configured[device & 15]) {
        TS2_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, R_SMEM));
        configured[device & 15] = true;
    }
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster, attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(R_THREADS);
    cfg.dynamicSmemBytes = R_SMEM;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tm[0], tm[1], tm[2], tm[3], p);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(TS2_ERR_CUDA, "kernel launch failed: %s (%s:%d)", cudaGetErrorString(e), __FILE__, __LINE__);
    }
    return TS2_OK;
}

} // namespace

// K split and estimated time (us) of one contraction in this kernel (see make_plan in gemm.cu for the others'), from measured
// launches one behind the other: 512 x 256 x 2048 e4m3 in 8 splits 7.7, 512 x 256 x 2048 fp16 8.4, 77 x 768 x 6144 8.6; without
// splits 300 x 2048 x 256 5.8, two CTAs an SM 6144 x 768 from 1000 tokens 10.2, from 4000 20.2; more CTAs than the SMs hold
// at once, and clusters on more than every SM once, are slower than any other way (96 tiles in 8 splits 30)
double gemm_row_plan(int device, int kind, int64_t M, int64_t N, int64_t K, int *splits)
{
    const int es = kind == KIND_F16 ? 2 : 1, sms = sm_count(device), k_blocks = (int)ceil_div(K, STAGE_ROW_BYTES / es);
    const long long tiles = ceil_div(M, BM) * ceil_div(N, R_BN);
    double best = 1e30;
    *splits = 1;
    for (int s = 1; s <= R_MAX_SPLITS; s *= 2) {
        const int per = (int)ceil_div(k_blocks, s);
        const long long ctas = tiles * s;
        if ((int)ceil_div(k_blocks, per) != s || (s > 1 && (per < 2 || ctas > sms)) || ctas > 2 * sms)
            continue;
        const double t = s > 1 ? 6.8 + 0.3 * per : ctas <= sms ? 5.5 + 0.28 * per : 6.9 + 0.42 * per;
        if (t < best) {
            best = t;
            *splits = s;
        }
    }
    return best;
}

bool gemm_row_takes_pair(int device, const GemmArgs &a, const GemmArgs &b)
{
    int s1, s2;
    gemm_row_plan(device, a.kind, a.M, a.N, a.K, &s1);
    gemm_row_plan(device, b.kind, b.M, b.N, b.K, &s2);
    const long long t1 = ceil_div(a.M, BM) * ceil_div(a.N, R_BN), t2 = ceil_div(b.M, BM) * ceil_div(b.N, R_BN);
    return t1 * s1 + t2 <= 2 * sm_count(device);
}

int gemm_row(const RowGemm &r)
{
    const GemmArgs &a = r.a;
    const GemmArgs *const list[2] = {&a, r.second};
    double flops = 0, bytes = 0;
    for (const GemmArgs *g : list) {
        if (!g)
            continue;
        const bool add = g->epi.out_kind == TS2_OUT_F32_ADD;
        if (g->M <= 0 || g->N <= 0 || g->K <= 0 || g->mn_major != (g == r.second) || g->group_mode || g->epi.pair_stride || g->epi.bwd_wg ||
            g->kind == KIND_BF16 || g->epi.col_scale || (g->epi.out_kind != TS2_OUT_F32 && !add) ||
            (g == &a ? r.op.form != ROW_NORM_BWD || add || g->N % 128 : g->N % 32 || ((uintptr_t)g->C & 15) || ((g->ldc * 4) & 15)))
            return fail(TS2_ERR_INVALID_ARG, "gemm_row: bad arguments");
        flops += 2.0 * g->M * g->N * g->K;
        bytes += ((double)g->M + g->N) * g->K * (g->kind == KIND_F16 ? 2 : 1) + (double)g->M * g->N * (add ? 8 : 4);
    }
    TS2_CUDA(cudaSetDevice(a.device));
    RowParams p;
    CUtensorMap tm[4];
    int rc, s[2] = {1, 1};
    const long long slots = 2 * sm_count(a.device);
    gemm_row_plan(a.device, a.kind, a.M, a.N, a.K, &s[0]);
    if (r.second) {
        // one cluster size for the launch: the first contraction, which the next kernel waits for, has its choice as far as
        // both stay within one wave; the second takes the same or none
        const long long t1 = ceil_div(a.M, BM) * ceil_div(a.N, R_BN), t2 = ceil_div(r.second->M, BM) * ceil_div(r.second->N, R_BN);
        const int k1 = row_problem(a, 1).k_blocks, k2 = row_problem(*r.second, 1).k_blocks;
        while (s[0] > 1 && (t1 * s[0] + t2 > slots || (int)ceil_div(k1, ceil_div(k1, s[0])) != s[0]))
            s[0] /= 2;
        s[1] = s[0] > 1 && (t1 + t2) * s[0] <= slots / 2 && (int)ceil_div(k2, ceil_div(k2, s[0])) == s[0] && k2 >= 4 * s[0] ? s[0] : 1;
    }
    const int cluster = s[0]; // s[1] is the same or 1
    int grid = 0;
    for (int i = 0; i < 2; ++i) {
        const GemmArgs &g = list[i] ? *list[i] : a;
        p.pr[i] = row_problem(g, s[i]);
        if ((rc = row_maps(g, &tm[2 * i], &tm[2 * i + 1])) != TS2_OK)
            return rc;
        if (list[i])
            grid += (int)ceil_div((int64_t)p.pr[i].tiles * s[i], cluster) * cluster;
        if (i == 0)
            p.first2 = grid;
    }
    p.op = r.op;
    p.status = device_status_word(a.device);
    if (!p.status)
        return fail(TS2_ERR_CUDA, "gemm: no device status word");
    const GemmTimed timed = gemm_timed_begin(a.stream);
    const int k1 = a.kind, k2 = r.second ? r.second->kind : k1 == KIND_I8 ? KIND_F16 : k1; // of none: any that is built
    if (k1 == KIND_E4M3 && k2 == KIND_E4M3)
        rc = launch_row<0, 0>(a.device, a.stream, grid, cluster, tm, p);
    else if (k1 == KIND_F16 && k2 == KIND_F16)
        rc = launch_row<1, 1>(a.device, a.stream, grid, cluster, tm, p);
    else if (k1 == KIND_I8 && k2 == KIND_F16)
        rc = launch_row<2, 1>(a.device, a.stream, grid, cluster, tm, p);
    else
        return fail(TS2_ERR_UNSUPPORTED, "gemm_row: unsupported pair of operand formats");
    gemm_timed_end(timed, a.stream, flops, bytes, a.tag);
    return rc;
}

} // namespace ts2
