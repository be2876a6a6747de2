// tcgen05 attention backward, dQ = dS . K from the score gradients that the dK / dV kernel left (head width 128, sm_100a).
// References: GradQ, src/gpt/compute/layer_att_reference.h:41-212; Fp16AttGradQ, gpu_att_fp16.cu.
//
// One CTA per (128 nodes, head), two per SM.  For every block of 128 keys that any of its nodes may attend to, two steps
// of 64 keys: the two 64-node dS^T tiles' rows (8 KB each, already in the swizzled form the MMA reads) and the K rows
// (16 KB) come into a 3-stage ring, and four MMAs of 16 keys add to the 128 x 128 accumulator; both operands are read
// MN-major.  6 warps: producer, MMA issuer, 4 epilogue warps (one per TMEM lane quarter).
// What bounds it: the bytes of dS (2 per (node, key) pair), read once from HBM or L2.  Every wait is bounded.
#include "att_tc.cuh"

namespace ts2 {

namespace {

constexpr int DQ_THREADS = 192;
constexpr int DQ_STAGES = 3;
constexpr int DQ_STAGE_BYTES = 2 * 8192 + KV_BYTES; // 64 keys: dS^T of two 64-node tiles, K
constexpr int DQ_BAR_OFF = DQ_STAGES * DQ_STAGE_BYTES;
constexpr int DQ_SMEM = DQ_BAR_OFF + 256;
constexpr int DS_TILE_BYTES = TC_BM * TC_BN * 2;

struct AttBwdDqParams {
    int T, n_blocks, ds_tiles;
    const int *span_start, *span_finish;
    const int4 *blocks; // see att_layout
    const uint8_t *ds;
    int32_t *status;
};

template <bool OUT16>
__global__ void __launch_bounds__(DQ_THREADS, 2)
    att_bwd_dq_ds_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmOut, const AttBwdDqParams p)
{
    extern __shared__ __align__(1024) uint8_t att_dq_smem[];
    uint8_t *smem = att_dq_smem;
    if (smem_u32(smem) & 1023) { // the swizzled tiles need a 1024-byte aligned base; refuse instead of computing garbage
        if (threadIdx.x == 0)
            atomicOr(p.status, TS2_STATUS_BAD_ARG);
        return;
    }
    uint64_t *bars = (uint64_t *)(smem + DQ_BAR_OFF);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + DQ_STAGES), done = smem_u32(bars + 2 * DQ_STAGES);
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * DQ_STAGES + 1);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    int *rng = (int *)(tmem_slot + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nb = blockIdx.x, h = blockIdx.y, r0 = nb * TC_BM, col0 = h * TC_HD;

    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 128);
        tmem_relinquish();
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < DQ_STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(done, 1);
        *abort_flag = 0;
        rng[0] = 0x7fffffff;
        rng[1] = -1;
        fence_barrier_init();
        prefetch_tmap(&tmK);
    }
    __syncthreads();
    grid_dep_wait();
    if (threadIdx.x < TC_BM && r0 + (int)threadIdx.x < p.T) {
        const int a = p.span_start[r0 + threadIdx.x], e = p.span_finish[r0 + threadIdx.x];
        if (e >= a) {
            atomicMin(&rng[0], a);
            atomicMax(&rng[1], e);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_acc = *tmem_slot;
    const int kb0 = rng[1] >= rng[0] ? rng[0] / TC_BM : 0, kb1 = rng[1] >= rng[0] ? rng[1] / TC_BM : -1;
    const long long head_tiles = (long long)h * p.blocks[p.n_blocks].z;
    // first dS^T tile of this node block under key block kb, -1: that block's nodes and this one do not meet
    auto tile_of = [&](int kb) -> long long {
        const int4 tb = p.blocks[kb];
        const long long t = head_tiles + tb.z + 2 * nb - tb.x;
        return tb.y > 0 && 2 * nb >= tb.x && 2 * nb + 2 <= tb.x + tb.y && t + 2 <= p.ds_tiles ? t : -1;
    };

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            for (int kb = kb0; kb <= kb1 && ok; ++kb) {
                const long long t = tile_of(kb);
                if (t < 0)
                    continue;
                for (int half = 0; half < 2; ++half, ++it) {
                    const int st = it % DQ_STAGES;
                    if (!(ok = mbar_wait(empty0 + 8 * st, ((it / DQ_STAGES) & 1) ^ 1, abort_flag)))
                        break;
                    const uint32_t fb = full0 + 8 * st, sa = smem_u32(smem + st * DQ_STAGE_BYTES), sk = sa + 2 * 8192;
                    mbar_arrive_expect_tx(fb, DQ_STAGE_BYTES);
                    bulk_load(sa, p.ds + t * DS_TILE_BYTES + half * 8192, 8192, fb);
                    bulk_load(sa + 8192, p.ds + (t + 1) * DS_TILE_BYTES + half * 8192, 8192, fb);
                    tma_load_2d(sk, &tmK, fb, col0, kb * TC_BM + half * 64);
                    tma_load_2d(sk + KV_BYTES / 2, &tmK, fb, col0 + 64, kb * TC_BM + half * 64);
                }
            }
            if (*abort_flag) { // copies in flight must land before the CTA gives its shared memory back (bounded)
                const long long t0 = clock64();
                for (int i = max(0, it - DQ_STAGES); i < it; ++i)
                    while (!mbar_try_wait(full0 + 8 * (i % DQ_STAGES), (i / DQ_STAGES) & 1) && clock64() - t0 < 200000000ll) {
                    }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = umma_idesc_f16(TC_HD, true, true);
            int it = 0;
            bool ok = true;
            for (int kb = kb0; kb <= kb1 && ok; ++kb) {
                if (tile_of(kb) < 0)
                    continue;
                for (int half = 0; half < 2; ++half, ++it) {
                    const int st = it % DQ_STAGES;
                    if (!(ok = mbar_wait(full0 + 8 * st, (it / DQ_STAGES) & 1, abort_flag)))
                        break;
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + st * DQ_STAGE_BYTES);
                    // 16 keys = 16 rows of 128 bytes per step in both operands; 64-wide atoms 8 KB apart
                    umma_f16_x4(tmem_acc, umma_smem_desc(sa, 8192, 1024), umma_smem_desc(sa + 2 * 8192, 8192, 1024), idesc, it > 0 ? 1u : 0u, 128u, 128u);
                    tc_commit(empty0 + 8 * st);
                }
            }
            tc_commit(done); // also without any step: the epilogue then writes zeros
        }
    } else {
        const int quarter = warp & 3;
        bool any = false;
        for (int kb = kb0; kb <= kb1 && !any; ++kb)
            any = tile_of(kb) >= 0;
        bool ok = __all_sync(0xffffffffu, mbar_wait(done, 0, abort_flag));
        tc_fence_after();
        // a warp's 32 rows in blocks of 32 rows x 128 bytes through the idle ring (every MMA is complete), one TMA store each
        uint8_t *const stg = smem + quarter * (OUT16 ? 8192 : 16384);
        constexpr int BLOCKS = OUT16 ? 2 : 4;
#pragma unroll 1
        for (int b = 0; b < BLOCKS; ++b) {
            uint8_t *blk = stg + b * 4096;
            auto at = [&](int c) { return (uint4 *)(blk + lane * 128 + ((c ^ (lane & 7)) << 4)); };
#pragma unroll
            for (int hf = 0; hf < (OUT16 ? 2 : 1); ++hf) {
                uint32_t r[32];
                if (any && ok) {
                    tmem_ld32(tmem_acc + ((uint32_t)(quarter * 32) << 16) + (OUT16 ? b * 64 + hf * 32 : b * 32), r);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        r[i] = 0u;
                }
                if constexpr (OUT16) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const __half2 h0 = sat_half2(__uint_as_float(r[8 * i]), __uint_as_float(r[8 * i + 1])),
                                      h1 = sat_half2(__uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3])),
                                      h2 = sat_half2(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5])),
                                      h3 = sat_half2(__uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7]));
                        *at(4 * hf + i) = make_uint4(*(const uint32_t *)&h0, *(const uint32_t *)&h1, *(const uint32_t *)&h2, *(const uint32_t *)&h3);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        *at(i) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                tma_store_2d(&tmOut, smem_u32(blk), col0 + b * (OUT16 ? 64 : 32), r0 + quarter * 32);
                bulk_commit();
            }
        }
        if (lane == 0)
            bulk_wait_read<0>(); // shared memory must outlive the stores that read it
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1)
        tmem_dealloc(tmem_acc, 128);
    if (threadIdx.x == 0 && *abort_flag)
        atomicOr(p.status, TS2_STATUS_WAIT_TIMEOUT);
}

} // namespace

int attention_backward_dq_ds(const Ctx &c, const __half *k, const AttBwdPlan &plan, const int *span_start, const int *span_finish, int T, int H,
                             void *dq, bool out16)
{
    static bool configured[16] = {};
    if (!configured[c.device & 15]) {
        TS2_CUDA(cudaFuncSetAttribute(att_bwd_dq_ds_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, DQ_SMEM));
        TS2_CUDA(cudaFuncSetAttribute(att_bwd_dq_ds_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, DQ_SMEM));
        configured[c.device & 15] = true;
    }
    const int Q = H * TC_HD;
    CUtensorMap tK, tOut;
    int rc;
    if ((rc = make_tensor_map(&tK, k, 2, Q, T, Q, TC_BN)) != TS2_OK)
        return rc;
    if ((rc = make_tensor_map(&tOut, dq, out16 ? 2 : 4, Q, T, Q, 32)) != TS2_OK) // boxes of 128 bytes x 32 rows
        return rc;
    AttBwdDqParams p;
    p.T = T;
    p.n_blocks = (int)ceil_div(T, TC_BM);
    p.ds_tiles = (int)std::min<size_t>(plan.ds_bytes / DS_TILE_BYTES, 0x7fffffff);
    p.span_start = span_start;
    p.span_finish = span_finish;
    p.blocks = (const int4 *)plan.layout;
    p.ds = (const uint8_t *)plan.ds;
    p.status = device_status_word(c.device);
    if (!p.status)
        return fail(TS2_ERR_CUDA, "attention: no device status word");
    const dim3 grid((unsigned)p.n_blocks, (unsigned)H);
    if (out16)
        TS2_LAUNCH((att_bwd_dq_ds_kernel<true>), grid, DQ_THREADS, DQ_SMEM, c.stream, tK, tOut, p);
    else
        TS2_LAUNCH((att_bwd_dq_ds_kernel<false>), grid, DQ_THREADS, DQ_SMEM, c.stream, tK, tOut, p);
    return TS2_OK;
}

} // namespace ts2
