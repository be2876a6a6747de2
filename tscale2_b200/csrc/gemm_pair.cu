// The contraction on pairs of CTAs (tcgen05 cta_group::2), for problems with enough 256 x 256 tiles.
//
// Two CTAs of a cluster work on one tile: each holds 128 rows of A and 128 of the tile's 256 columns of B in its shared
// memory, the leader's MMA thread issues one 256 x 256 MMA that reads both, and each CTA's tensor memory receives its own
// 128 rows x 256 columns.  Against a 128 x 256 tile per CTA (gemm.cu) a K block brings 32 KB instead of 48 KB into an SM:
// a third less L2 and shared-memory traffic for the same work, and room for a ring of 4 stages beside 96 KB of epilogue
// staging.  The residual input of the accumulate form arrives in the staging blocks by TMA, one block ahead, instead of by
// 16-byte loads of 32 different rows.
// What bounds it: at K = 768 the main loop alone runs at 2900 TFLOP/s (e4m3, random operands), which is where this part's
// power limit holds the tensor pipe; the tile's stores add the rest (65536 x 6144 x 768, fp16 output: 213 us without
// epilogue, 238 without the stores, 298 with them).  Whole steps, pairs against single CTAs, ms per pass: 12 blocks x dim
// 768 x 65536 tokens 195.2 -> 189.6, 4 blocks x dim 2048 x 32768 tokens 159.6 -> 155.6, scoring in fp16 34.4 -> 32.4.
//
//   warp 0      TMA producer of its CTA's halves; all copies of a stage complete on the LEADER's full barrier
//   warp 1      tensor-memory owner; in the leader its first thread issues the MMAs and commits them to both CTAs
//   warps 2..   epilogue of the CTA's 128 rows: 8 warps, or 16 in the gated-activation form
// Units (tile, K split) are assigned statically to clusters.  Every wait is bounded, as in gemm.cu; a CTA leaves only
// after a cluster barrier, so no barrier or copy of its peer can still refer to it.
#include "gemm_params.cuh"
#include "row_math.cuh"

namespace ts2 {

namespace {

constexpr int PM = 256, PN = 256; // the pair's tile
constexpr int P_HALF_BYTES = 128 * STAGE_ROW_BYTES; // a CTA's half of either operand, one K block
constexpr int P_STAGE_BYTES = 2 * P_HALF_BYTES;
constexpr int P_THREADS = 320, P_THREADS_16 = 576;
constexpr bool epi8(int form) { return form == P_F32 || form == P_NORM || form == P_NORM_BWD; } // 8 epilogue warps, else 16
constexpr bool is_bwd(int form) { return form == P_ACT_BWD || form == P_GATE_BWD; }
// shared memory of a form: ring, epilogue staging, barriers, alignment slack
template <int FORM>
struct PairSmem {
    static constexpr int STAGES = is_bwd(FORM) ? 3 : 4;
    static constexpr int STG_OFF = STAGES * P_STAGE_BYTES;
    static constexpr int BAR_OFF = STG_OFF + (is_bwd(FORM) ? 16 * 2 * 4096 : 8 * 3 * 4096);
    static constexpr int TOTAL = BAR_OFF + 1024 + 1024;
    static_assert(TOTAL <= 232448, "shared memory budget");
};

__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_to_leader(uint32_t addr)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// a copy into this CTA's shared memory that completes on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void *tmap, uint32_t bar, int c0, int c1)
{
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                 "l"(tmap), "r"(bar), "r"(c0), "r"(c1)
                 : "memory");
}
template <int MMA>
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    if constexpr (MMA == 0)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
                     "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                     : "memory");
    else if constexpr (MMA == 1)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
                     "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                     : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
                     "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                     : "memory");
}
// arrives at the barrier at this offset in both CTAs when the MMAs issued so far are complete
__device__ __forceinline__ void commit_both(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ void commit_own(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

struct PairUnit {
    int m0, n0, nt, kb0, kb1;
};

__device__ __forceinline__ PairUnit pair_unit(const GemmParams &p, int u)
{
    PairUnit t;
    const int tile = u / p.splits, split = u - tile * p.splits;
    int mt;
    if (p.n_fast) {
        t.nt = tile % p.n_tiles;
        mt = tile / p.n_tiles;
    } else {
        mt = tile % p.m_tiles;
        t.nt = tile / p.m_tiles;
    }
    t.m0 = mt * PM;
    t.n0 = t.nt * (p.pair_stride ? PN / 2 : PN);
    t.kb0 = split * p.kb_per_split;
    t.kb1 = min(p.k_blocks, t.kb0 + p.kb_per_split);
    return t;
}

// 16-byte piece c of row r of a 32 x 128 byte block in the 128-byte swizzle
__device__ __forceinline__ uint32_t piece(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

// FORM of the epilogue (PairForm)
template <int ES, int MMA, bool MN, int FORM>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(epi8(FORM) ? P_THREADS : P_THREADS_16, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmCin,
                     const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmY, const GemmParams p)
{
    constexpr int ELEMS_PER_ROW = STAGE_ROW_BYTES / ES;
    constexpr int UMMA_K = 32 / ES, K_STEPS = 4, BK = ELEMS_PER_ROW;
    constexpr bool GATED = FORM == P_GATED;
    constexpr int EPI_WARPS = epi8(FORM) ? 8 : 16;
    constexpr int P_STAGES = PairSmem<FORM>::STAGES, P_STG_OFF = PairSmem<FORM>::STG_OFF, P_BAR_OFF = PairSmem<FORM>::BAR_OFF;

    extern __shared__ uint8_t pair_smem[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)pair_smem + 1023) & ~(uintptr_t)1023); // the same offset in both CTAs
    uint64_t *bars = (uint64_t *)(smem + P_BAR_OFF);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + P_STAGES), tfull0 = smem_u32(bars + 2 * P_STAGES),
                   tempty0 = smem_u32(bars + 2 * P_STAGES + 2), drain = smem_u32(bars + 2 * P_STAGES + 4),
                   cin0 = smem_u32(bars + 2 * P_STAGES + 5); // [warp][3]: residual block landed; the backward forms: see there
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * P_STAGES + 5 + 24);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    if (threadIdx.x == 0) {
        for (int s = 0; s < P_STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull0 + 8 * a, 1);
            mbar_init(tempty0 + 8 * a, 2 * EPI_WARPS); // the leader's counts the epilogue warps of both CTAs
        }
        for (int i = 0; i < 24; ++i)
            mbar_init(cin0 + 8 * i, is_bwd(FORM) && i >= 16 ? 2 : 1);
        mbar_init(drain, 1);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
        prefetch_tmap(&tmC);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync(); // both CTAs' barriers exist
    tc_fence_after();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;

    const int units = p.m_tiles * p.n_tiles * p.splits;
    const int first = (int)blockIdx.x >> 1, step = (int)gridDim.x >> 1;

    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            int stage = 0, issued = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int u = first; u < units && ok; u += step) {
                const PairUnit un = pair_unit(p, u);
                const int am = un.m0 + (int)rank * 128;
                const int bn = GATED ? un.n0 + (int)rank * p.pair_stride : un.n0 + (int)rank * 128;
                for (int kb = un.kb0; kb < un.kb1; ++kb) {
                    if (!mbar_wait(empty0 + 8 * stage, phase ^ 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    const uint32_t fb = map_to_leader(full0 + 8 * stage);
                    if (rank == 0)
                        mbar_arrive_expect_tx(full0 + 8 * stage, 2 * P_STAGE_BYTES);
                    const uint32_t sa = smem_u32(smem + stage * P_STAGE_BYTES), sb = sa + P_HALF_BYTES;
                    const int k0 = kb * BK;
                    if constexpr (!MN) {
                        tma_load_2d_pair(sa, &tmA, fb, k0, am);
                        tma_load_2d_pair(sb, &tmB, fb, k0, bn);
                    } else {
#pragma unroll
                        for (int j = 0; j < 128 / ELEMS_PER_ROW; ++j)
                            tma_load_2d_pair(sa + j * BK * STAGE_ROW_BYTES, &tmA, fb, am + j * ELEMS_PER_ROW, k0);
#pragma unroll
                        for (int j = 0; j < 128 / ELEMS_PER_ROW; ++j)
                            tma_load_2d_pair(sb + j * BK * STAGE_ROW_BYTES, &tmB, fb, bn + j * ELEMS_PER_ROW, k0);
                    }
                    ++issued;
                    if (++stage == P_STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok && rank == 0) {
                // abort path: copies of both CTAs complete on the leader's barriers: wait (bounded) for those in flight; the
                // cluster barrier at the end keeps the peer here as long
                int s = stage;
                uint32_t ph = phase;
                for (int i = 0; i < min(issued, P_STAGES); ++i) {
                    if (--s < 0) {
                        s = P_STAGES - 1;
                        ph ^= 1;
                    }
                    long long t0 = clock64();
                    while (!mbar_try_wait(full0 + 8 * s, ph) && clock64() - t0 < 200000000ll) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer (leader) -----------------------
        if (lane == 0 && rank == 0) {
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            for (int u = first; u < units && ok; u += step) {
                const PairUnit un = pair_unit(p, u);
                if (!mbar_wait(tempty0 + 8 * acc, acc_phase ^ 1, abort_flag))
                    break;
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + acc * PN;
                for (int kb = un.kb0; kb < un.kb1; ++kb) {
                    if (!mbar_wait(full0 + 8 * stage, phase, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + stage * P_STAGE_BYTES), sb = sa + P_HALF_BYTES;
                    const uint32_t lbo = MN ? BK * STAGE_ROW_BYTES : 16;
                    const uint64_t adesc = umma_smem_desc(sa, lbo, 1024), bdesc = umma_smem_desc(sb, lbo, 1024);
                    const uint32_t kstep = MN ? (UMMA_K * STAGE_ROW_BYTES) >> 4 : (UMMA_K * ES) >> 4;
#pragma unroll
                    for (int k = 0; k < K_STEPS; ++k)
                        umma_pair<MMA>(tmem_d, adesc + (uint64_t)(k * kstep), bdesc + (uint64_t)(k * kstep), p.idesc, (kb > un.kb0 || k > 0) ? 1u : 0u);
                    commit_both(empty0 + 8 * stage);
                    if (++stage == P_STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (ok)
                    commit_both(tfull0 + 8 * acc);
                acc ^= 1;
                if (acc == 0)
                    acc_phase ^= 1;
            }
            // every MMA issued so far has completed once this commit arrives
            commit_own(drain);
            long long t0 = clock64();
            while (!mbar_try_wait(drain, 0) && clock64() - t0 < 1500000000ll) {
            }
        }
    } else {
        // ------------------------------ epilogue ----------------------------------
        const int quarter = warp & 3;
        const int ew = warp - 2;
        float alpha = p.alpha;
        if (p.splits > 1) {
            alpha = 1.f; // partial tiles leave unscaled; the reduction applies the epilogue
        } else {
            if (p.dyn_scale)
                alpha *= __ldg(p.dyn_scale);
            if (p.dyn_scale2)
                alpha *= __ldg(p.dyn_scale2);
        }
        const bool scaled = p.splits == 1;
        const int row_in_cta = quarter * 32 + lane;
        int acc = 0;
        uint32_t acc_phase = 0;
        if constexpr (GATED) {
            // see gemm.cu: TMEM columns [0, 128) hold the wide tile, [128, 256) the gate tile; warp part j of a lane
            // quarter takes wide columns [32 j, +32) and the gate columns under them
            const int part = ew >> 2;
            uint8_t *const stg = smem + P_STG_OFF + ew * 6144; // three blocks of 32 rows x 64 bytes (64-byte swizzle)
            int sblk = 0;
            for (int u = first; u < units; u += step) {
                const PairUnit un = pair_unit(p, u);
                if (!__all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, acc_phase, abort_flag)))
                    break;
                tc_fence_after();
                const int m0 = un.m0 + (int)rank * 128;
                const long long row = m0 + row_in_cta;
                const int wcol = un.n0 + part * 32, gcol = p.pair_stride + wcol;
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * PN;
                auto value = [&](uint32_t r) { return (MMA == 2) ? (float)(int)r : __uint_as_float(r); };
                auto stage_store16 = [&](const float *v, int col) {
                    uint8_t *blk = stg + sblk * 2048, *srow = blk + lane * 64;
                    sblk = sblk == 2 ? 0 : sblk + 1;
                    const int sw = (lane >> 1) & 3;
                    if (lane == 0)
                        bulk_wait_read<2>(); // the store that last used this block has read it
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        __half2 h0 = sat_half2(v[8 * i], v[8 * i + 1]), h1 = sat_half2(v[8 * i + 2], v[8 * i + 3]),
                                h2 = sat_half2(v[8 * i + 4], v[8 * i + 5]), h3 = sat_half2(v[8 * i + 6], v[8 * i + 7]);
                        *(uint4 *)(srow + ((i ^ sw) << 4)) = make_uint4(*(uint32_t *)&h0, *(uint32_t *)&h1, *(uint32_t *)&h2, *(uint32_t *)&h3);
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        if (col < p.N)
                            tma_store_2d(&tmC, smem_u32(blk), col, m0 + quarter * 32);
                        bulk_commit();
                    }
                };
                float wv[32], sum2 = 0.f;
                {
                    uint32_t r[32];
                    tmem_ld32(taddr + part * 32, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        wv[i] = value(r[i]) * alpha;
                        sum2 = fmaf(wv[i], wv[i], sum2);
                    }
                }
#pragma unroll 1
                for (int oc = 1; oc < 4; ++oc) {
                    uint32_t r[32];
                    tmem_ld32(taddr + ((part + oc) & 3) * 32, r);
                    tmem_ld_wait();
                    float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const float v = value(r[i]) * alpha;
                        s4[i & 3] = fmaf(v, v, s4[i & 3]);
                    }
                    sum2 += (s4[0] + s4[1]) + (s4[2] + s4[3]);
                }
                float gv[32];
                {
                    uint32_t r[32];
                    tmem_ld32(taddr + 128 + part * 32, r);
                    tmem_ld_wait();
                    // the accumulator is read: the next tile may have it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive_cluster(map_to_leader(tempty0 + 8 * acc));
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        gv[i] = value(r[i]) * alpha;
                }
                acc ^= 1;
                if (acc == 0)
                    acc_phase ^= 1;
                const float tscale = tile_scale(sum2);
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    wv[i] *= tscale;
                if (part == 0 && row < p.M)
                    p.act_scale[row * p.n_tiles + un.nt] = tscale;
                stage_store16(wv, wcol);
                stage_store16(gv, gcol);
                if (row < p.M) {
                    const size_t aidx = (size_t)row * p.act_ld + wcol;
                    if (p.act_kind == 0) {
                        // sigmoid(2 g) = 0.5 + 0.5 tanh(g): one MUFU op; its 2^-11 error is far below the e4m3 step
                        const float hm = 0.5f * p.act_mult;
                        auto gated = [&](int e) {
                            float th;
                            asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(gv[e]));
                            return fmaf(th, hm, hm) * wv[e];
                        };
#pragma unroll
                        for (int j = 0; j < 2; ++j) { // 16 e4m3 bytes per store
                            uint32_t w4[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const int e = 16 * j + 4 * i;
                                __nv_fp8x4_e4m3 pk(make_float4(gated(e), gated(e + 1), gated(e + 2), gated(e + 3)));
                                w4[i] = pk.__x;
                            }
                            *(uint4 *)((uint8_t *)p.act_out + aidx + 16 * j) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float4 a = make_float4(lolu_mult(gv[4 * i]) * wv[4 * i] * p.act_mult, lolu_mult(gv[4 * i + 1]) * wv[4 * i + 1] * p.act_mult,
                                                         lolu_mult(gv[4 * i + 2]) * wv[4 * i + 2] * p.act_mult,
                                                         lolu_mult(gv[4 * i + 3]) * wv[4 * i + 3] * p.act_mult);
                            if (p.act_kind == 2)
                                Fast<2>::store4(p.act_out, aidx + 4 * i, a);
                            else
                                Fast<1>::store4(p.act_out, aidx + 4 * i, a);
                        }
                    }
                }
            }
        } else if constexpr (is_bwd(FORM)) {
            // Backward of the gated activation (ffn_act_backward in kernels_elem.cu, same arithmetic) on the accumulator: a warp
            // takes 32 rows x 64 columns; the two warps of a 128-wide normalisation tile add their halves of its projection.
            // [wide | gate] values arrive by TMA in two 4 KB blocks per warp, a tile ahead; both gradients leave through the gate's
            // block.  As a kernel of its own this read the product back: 65536 x 3072 x 768 took 155 + 309 us, both bound by
            // their bytes; the product (2 x 403 MB of 2 GB) no longer goes through memory, 329 us.
            // P_GATE_BWD, the attention gate (att_gate_backward): o in place of the wide values, the gradient of o in place of
            // theirs, which leaves through o's block, and the sum of the products of both over the 128 columns of a head.
            // 65536 x 1536 x 768 as two kernels 82 + 158 us, in one 184.
            constexpr bool ATT = FORM == P_GATE_BWD;
            const int part = ew >> 2, gate0 = ATT ? 3 * p.N : p.N; // first gate column
            uint8_t *const wblk = smem + P_STG_OFF + ew * 8192, *const gblk = wblk + 4096;
            const uint32_t in_bar = cin0 + 8 * ew, mate = cin0 + 8 * (16 + (ew & 3) + 4 * (part >> 1)); // mate: both warps of a tile
            const volatile float *const theirs = (const volatile float *)(smem + P_STG_OFF + (ew ^ 4) * 8192 + 4096 + 2048) + lane;
            float *const mine = (float *)(gblk + 2048) + lane;
            auto fetch = [&](int u, bool gate) { // lane 0
                const PairUnit un = pair_unit(p, u);
                const int col = un.n0 + part * 64, r0 = un.m0 + (int)rank * 128 + quarter * 32;
                if (!gate)
                    mbar_arrive_expect_tx(in_bar, 8192);
                if (gate)
                    tma_load_2d(smem_u32(gblk), &tmCin, in_bar, gate0 + col, r0);
                else
                    tma_load_2d(smem_u32(wblk), ATT ? &tmX : &tmCin, in_bar, col, r0);
            };
            if (lane == 0 && first < units) {
                fetch(first, false);
                fetch(first, true);
            }
            uint32_t in_phase = 0;
            bool ok = true, coming = true; // coming: blocks of the next tile are on their way
            for (int u = first; u < units; u += step) {
                const PairUnit un = pair_unit(p, u);
                const int m0 = un.m0 + (int)rank * 128, col = un.n0 + part * 64;
                const long long row = m0 + row_in_cta;
                const float scale = !ATT && row < p.M && col < p.N ? p.act_scale[row * (p.N >> 7) + (col >> 7)] : 0.f;
                ok = __all_sync(0xffffffffu, mbar_wait(in_bar, in_phase, abort_flag));
                if (!ok)
                    break;
                in_phase ^= 1;
                coming = false;
                ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, acc_phase, abort_flag));
                if (!ok)
                    break;
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * PN + part * 64;
                const __half2 one = __float2half2_rn(1.f), two = __float2half2_rn(2.f);
                __half2 dw[32]; // gradient of the normalised wide values (of o)
                uint32_t dg[16];
                float proj = 0.f;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t r[32];
                    tmem_ld32(taddr + h * 32, r);
                    tmem_ld_wait();
                    if (h == 1) { // the accumulator is read: the next tile may have it
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0)
                            mbar_arrive_cluster(map_to_leader(tempty0 + 8 * acc));
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint4 w4 = *(const uint4 *)(wblk + piece(lane, 4 * h + i)), g4 = *(const uint4 *)(gblk + piece(lane, 4 * h + i));
                        const uint32_t wv[4] = {w4.x, w4.y, w4.z, w4.w}, gv[4] = {g4.x, g4.y, g4.z, g4.w};
                        __half2 dgate[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int e = 8 * i + 2 * j;
                            const __half2 g = sat_half2(__uint_as_float(r[e]) * alpha, __uint_as_float(r[e + 1]) * alpha);
                            const __half2 w = h2_from_bits(wv[j]), m = lolu_mult_h2(h2_from_bits(gv[j]));
                            dgate[j] = __hmul2(g, __hmul2(w, __hmul2(__hmul2(m, two), __hsub2(one, m))));
                            const __half2 d = __hmul2(g, m);
                            dw[16 * h + 4 * i + j] = d;
                            if constexpr (ATT) { // from the fp16 values the attention kernels will read
                                const float2 a = __half22float2(d), b = __half22float2(w);
                                proj = fmaf(a.x, b.x, fmaf(a.y, b.y, proj));
                            } else {
                                const float2 pr = __half22float2(__hmul2(w, d));
                                proj += pr.x + pr.y;
                            }
                        }
                        if constexpr (ATT) // over the values it came from, which only this thread reads
                            *(uint4 *)(wblk + piece(lane, 4 * h + i)) =
                                make_uint4(bits_from_h2(dw[16 * h + 4 * i]), bits_from_h2(dw[16 * h + 4 * i + 1]),
                                           bits_from_h2(dw[16 * h + 4 * i + 2]), bits_from_h2(dw[16 * h + 4 * i + 3]));
                        dg[8 * h + 2 * i] = e4m3x4_from_h2(dgate[0], dgate[1]);
                        dg[8 * h + 2 * i + 1] = e4m3x4_from_h2(dgate[2], dgate[3]);
                    }
                }
                __syncwarp(); // every lane has read its row of the gate's block
                uint8_t *const srow = gblk + lane * 64; // blocks of 32 rows x 64 bytes (64-byte swizzle)
                const int sw = (lane >> 1) & 3;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    *(uint4 *)(srow + ((i ^ sw) << 4)) = make_uint4(dg[4 * i], dg[4 * i + 1], dg[4 * i + 2], dg[4 * i + 3]);
                *mine = proj;
                // first phase: both halves are written; second: both are read.  Two phases per tile: the parities are fixed
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(mate);
                ok = __all_sync(0xffffffffu, mbar_wait(mate, 0, abort_flag));
                if (!ok)
                    break;
                proj += *theirs;
                if (ATT && (part & 1) == 0 && row < p.M && col < p.N)
                    p.bwd_dscale[row * (p.N >> 7) + (col >> 7)] = proj;
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(mate);
                ok = __all_sync(0xffffffffu, mbar_wait(mate, 1, abort_flag));
                if (!ok)
                    break;
                if constexpr (!ATT) {
                    const __half2 nproj = __float2half2_rn(proj * (-1.f / 128)), sc = __float2half2_rn(scale);
                    uint32_t dx[16];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint4 w4 = *(const uint4 *)(wblk + piece(lane, i));
                        const uint32_t wv[4] = {w4.x, w4.y, w4.z, w4.w};
                        __half2 d[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            d[j] = __hmul2(sc, __hfma2(h2_from_bits(wv[j]), nproj, dw[4 * i + j]));
                        dx[2 * i] = e4m3x4_from_h2(d[0], d[1]);
                        dx[2 * i + 1] = e4m3x4_from_h2(d[2], d[3]);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        *(uint4 *)(srow + 2048 + ((i ^ sw) << 4)) = make_uint4(dx[4 * i], dx[4 * i + 1], dx[4 * i + 2], dx[4 * i + 3]);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    if (col < p.N) {
                        tma_store_2d(&tmC, smem_u32(gblk), gate0 + col, m0 + quarter * 32);
                        if constexpr (ATT)
                            tma_store_2d(&tmY, smem_u32(wblk), col, m0 + quarter * 32);
                        else
                            tma_store_2d(&tmC, smem_u32(gblk) + 2048, col, m0 + quarter * 32);
                    }
                    bulk_commit();
                    if (u + step < units) {
                        if constexpr (!ATT)
                            fetch(u + step, false);
                        bulk_wait_read<0>(); // the stores have read their blocks
                        if constexpr (ATT)
                            fetch(u + step, false);
                        fetch(u + step, true);
                    }
                }
                coming = u + step < units;
                __syncwarp();
                acc ^= 1;
                if (acc == 0)
                    acc_phase ^= 1;
            }
            // abort path: blocks may still be on their way into this CTA's shared memory
            if (!ok && lane == 0 && coming) {
                long long t0 = clock64();
                while (!mbar_try_wait(in_bar, in_phase) && clock64() - t0 < 200000000ll) {
                }
            }
        } else if constexpr (FORM == P_LSE) {
            // Scoring: nothing of the logits leaves the chip but each row's maximum and sum per 64 columns (an eighth of a percent
            // of their bytes) and the target's logit.  12000 x 50304 logits x 768, fp16: 700 us and 26 for the sum over the partial
            // results, where logits in memory (2.4 GB written and read) took 790 and 320.  18 warps leave 96 registers
            // a thread: 44 bytes spilled, 56 loaded.
            const int part = ew >> 2;
            for (int u = first; u < units; u += step) {
                const PairUnit un = pair_unit(p, u);
                const long long row = un.m0 + (int)rank * 128 + row_in_cta;
                const int col = un.n0 + part * 64;
                const int target = row < p.M ? p.lse_target[row] - col : -1; // 0 .. 63: in this thread's columns
                if (!__all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, acc_phase, abort_flag)))
                    break;
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * PN + part * 64;
                float v[64], mx = -INFINITY;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t r[32];
                    tmem_ld32(taddr + h * 32, r);
                    tmem_ld_wait();
                    if (h == 1) { // the accumulator is read: the next tile may have it
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0)
                            mbar_arrive_cluster(map_to_leader(tempty0 + 8 * acc));
                    }
                    const bool cols = col + h * 32 < p.N; // N is a multiple of 32
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float4 b = p.lse_bias && cols ? __ldg((const float4 *)(p.lse_bias + col + h * 32) + i) : make_float4(0, 0, 0, 0);
                        auto val = [&](int k) { return (MMA == 2) ? (float)(int)r[4 * i + k] : __uint_as_float(r[4 * i + k]); };
                        float *o = v + 32 * h + 4 * i;
                        o[0] = cols ? fmaf(val(0), alpha, b.x) : -INFINITY;
                        o[1] = cols ? fmaf(val(1), alpha, b.y) : -INFINITY;
                        o[2] = cols ? fmaf(val(2), alpha, b.z) : -INFINITY;
                        o[3] = cols ? fmaf(val(3), alpha, b.w) : -INFINITY;
                        mx = fmaxf(mx, fmaxf(fmaxf(o[0], o[1]), fmaxf(o[2], o[3])));
                    }
                }
                if (__any_sync(0xffffffffu, (unsigned)target < 64u)) { // one tile in a hundred or so
                    float x = 0.f;
#pragma unroll
                    for (int i = 0; i < 64; ++i)
                        x = i == target ? v[i] : x;
                    if ((unsigned)target < 64u)
                        p.lse_logit[row] = x;
                }
                float s4[4] = {0.f, 0.f, 0.f, 0.f};
                const float ref = mx == -INFINITY ? 0.f : mx;
#pragma unroll
                for (int i = 0; i < 64; ++i) {
                    float e;
                    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(v[i] - ref));
                    s4[i & 3] += e;
                }
                if (row < p.M)
                    p.lse_partial[(size_t)(un.nt * 4 + part) * p.M + row] = make_float2(mx, (s4[0] + s4[1]) + (s4[2] + s4[3]));
                acc ^= 1;
                if (acc == 0)
                    acc_phase ^= 1;
            }
        } else if constexpr (FORM == P_16) {
            // Sixteen warps, four per lane quarter, 64 columns of the tile each: one block of 32 rows x 128 bytes in the 128-byte
            // swizzle and one store per tile.  With eight warps a tile of K = 768 took 3.6 us, 2.6 of them its main loop and
            // hardly any of the difference the stores themselves: a warp's chain of tensor-memory load, conversion, shared
            // memory, fence and store is latency, and twice the warps hide twice as much of it.
            const int part = ew >> 2;
            uint8_t *const blk = smem + P_STG_OFF + ew * 4096;
            for (int u = first; u < units; u += step) {
                const PairUnit un = pair_unit(p, u);
                const int m0 = un.m0 + (int)rank * 128;
                const long long row = m0 + row_in_cta;
                float rs = alpha;
                if (p.row_scale && row < p.M)
                    rs *= __ldg(p.row_scale + row);
                if (!__all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, acc_phase, abort_flag)))
                    break;
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * PN + part * 64;
                const int col = un.n0 + part * 64;
                if (lane == 0)
                    bulk_wait_read<0>(); // the previous tile's store has read the block
                __syncwarp();
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t r[32];
                    tmem_ld32(taddr + h * 32, r);
                    tmem_ld_wait();
                    if (h == 1) { // the accumulator is read: the next tile may have it
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0)
                            mbar_arrive_cluster(map_to_leader(tempty0 + 8 * acc));
                    }
                    const bool cols = p.col_scale && col + h * 32 < p.N;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint32_t pk[4];
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            const int e = 8 * i + 4 * j;
                            float4 cs = make_float4(rs, rs, rs, rs);
                            if (cols) {
                                const float4 c = __ldg((const float4 *)(p.col_scale + col + h * 32 + e));
                                cs = make_float4(c.x * rs, c.y * rs, c.z * rs, c.w * rs);
                            }
                            auto val = [&](int k) { return (MMA == 2) ? (float)(int)r[k] : __uint_as_float(r[k]); };
                            const float v0 = val(e) * cs.x, v1 = val(e + 1) * cs.y, v2 = val(e + 2) * cs.z, v3 = val(e + 3) * cs.w;
                            if (p.out_kind == TS2_OUT_F16) {
                                const __half2 h0 = sat_half2(v0, v1), h1 = sat_half2(v2, v3);
                                pk[2 * j] = *(const uint32_t *)&h0, pk[2 * j + 1] = *(const uint32_t *)&h1;
                            } else {
                                const __nv_bfloat162 h0 = __floats2bfloat162_rn(v0, v1), h1 = __floats2bfloat162_rn(v2, v3);
                                pk[2 * j] = *(const uint32_t *)&h0, pk[2 * j + 1] = *(const uint32_t *)&h1;
                            }
                        }
                        *(uint4 *)(blk + piece(lane, 4 * h + i)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                    }
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    if (col < p.N)
                        tma_store_2d(&tmC, smem_u32(blk), col, m0 + quarter * 32);
                    bulk_commit();
                }
                acc ^= 1;
                if (acc == 0)
                    acc_phase ^= 1;
            }
        } else if constexpr (FORM == P_NORM || FORM == P_NORM_BWD) {
            // The row-wise step behind a layer's last contraction: a thread has the 128 columns of a normalisation tile of its
            // row, 32 at a time through the warp's three staging buffers.  A buffer is taken again when all stores but the most
            // recent one have read theirs: `cur` holds the block that was fetched ahead, `prev` was stored from last, the third
            // one is free.
            // P_NORM: C = c_in + product, and its tile normalisation, which as a kernel of its own read C back (65536 x 768,
            // e4m3: contraction 121 and normalisation 48 -> 138 us).  P_NORM_BWD: the product d (scale-free, times dyn_scale2) is
            // the gradient of the normalised x; the accumulator is read twice, beside x for the two sums over the tile and beside
            // g for the result; the product used to go through memory (65536 x 768, e4m3: contraction 239 and normalisation 114
            // -> 277 us).
            // What bounds both: 128 values a thread stay in registers from one pass to the next, and ten warps leave 168 registers
            // a thread: they spill (stored / loaded bytes a thread, e4m3: 332 / 396, backward 152 / 340; fp16 452 / 552).  0.52 GB in
            // 115 us and 1.05 GB in 277 are 4.5 and 3.8 TB/s.
            constexpr bool BWD = FORM == P_NORM_BWD;
            const int half = ew >> 2;
            uint8_t *const stg = smem + P_STG_OFF + ew * (3 * 4096);
            const uint32_t cin_bar = cin0 + 8 * 3 * ew;
            int cur = 0, prev = 2;
            uint32_t cin_phase = 0; // one bit per buffer
            auto fetch = [&](const CUtensorMap *tm, int u, int b, int to) {
                if (lane == 0) {
                    const PairUnit un = pair_unit(p, u);
                    mbar_arrive_expect_tx(cin_bar + 8 * to, 4096);
                    tma_load_2d(smem_u32(stg + to * 4096), tm, cin_bar + 8 * to, un.n0 + half * 128 + b * 32, un.m0 + (int)rank * 128 + quarter * 32);
                }
            };
            const CUtensorMap *const first_in = BWD ? &tmX : &tmCin;
            if (first < units)
                fetch(first_in, first, 0, 0);
            bool ok = true;
            float mx = 0.f;
            for (int u = first; u < units; u += step) {
                const PairUnit un = pair_unit(p, u);
                const int m0 = un.m0 + (int)rank * 128, col = un.n0 + half * 128;
                const bool inside = col < p.N;
                ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, acc_phase, abort_flag));
                if (!ok)
                    break;
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * PN + half * 128;
                auto value = [&](uint32_t r) { return (MMA == 2) ? (float)(int)r : __uint_as_float(r); };
                auto release = [&]() { // the accumulator is read: the next tile may have it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive_cluster(map_to_leader(tempty0 + 8 * acc));
                };
                // the block that was fetched ahead is in `cur`; the one after it goes into the free buffer
                auto landed = [&](const CUtensorMap *tm, int nu, int nb) {
                    const int free_buf = 3 - cur - prev;
                    if (lane == 0)
                        bulk_wait_read<1>();
                    if (nu < units)
                        fetch(tm, nu, nb, free_buf);
                    const bool got = __all_sync(0xffffffffu, mbar_wait(cin_bar + 8 * cur, (cin_phase >> cur) & 1, abort_flag));
                    cin_phase ^= 1u << cur;
                    return got;
                };
                auto stored = [&](const CUtensorMap *tm, int x) { // the block in `cur` leaves; a group is committed also for a clipped one
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        if (inside)
                            tma_store_2d(tm, smem_u32(stg + cur * 4096), x, m0 + quarter * 32);
                        bulk_commit();
                    }
                    const int next = 3 - cur - prev;
                    prev = cur;
                    cur = next;
                };
                float keep[4][32], sum2 = 0.f;
                if constexpr (!BWD) {
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        uint32_t r[32];
                        tmem_ld32(taddr + b * 32, r);
                        tmem_ld_wait();
                        if (b == 3)
                            release();
                        if (!(ok = landed(&tmCin, b < 3 ? u : u + step, (b + 1) & 3)))
                            break;
                        uint8_t *blk = stg + cur * 4096;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            float4 *q = (float4 *)(blk + piece(lane, i));
                            const float4 c = *q;
                            const float4 o = make_float4(c.x + value(r[4 * i]) * alpha, c.y + value(r[4 * i + 1]) * alpha, c.z + value(r[4 * i + 2]) * alpha,
                                                         c.w + value(r[4 * i + 3]) * alpha);
                            *q = o;
                            sum2 += dot4(o, o);
                            keep[b][4 * i] = o.x, keep[b][4 * i + 1] = o.y, keep[b][4 * i + 2] = o.z, keep[b][4 * i + 3] = o.w;
                        }
                        stored(&tmC, col + b * 32);
                    }
                    if (!ok)
                        break;
                    // `cur` now holds the next tile's first block (or nothing): the normalised rows leave from the free buffer
                    const float scale = tile_scale(sum2), mult = p.act_mult;
                    auto leave = [&](const CUtensorMap *tm, int x, auto words) { // words(i): 16-byte piece i of this row
                        const int buf = 3 - cur - prev;
                        if (lane == 0)
                            bulk_wait_read<1>();
                        __syncwarp();
                        uint8_t *blk = stg + buf * 4096;
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            *(uint4 *)(blk + piece(lane, i)) = words(i);
                        fence_proxy_async();
                        __syncwarp();
                        if (lane == 0) {
                            if (inside)
                                tma_store_2d(tm, smem_u32(blk), x, m0 + quarter * 32);
                            bulk_commit();
                        }
                        prev = buf;
                    };
                    auto half8 = [&](const float *v, float s) {
                        float f[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            f[j] = v[j] * scale * s;
                        return make_uint4(bits_from_h2(sat_half2(f[0], f[1])), bits_from_h2(sat_half2(f[2], f[3])), bits_from_h2(sat_half2(f[4], f[5])),
                                          bits_from_h2(sat_half2(f[6], f[7])));
                    };
                    if constexpr (MMA == 1) {
#pragma unroll
                        for (int hb = 0; hb < 2; ++hb)
                            leave(&tmX, col + hb * 64, [&](int i) { return half8(&keep[2 * hb + (i >> 2)][(i & 3) * 8], mult); });
                    } else {
                        leave(&tmX, col, [&](int i) {
                            uint32_t w[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float *v = &keep[i >> 1][(i & 1) * 16 + 4 * j];
                                const float4 f = scale4(scale4(make_float4(v[0], v[1], v[2], v[3]), scale), mult);
                                if (MMA == 0) {
                                    __nv_fp8x4_e4m3 pk(f);
                                    w[j] = pk.__x;
                                } else {
                                    w[j] = sat_i8(f.x) | (sat_i8(f.y) << 8) | (sat_i8(f.z) << 16) | (sat_i8(f.w) << 24);
                                }
                            }
                            return make_uint4(w[0], w[1], w[2], w[3]);
                        });
                    }
                    if (p.norm16) {
#pragma unroll
                        for (int hb = 0; hb < 2; ++hb)
                            leave(&tmY, col + hb * 64, [&](int i) { return half8(&keep[2 * hb + (i >> 2)][(i & 3) * 8], 1.f); });
                    }
                } else {
                    float dp = 0.f;
                    const float rs = p.row_scale && m0 + row_in_cta < p.M ? alpha * __ldg(p.row_scale + m0 + row_in_cta) : alpha;
                    const float dyn = p.norm_dyn ? __ldg(p.norm_dyn) : 1.f;
#pragma unroll
                    for (int b = 0; b < 4; ++b) { // x beside the product: both sums over the tile
                        uint32_t r[32];
                        tmem_ld32(taddr + b * 32, r);
                        tmem_ld_wait();
                        if (!(ok = landed(b < 3 ? &tmX : &tmCin, u, (b + 1) & 3)))
                            break;
                        const uint8_t *blk = stg + cur * 4096;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float4 x = *(const float4 *)(blk + piece(lane, i));
                            const float4 d = scale4(make_float4(value(r[4 * i]) * rs, value(r[4 * i + 1]) * rs, value(r[4 * i + 2]) * rs, value(r[4 * i + 3]) * rs), dyn);
                            sum2 += dot4(x, x);
                            dp += dot4(x, d);
                            keep[b][4 * i] = x.x, keep[b][4 * i + 1] = x.y, keep[b][4 * i + 2] = x.z, keep[b][4 * i + 3] = x.w;
                        }
                        // nothing leaves from this buffer: every lane has read its row.  An empty group keeps the count of those that
                        // may still be reading.
                        __syncwarp();
                        if (lane == 0)
                            bulk_commit();
                        const int next = 3 - cur - prev;
                        prev = cur;
                        cur = next;
                    }
                    if (!ok)
                        break;
                    const float sigma = sum2 != 0.f ? dp / sum2 : 0.f, scale = sum2 != 0.f ? sqrtf(128.f / sum2) : 0.f;
                    const bool row_in = m0 + row_in_cta < p.M && inside;
#pragma unroll
                    for (int b = 0; b < 4; ++b) { // g beside it once more
                        uint32_t r[32];
                        tmem_ld32(taddr + b * 32, r);
                        tmem_ld_wait();
                        if (b == 3)
                            release();
                        if (!(ok = landed(b < 3 ? &tmCin : &tmX, b < 3 ? u : u + step, (b + 1) & 3)))
                            break;
                        uint8_t *blk = stg + cur * 4096;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            float4 *q = (float4 *)(blk + piece(lane, i));
                            const float4 g = p.norm_add ? *q : make_float4(0, 0, 0, 0);
                            const float4 d = scale4(make_float4(value(r[4 * i]) * rs, value(r[4 * i + 1]) * rs, value(r[4 * i + 2]) * rs, value(r[4 * i + 3]) * rs), dyn);
                            const float *x = &keep[b][4 * i];
                            const float4 o = make_float4(g.x + scale * (d.x - x[0] * sigma), g.y + scale * (d.y - x[1] * sigma),
                                                         g.z + scale * (d.z - x[2] * sigma), g.w + scale * (d.w - x[3] * sigma));
                            *q = o;
                            if (row_in)
                                mx = absmax4(mx, o);
                        }
                        stored(&tmC, col + b * 32);
                    }
                    if (!ok)
                        break;
                }
                acc ^= 1;
                if (acc == 0)
                    acc_phase ^= 1;
            }
            if constexpr (BWD) {
                mx = warp_max(mx);
                if (ok && lane == 0 && first < units)
                    absmax_report(mx, p.norm_absmax, p.norm_health, p.norm_step);
            }
            // abort path: a block may still be on its way into this CTA's shared memory
            if (!ok && lane == 0) {
                long long t0 = clock64();
                for (int i = 0; i < 3; ++i)
                    while (!mbar_try_wait(cin_bar + 8 * i, (cin_phase >> i) & 1) && clock64() - t0 < 200000000ll) {
                    }
            }
        } else {
            // The two warps of a quarter take 128 columns each, in 4 blocks of 32 rows x 32 columns.  Blocks go through the
            // warp's three staging buffers in turn; before a buffer is refilled all stores but the two most recent must have
            // read theirs (a group is committed for every block, also a clipped one, so that the count stays right).
            const int half = ew >> 2;
            uint8_t *const stg = smem + P_STG_OFF + ew * (3 * 4096);
            const uint32_t cin_bar = cin0 + 8 * 3 * ew;
            const bool partial = p.splits > 1;
            const bool add = !partial && p.out_kind == TS2_OUT_F32_ADD;
            int buf = 0;
            uint32_t cin_phase = 0; // one bit per buffer
            // residual block `b` (0..3) of unit u into buffer `to`
            auto fetch_cin = [&](int u, int b, int to) {
                if (lane == 0) {
                    const PairUnit un = pair_unit(p, u);
                    mbar_arrive_expect_tx(cin_bar + 8 * to, 4096);
                    tma_load_2d(smem_u32(stg + to * 4096), &tmCin, cin_bar + 8 * to, un.n0 + half * 128 + b * 32,
                                un.m0 + (int)rank * 128 + quarter * 32);
                }
            };
            if (add && first < units)
                fetch_cin(first, 0, 0);
            bool ok = true;
            for (int u = first; u < units; u += step) {
                const PairUnit un = pair_unit(p, u);
                const int m0 = un.m0 + (int)rank * 128;
                const long long row = m0 + row_in_cta;
                float rs = alpha;
                if (scaled && p.row_scale && row < p.M)
                    rs *= __ldg(p.row_scale + row);
                ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, acc_phase, abort_flag));
                if (!ok)
                    break;
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * PN + half * 128;
                auto release = [&]() { // the accumulator is read: the next tile may have it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive_cluster(map_to_leader(tempty0 + 8 * acc));
                };
                auto scale32 = [&](const uint32_t (&r)[32], int col, float *v) {
                    if (scaled && p.col_scale && col < p.N) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float4 cs = __ldg((const float4 *)(p.col_scale + col) + i);
                            const float c4[4] = {cs.x * rs, cs.y * rs, cs.z * rs, cs.w * rs};
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                v[4 * i + e] = ((MMA == 2) ? (float)(int)r[4 * i + e] : __uint_as_float(r[4 * i + e])) * c4[e];
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            v[i] = ((MMA == 2) ? (float)(int)r[i] : __uint_as_float(r[i])) * rs;
                    }
                };
#pragma unroll 1
                for (int b = 0; b < 4; ++b) {
                    uint32_t r[32];
                    tmem_ld32(taddr + b * 32, r);
                    tmem_ld_wait();
                    if (b == 3)
                        release();
                    const int col = un.n0 + half * 128 + b * 32;
                    uint8_t *blk = stg + buf * 4096;
                    const int next_buf = buf == 2 ? 0 : buf + 1;
                    if (add) {
                        // the next block's residual input goes into the next buffer, whose last store but one has read it
                        if (lane == 0)
                            bulk_wait_read<1>();
                        if (b < 3)
                            fetch_cin(u, b + 1, next_buf);
                        else if (u + step < units)
                            fetch_cin(u + step, 0, next_buf);
                        ok = __all_sync(0xffffffffu, mbar_wait(cin_bar + 8 * buf, (cin_phase >> buf) & 1, abort_flag));
                        if (!ok)
                            break;
                        cin_phase ^= 1u << buf;
                    } else {
                        if (lane == 0)
                            bulk_wait_read<2>();
                        __syncwarp();
                    }
                    float v[32];
                    scale32(r, col, v);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        float4 *q = (float4 *)(blk + piece(lane, i));
                        float4 o = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                        if (add) {
                            const float4 c = *q;
                            o = make_float4(o.x + c.x, o.y + c.y, o.z + c.z, o.w + c.w);
                        }
                        *q = o;
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        if (partial)
                            tma_store_2d(&tmC, smem_u32(blk), half * 128 + b * 32, u * PM + (int)rank * 128 + quarter * 32);
                        else if (col < p.N)
                            tma_store_2d(&tmC, smem_u32(blk), col, m0 + quarter * 32);
                        bulk_commit();
                    }
                    buf = next_buf;
                }
                if (!ok)
                    break;
                acc ^= 1;
                if (acc == 0)
                    acc_phase ^= 1;
            }
            // abort path: a residual block may still be on its way into this CTA's shared memory
            if (!ok && add && lane == 0) {
                long long t0 = clock64();
                for (int i = 0; i < 3; ++i)
                    while (!mbar_try_wait(cin_bar + 8 * i, (cin_phase >> i) & 1) && clock64() - t0 < 200000000ll) {
                    }
            }
        }
        if (lane == 0)
            bulk_wait_read<0>(); // the staging blocks must outlive the stores that read them
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync(); // nothing of the peer refers to this CTA any more
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    if (threadIdx.x == 0 && *abort_flag)
        atomicOr(p.status, TS2_STATUS_WAIT_TIMEOUT);
}

template <int ES, int MMA, bool MN, int FORM>
int launch_pair(int device, cudaStream_t stream, int grid, const CUtensorMap &tmA, const CUtensorMap &tmB, const CUtensorMap &tmC,
                const CUtensorMap &tmCin, const CUtensorMap &tmX, const CUtensorMap &tmY, const GemmParams &p)
{
    auto kern = gemm_pair_kernel<ES, MMA, MN, FORM>;
    static bool configured[16] = {};
    if (!configured[device & 15]) {
        TS2_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PairSmem<FORM>::TOTAL));
        configured[device & 15] = true;
    }
    TS2_LAUNCH((kern), grid, epi8(FORM) ? P_THREADS : P_THREADS_16, PairSmem<FORM>::TOTAL, stream, tmA, tmB, tmC, tmCin, tmX, tmY, p);
    return TS2_OK;
}

} // namespace

int gemm_pair_launch(int device, cudaStream_t stream, int es, int mma, bool mn, PairForm form, int grid, const CUtensorMap &tmA,
                     const CUtensorMap &tmB, const CUtensorMap &tmC, const CUtensorMap &tmCin, const CUtensorMap &tmX, const CUtensorMap &tmY,
                     const GemmParams &p)
{
#define TS2_PAIR_CASE(ES_, MMA_, MN_, FORM_)                          \
    if (es == ES_ && mma == MMA_ && mn == MN_ && form == FORM_)       \
        return launch_pair<ES_, MMA_, MN_, FORM_>(device, stream, grid, tmA, tmB, tmC, tmCin, tmX, tmY, p);
#define TS2_PAIR_CASES(ES_, MMA_)              \
    TS2_PAIR_CASE(ES_, MMA_, false, P_F32)     \
    TS2_PAIR_CASE(ES_, MMA_, false, P_16)      \
    TS2_PAIR_CASE(ES_, MMA_, false, P_GATED)   \
    TS2_PAIR_CASE(ES_, MMA_, false, P_NORM)    \
    TS2_PAIR_CASE(ES_, MMA_, false, P_LSE)     \
    TS2_PAIR_CASE(ES_, MMA_, false, P_NORM_BWD) \
    TS2_PAIR_CASE(ES_, MMA_, true, P_F32)      \
    TS2_PAIR_CASE(ES_, MMA_, true, P_16)
    TS2_PAIR_CASES(1, 0)
    TS2_PAIR_CASE(1, 0, false, P_ACT_BWD)
    TS2_PAIR_CASE(1, 0, false, P_GATE_BWD)
    TS2_PAIR_CASES(2, 1)
    TS2_PAIR_CASES(1, 2)
#undef TS2_PAIR_CASES
#undef TS2_PAIR_CASE
    return fail(TS2_ERR_UNSUPPORTED, "gemm: unsupported configuration");
}

} // namespace ts2
