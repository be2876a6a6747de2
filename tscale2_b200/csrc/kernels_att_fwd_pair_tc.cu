// Attention forward for many nodes (head width 128, sm_100a): a CTA works on two blocks of 128 nodes of a head at a time.
// Same operands, results and rules as kernels_att_tc.cu (the zero "sink" vector is the initial state m = 0, l = 1; O is
// rescaled only where a row's maximum grew by more than 8), without its form that also applies the gate: the operator call
// (ts2_attention_forward) asks the rule below, the gated forward of training and scoring stays with the other kernel.
//
//   warp 0       TMA producer; draws the work items (pair of blocks, head) from a counter and finds their key ranges
//   warp 1       TMEM owner and MMA issuer: S_i = Q_i . K^T (128 x 128), O_i += P_i . V with P_i from tensor memory
//   warps 4-7    softmax of block 0, thread = row: 128 scores from TMEM into registers, maximum, exponentials and sum
//   warps 8-11   the same for block 1           without an exchange, P (fp16) back into TMEM where its scores were
// TMEM (512 columns): S_0, S_1 (P_i over S_i), O_0, O_1.  Shared memory: Q_0, Q_1, a ring of four 32 KB stages through which
// K and V tiles of 128 keys pass in the order K(0) V(0) K(1) V(1) ..; 4 KB of staging a warp.
// One CTA per SM; items run into each other: the next item's copies and first products go on while a block is written out.
//
// What bounds it: the exponentials, 16 a clock and SM: 1024 clocks per 128 x 128 scores, as much as the MMAs of four such
// tiles.  While one block's warps wait for their products the other block's compute.  Both kernels' times and where the line
// between them lies: attention_forward_takes_pairs.
// MMAs of one issuing thread complete in order: S_i(k + 1) is issued behind the product that reads P_i(k), over which it
// writes, and its completion tells the softmax that O_i is up to date.  Every wait is bounded; a give-up raises the status word.
#include "att_tc.cuh"

namespace ts2 {

namespace {

constexpr int FP_THREADS = 384;
constexpr int FP_TILE_BYTES = TC_BM * TC_HD * 2; // 32 KB: two 64-column atoms of 128 rows
constexpr int FP_STAGES = 4;
constexpr int FP_RING_OFF = 2 * FP_TILE_BYTES;
constexpr int FP_STG_OFF = FP_RING_OFF + FP_STAGES * FP_TILE_BYTES;
constexpr int FP_BAR_OFF = FP_STG_OFF + 8 * 4096;
constexpr int FP_SMEM = FP_BAR_OFF + 512;
static_assert(FP_SMEM <= 232448, "shared memory budget");
constexpr int FP_ITEMS = 4; // slots of the item ring

struct FwdPairParams {
    int T, H, n_pairs;
    const int *span_start, *span_finish;
    float *lse;
    int *counter; // {next item, finished CTAs}, zero between launches (the last CTA resets them)
    int32_t *status;
};

// key tiles of the two blocks: block i takes tiles [a[i], b[i]] (none: a > b), K and V are fetched for [ks, ke]
struct FwdItem {
    int pair, h, ks, ke, a[2], b[2];
};

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
                 "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
// two fp32 values in one register pair
__device__ __forceinline__ uint64_t f32x2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f32x2_split(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__global__ void __launch_bounds__(FP_THREADS, 1)
    att_fwd_pair_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                           const __grid_constant__ CUtensorMap tmO, const FwdPairParams p)
{
    extern __shared__ __align__(1024) uint8_t att_fp_smem[];
    uint8_t *smem = att_fp_smem;
    if (smem_u32(smem) & 1023) { // the swizzled tiles need a 1024-byte aligned base; refuse instead of computing garbage
        if (threadIdx.x == 0)
            atomicOr(p.status, TS2_STATUS_BAD_ARG);
        return;
    }
    const uint32_t sQ = smem_u32(smem), sRing = sQ + FP_RING_OFF;
    uint64_t *bars = (uint64_t *)(smem + FP_BAR_OFF);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + 4), q_full0 = smem_u32(bars + 8), q_empty0 = smem_u32(bars + 10),
                   s_full0 = smem_u32(bars + 12), p_full0 = smem_u32(bars + 14), o_full0 = smem_u32(bars + 16), o_free0 = smem_u32(bars + 18),
                   rfull0 = smem_u32(bars + 20), rempty0 = smem_u32(bars + 24);
    uint32_t *tmem_slot = (uint32_t *)(bars + 28);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    volatile FwdItem *items = (volatile FwdItem *)(bars + 30); // [FP_ITEMS], 32 bytes each

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < FP_STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(q_full0 + 8 * i, 1);
            mbar_init(q_empty0 + 8 * i, 1);
            mbar_init(s_full0 + 8 * i, 1);
            mbar_init(p_full0 + 8 * i, 4);
            mbar_init(o_full0 + 8 * i, 1);
            mbar_init(o_free0 + 8 * i, 4);
        }
        for (int s = 0; s < FP_ITEMS; ++s) {
            mbar_init(rfull0 + 8 * s, 1);
            mbar_init(rempty0 + 8 * s, 1 + 8);
        }
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmQ);
        prefetch_tmap(&tmK);
        prefetch_tmap(&tmV);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_wait();
    const uint32_t tmem = *tmem_slot;
    const int n_items = p.n_pairs * p.H;
    int rslot = 0;
    uint32_t rphase = 0;
    auto step_ring = [&]() {
        if (++rslot == FP_ITEMS) {
            rslot = 0;
            rphase ^= 1;
        }
    };

    // The softmax warps hold a row's 128 scores: they take registers over from the other four warps.  The launch gives 384 x 168;
    // 128 x 72 + 256 x 216 is as much.
    static_assert(FP_THREADS * 168 == 128 * 72 + 256 * 216, "registers of the block");
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        if (warp == 0) {
            // ------------------------------ TMA producer ------------------------------
            int next = lane == 0 ? atomicAdd(p.counter, 1) : 0;
            bool ok = true;
            uint32_t seq = 0, kv_phase = 0xf, q_phase = 3; // phase bits: per stage, per block; the first wait on a fresh barrier passes
            uint32_t q_used = 0; // blocks whose queries were ever copied
            while (ok) {
                next = __shfl_sync(0xffffffffu, next, 0);
                FwdItem it;
                it.pair = -1;
                if (next < n_items) {
                    // the later blocks of a sequence have the most keys: they come first
                    it.pair = p.n_pairs - 1 - next / p.H;
                    it.h = next % p.H;
                    it.ks = 0x7fffffff;
                    it.ke = -1;
    #pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        int lo = 0x7fffffff, hi = -1;
    #pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int t = it.pair * 256 + i * 128 + j * 32 + lane;
                            if (t < p.T) {
                                const int st = p.span_start[t], fi = p.span_finish[t];
                                if (fi >= st) {
                                    lo = min(lo, st);
                                    hi = max(hi, fi);
                                }
                            }
                        }
                        lo = __reduce_min_sync(0xffffffffu, lo);
                        hi = __reduce_max_sync(0xffffffffu, hi);
                        it.a[i] = hi >= 0 ? max(lo, 0) / TC_BM : 1; // a span may start before the first key
                        it.b[i] = hi >= 0 ? hi / TC_BM : 0;
                        if (hi >= 0) {
                            it.ks = min(it.ks, it.a[i]);
                            it.ke = max(it.ke, it.b[i]);
                        }
                    }
                    if (it.ke < 0)
                        it.ks = 0;
                }
                if (lane == 0) {
                    ok = mbar_wait(rempty0 + 8 * rslot, rphase ^ 1, abort_flag);
                    if (ok) {
                        volatile FwdItem &s = items[rslot];
                        s.pair = it.pair;
                        s.h = it.h;
                        s.ks = it.ks;
                        s.ke = it.ke;
                        s.a[0] = it.a[0], s.a[1] = it.a[1], s.b[0] = it.b[0], s.b[1] = it.b[1];
                        mbar_arrive(rfull0 + 8 * rslot);
                    }
                }
                step_ring();
                if (it.pair < 0)
                    break;
                if (lane == 0 && ok) {
                    next = atomicAdd(p.counter, 1); // its latency hides behind this item's copies
                    const int col0 = it.h * TC_HD, r0 = it.pair * 256, nk = it.ke - it.ks + 1;
                    auto load_q = [&](int i) {
                        if (it.a[i] > it.b[i])
                            return true;
                        if (!mbar_wait(q_empty0 + 8 * i, (q_phase >> i) & 1, abort_flag))
                            return false;
                        q_phase ^= 1u << i;
                        q_used |= 1u << i;
                        mbar_arrive_expect_tx(q_full0 + 8 * i, FP_TILE_BYTES);
                        tma_load_2d(sQ + i * FP_TILE_BYTES, &tmQ, q_full0 + 8 * i, col0, r0 + i * 128);
                        tma_load_2d(sQ + i * FP_TILE_BYTES + FP_TILE_BYTES / 2, &tmQ, q_full0 + 8 * i, col0 + 64, r0 + i * 128);
                        return true;
                    };
                    auto load = [&](const CUtensorMap *tm, int row) {
                        const int st = seq & (FP_STAGES - 1);
                        if (!mbar_wait(empty0 + 8 * st, (kv_phase >> st) & 1, abort_flag))
                            return false;
                        kv_phase ^= 1u << st;
                        const uint32_t dst = sRing + st * FP_TILE_BYTES, fb = full0 + 8 * st;
                        mbar_arrive_expect_tx(fb, FP_TILE_BYTES);
                        tma_load_2d(dst, tm, fb, col0, row);
                        tma_load_2d(dst + FP_TILE_BYTES / 2, tm, fb, col0 + 64, row);
                        ++seq;
                        return true;
                    };
                    ok = load_q(0) && load_q(1);
                    for (int k = 0; k < 2 * nk && ok; ++k)
                        ok = load(k & 1 ? &tmV : &tmK, (it.ks + (k >> 1)) * TC_BM);
                }
                ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
            }
            if (lane == 0) {
                if (*abort_flag) { // copies in flight must land before the CTA gives its shared memory back (bounded)
                    const long long c0 = clock64();
                    for (int st = 0; st < FP_STAGES; ++st) // kv_phase: parity of the next wait on empty, and of the last copy's phase on full
                        while (seq > (uint32_t)st && !mbar_try_wait(full0 + 8 * st, (kv_phase >> st) & 1) && clock64() - c0 < 200000000ll) {
                        }
                    for (int i = 0; i < 2; ++i) // q_phase holds the parity of the next wait on q_empty, that of the last copy is its inverse ^ 1
                        while (((q_used >> i) & 1) && !mbar_try_wait(q_full0 + 8 * i, (q_phase >> i) & 1) && clock64() - c0 < 200000000ll) {
                        }
                }
                // every CTA passes here once, after its last draw
                if (atomicAdd(p.counter + 1, 1) == (int)gridDim.x - 1) {
                    p.counter[0] = 0;
                    p.counter[1] = 0;
                }
            }
        } else if (warp == 1) {
            // ------------------------------ MMA issuer --------------------------------
            if (lane == 0) {
                constexpr uint32_t idesc_qk = umma_idesc_f16(TC_BM, false, false), idesc_pv = umma_idesc_f16(TC_HD, false, true);
                uint32_t seq = 0, p_phase = 0, q_phase = 0, free_phase = 3, full_phase = 0; // full_phase: a bit per stage
                bool ok = true;
                while (ok) {
                    if (!mbar_wait(rfull0 + 8 * rslot, rphase, abort_flag))
                        break;
                    FwdItem it;
                    it.pair = items[rslot].pair, it.ks = items[rslot].ks, it.ke = items[rslot].ke;
                    it.a[0] = items[rslot].a[0], it.a[1] = items[rslot].a[1], it.b[0] = items[rslot].b[0], it.b[1] = items[rslot].b[1];
                    mbar_arrive(rempty0 + 8 * rslot);
                    step_ring();
                    if (it.pair < 0)
                        break;
                    for (int k = it.ks - 1; k <= it.ke && ok; ++k) {
                        const uint32_t nv = seq + 2 * (uint32_t)(k - it.ks) + 1, nk = nv + 1; // ring numbers of V(k), K(k + 1)
                        const int sv = nv & (FP_STAGES - 1), sk = nk & (FP_STAGES - 1);
    #pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint32_t tS = tmem + i * 128, tO = tmem + 256 + i * 128;
                            if (ok && k >= it.a[i] && k <= it.b[i]) { // O_i += P_i(k) . V(k)
                                ok = (k > it.a[i] || mbar_wait(o_free0 + 8 * i, (free_phase >> i) & 1, abort_flag)) &&
                                     mbar_wait(full0 + 8 * sv, (full_phase >> sv) & 1, abort_flag) && mbar_wait(p_full0 + 8 * i, (p_phase >> i) & 1, abort_flag);
                                if (!ok)
                                    break;
                                if (k == it.a[i])
                                    free_phase ^= 1u << i;
                                p_phase ^= 1u << i;
                                tc_fence_after();
                                const uint64_t dv = umma_smem_desc(sRing + sv * FP_TILE_BYTES, FP_TILE_BYTES / 2, 1024);
    #pragma unroll
                                for (int kk = 0; kk < 8; ++kk) // 16 keys = 8 columns of P, 16 rows of V
                                    umma_f16_ts(tO, tS + 8 * kk, dv + (uint64_t)(kk * 128), idesc_pv, (k > it.a[i] || kk > 0) ? 1u : 0u);
                                if (k == it.b[i])
                                    tc_commit(o_full0 + 8 * i);
                            }
                            if (ok && k + 1 >= it.a[i] && k + 1 <= it.b[i]) { // S_i(k + 1) = Q_i . K(k + 1)^T
                                ok = (k + 1 > it.a[i] || mbar_wait(q_full0 + 8 * i, (q_phase >> i) & 1, abort_flag)) &&
                                     mbar_wait(full0 + 8 * sk, (full_phase >> sk) & 1, abort_flag);
                                if (!ok)
                                    break;
                                if (k + 1 == it.a[i])
                                    q_phase ^= 1u << i;
                                tc_fence_after();
                                const uint64_t dq = umma_smem_desc(sQ + i * FP_TILE_BYTES, 16, 1024), dk = umma_smem_desc(sRing + sk * FP_TILE_BYTES, 16, 1024);
                                umma_f16_x4(tS, dq, dk, idesc_qk, 0u, 2u, 2u);
                                umma_f16_x4(tS, dq + (FP_TILE_BYTES / 2 >> 4), dk + (FP_TILE_BYTES / 2 >> 4), idesc_qk, 1u, 2u, 2u);
                                tc_commit(s_full0 + 8 * i);
                                if (k + 1 == it.b[i])
                                    tc_commit(q_empty0 + 8 * i);
                            }
                        }
                        if (!ok)
                            break;
                        // also for a tile neither block took: it must have landed before its stage is filled again
                        if (k >= it.ks) {
                            if (!(ok = mbar_wait(full0 + 8 * sv, (full_phase >> sv) & 1, abort_flag)))
                                break;
                            full_phase ^= 1u << sv;
                            tc_commit(empty0 + 8 * sv);
                        }
                        if (k < it.ke) {
                            if (!(ok = mbar_wait(full0 + 8 * sk, (full_phase >> sk) & 1, abort_flag)))
                                break;
                            full_phase ^= 1u << sk;
                            tc_commit(empty0 + 8 * sk);
                        }
                    }
                    seq += 2 * (uint32_t)(it.ke - it.ks + 1);
                }
            }
        }
    } else {
        // ------------------------------ softmax warps -----------------------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        const int grp = (warp - 4) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16, tS = tmem + grp * 128 + lane_addr, tO = tmem + 256 + grp * 128 + lane_addr;
        const uint32_t s_full = s_full0 + 8 * grp, p_full = p_full0 + 8 * grp, o_full = o_full0 + 8 * grp, o_free = o_free0 + 8 * grp;
        const float ds = att_dot_scale_tc();
        uint8_t *const stg = smem + FP_STG_OFF + (warp - 4) * 4096, *const srow = stg + lane * 128;
        uint32_t s_phase = 0, o_phase = 0;
        bool ok = true;
        while (ok) {
            ok = __all_sync(0xffffffffu, mbar_wait(rfull0 + 8 * rslot, rphase, abort_flag));
            if (!ok)
                break;
            const int pair = items[rslot].pair, h = items[rslot].h, ks = items[rslot].ks, ke = items[rslot].ke, ka = items[rslot].a[grp],
                      kb = items[rslot].b[grp];
            __syncwarp();
            if (lane == 0)
                mbar_arrive(rempty0 + 8 * rslot);
            step_ring();
            if (pair < 0)
                break;
            const int r0 = pair * 256 + grp * 128, t = r0 + row;
            const int st_row = t < p.T ? p.span_start[t] : 0, fi_row = t < p.T ? p.span_finish[t] : -1;
            float m_used = 0.f, l = 1.f; // the zero vector of weight 2^-m
            for (int k = ka; k <= kb; ++k) {
                ok = __all_sync(0xffffffffu, mbar_wait(s_full, s_phase, abort_flag));
                if (!ok)
                    break;
                s_phase ^= 1;
                tc_fence_after();
                uint32_t s[4][32];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    tmem_ld32(tS + c * 32, s[c]);
                tmem_ld_wait();
                const int key0 = k * TC_BM;
                const bool plain = __all_sync(0xffffffffu, key0 >= st_row && key0 + TC_BM - 1 <= fi_row);
                float mx;
                if (plain) { // the scores stay raw products and the scale rides in the exponent's fma
                    float r4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int i = 0; i < 32; i += 2)
                            r4[c] = fmaxf(r4[c], fmaxf(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])));
                    mx = fmaxf(fmaxf(r4[0], r4[1]), fmaxf(r4[2], r4[3])) * ds;
                } else {
                    float r4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const int key = key0 + c * 32 + i;
                            const float x = (key >= st_row && key <= fi_row) ? __uint_as_float(s[c][i]) * ds : -INFINITY;
                            s[c][i] = __float_as_uint(x);
                            r4[i & 3] = fmaxf(r4[i & 3], x);
                        }
                    mx = fmaxf(fmaxf(r4[0], r4[1]), fmaxf(r4[2], r4[3]));
                }
                const bool need = mx > m_used + 8.f;
                const bool warp_need = __any_sync(0xffffffffu, need);
                float rs = 1.f;
                if (need) {
                    rs = exp2f(m_used - mx);
                    m_used = mx;
                    l *= rs;
                }
                const float es = plain ? ds : 1.f;
                const uint64_t es2 = f32x2(es, es), nm2 = f32x2(-m_used, -m_used);
                uint64_t sum2[2] = {0ull, 0ull};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t pk[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float e0, e1;
                        f32x2_split(fma_f32x2(f32x2(__uint_as_float(s[c][2 * i]), __uint_as_float(s[c][2 * i + 1])), es2, nm2), e0, e1);
                        asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e0));
                        asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e1));
                        sum2[i & 1] = add_f32x2(sum2[i & 1], f32x2(e0, e1));
                        pk[i] = bits_from_h2(sat_half2(e0, e1));
                    }
                    tmem_st16(tS + c * 16, pk); // over scores this thread has read
                }
                float a0, a1;
                f32x2_split(add_f32x2(sum2[0], sum2[1]), a0, a1);
                l += a0 + a1;
                if (warp_need && k > ka) {
                    // every product so far is in O: S(k) was issued behind the last of them
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t r[32];
                        tmem_ld32(tO + c * 32, r);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            r[i] = __float_as_uint(__uint_as_float(r[i]) * rs);
                        tmem_st32(tO + c * 32, r);
                    }
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(p_full);
            }
            if (!ok)
                break;
            // epilogue: O / l and lse.  A warp's 32 rows in two halves of 64 columns through the warp's staging block: rows of 128
            // bytes with the 128-byte swizzle and TMA stores, which clip rows past T.
            const bool any = ka <= kb;
            if (any) {
                ok = __all_sync(0xffffffffu, mbar_wait(o_full, o_phase, abort_flag));
                if (!ok)
                    break;
                o_phase ^= 1;
                tc_fence_after();
            }
            const float inv = 1.f / l;
            const bool rows = r0 + quarter * 32 < p.T; // the warp has a row
            const int c0 = h * TC_HD;
#pragma unroll 1
            for (int hb = 0; hb < 2; ++hb) {
                if (lane == 0)
                    bulk_wait_read<0>(); // the staging block's last store has read it
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    uint32_t r[32];
                    if (any) {
                        tmem_ld32(tO + hb * 64 + q * 32, r);
                        tmem_ld_wait();
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            r[i] = 0u;
                    }
                    if (hb == 1 && q == 1 && any) { // O is read: the next item may have it
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0)
                            mbar_arrive(o_free);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const __half2 h0 = sat_half2(__uint_as_float(r[8 * i]) * inv, __uint_as_float(r[8 * i + 1]) * inv),
                                      h1 = sat_half2(__uint_as_float(r[8 * i + 2]) * inv, __uint_as_float(r[8 * i + 3]) * inv),
                                      h2 = sat_half2(__uint_as_float(r[8 * i + 4]) * inv, __uint_as_float(r[8 * i + 5]) * inv),
                                      h3 = sat_half2(__uint_as_float(r[8 * i + 6]) * inv, __uint_as_float(r[8 * i + 7]) * inv);
                        const uint4 o8 = make_uint4(bits_from_h2(h0), bits_from_h2(h1), bits_from_h2(h2), bits_from_h2(h3));
                        *(uint4 *)(srow + (((q * 4 + i) ^ (lane & 7)) << 4)) = o8;
                    }
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    if (rows)
                        tma_store_2d(&tmO, smem_u32(stg), c0 + hb * 64, r0 + quarter * 32);
                    bulk_commit();
                }
            }
            if (t < p.T)
                p.lse[(size_t)t * p.H + h] = m_used + log2f(l);
        }
        if (lane == 0)
            bulk_wait_read<0>(); // shared memory must outlive the stores that read it
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1)
        tmem_dealloc(tmem, 512);
    if (threadIdx.x == 0 && *abort_flag)
        atomicOr(p.status, TS2_STATUS_WAIT_TIMEOUT);
}

} // namespace

// Long causal sequences that start on tiles.  Whole calls, one block per CTA and two CTAs an SM (kernels_att_tc.cu) -> pairs, us:
//   4 x 4096 x 16 heads 418 -> 359, 4 x 4096 x 7 234 -> 206, 2 x 4096 x 14 235 -> 200; 3072 nodes, the shortest, 4 x 3072 x 16
//   forward and backward 907 -> 876, 4 x 3072 x 10 628 -> 616;
//   spans of 1024 keys on average (8 x 2048 x 16) 252 -> 253, shorter ones lose (16 x 1024 x 12 141 -> 147): an item's start and
//   end, which a second CTA on the SM hides;
//   sequences that start inside a tile 4 x 3000 x 16 296 -> 296, 5 x 3333 x 9 282 -> 296: more tiles need the mask, and a pair waits
//   for its slower block;
//   with a slope 4 x 4096 x 16 579 -> 595: its arithmetic, not the chain of hand-overs, is what the softmax warps then do;
//   few items 8 x 2048 x 4 110 -> 120, 1 x 4096 x 4 96 -> 108: less than three an SM leave a ragged end.
// Two nodes of a block are looked at, which is exact for causal sequences that start on tiles: a call waits for its kernel, so what
// the host does in front of it is added to it (all nodes: 64 x 1024 x 12 422 -> 454, 64 x 256 x 16 104 -> 110, two of 128 422 and 104).
bool attention_forward_takes_pairs(int device, const int *span_start, const int *span_finish, int T, int H, float slope)
{
    if (slope != 0.f || ceil_div(T, 2 * TC_BM) * H < 3ll * sm_count(device))
        return false;
    long long keys2 = 0; // twice the keys, from the first and the last node of each block
    for (int t0 = 0; t0 < T; t0 += TC_BM) {
        const int n = std::min(TC_BM, T - t0);
        for (int t : {t0, t0 + n - 1})
            if (span_finish[t] >= span_start[t]) {
                if (span_start[t] % (2 * TC_BM) != 0)
                    return false;
                keys2 += (long long)n * (span_finish[t] - span_start[t] + 1);
            }
    }
    return keys2 >= 3071ll * T; // what a causal sequence of 3072 nodes has
}

int attention_forward_pair_tc(const Ctx &c, const __half *q, const __half *k, const __half *v, const int *span_start, const int *span_finish,
                              int T, int H, __half *o, float *lse, int *counter)
{
    static bool configured[16] = {};
    if (!configured[c.device & 15]) {
        TS2_CUDA(cudaFuncSetAttribute(att_fwd_pair_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FP_SMEM));
        configured[c.device & 15] = true;
    }
    const int Q = H * TC_HD;
    CUtensorMap tmQ, tmK, tmV, tmO;
    int rc;
    if ((rc = make_tensor_map(&tmQ, q, 2, Q, T, Q, TC_BM)) != TS2_OK || (rc = make_tensor_map(&tmK, k, 2, Q, T, Q, TC_BM)) != TS2_OK ||
        (rc = make_tensor_map(&tmV, v, 2, Q, T, Q, TC_BM)) != TS2_OK || (rc = make_tensor_map(&tmO, o, 2, Q, T, Q, 32)) != TS2_OK)
        return rc;
    FwdPairParams p;
    p.T = T;
    p.H = H;
    p.n_pairs = (int)ceil_div(T, 2 * TC_BM);
    p.span_start = span_start;
    p.span_finish = span_finish;
    p.lse = lse;
    p.counter = counter;
    p.status = device_status_word(c.device);
    if (!p.status)
        return fail(TS2_ERR_CUDA, "attention: no device status word");
    const int grid = (int)std::min<long long>((long long)p.n_pairs * H, sm_count(c.device));
    TS2_LAUNCH((att_fwd_pair_tc_kernel), grid, FP_THREADS, FP_SMEM, c.stream, tmQ, tmK, tmV, tmO, p);
    return TS2_OK;
}

} // namespace ts2
