// tcgen05 attention backward, dK, dV and the score gradients dS (head width 128, sm_100a); dQ = dS . K follows in
// kernels_att_bwd_dq_tc.cu.  References: src/gpt/compute/layer_att_reference.h:41-212, gpu_att_fp16.cu / .cuh, which
// recompute S = K . Q^T and dP = V . dO^T for dQ, dK and dV each.
//
// Work items are (block of 128 keys, head).  One CTA per SM takes items from a counter and keeps K and V of its item in
// shared memory while 64-node tiles of Q and dO stream through a ring that runs on across items:
//   S^T  = K . Q^T,  dP^T = V . dO^T          128 x 64 each, fp32, into one of TWO S / dP buffer pairs in TMEM
//   compute: P^T = 2^(S^T ds - lse) masked (fp16, back into TMEM);  dS^T = P^T (dP^T - dscale) c2 (fp16, shared memory)
//   dV += P^T . dO (P^T the TMEM A operand),  dK += dS^T . Q (dS^T the shared-memory A operand);  dS^T -> global memory
// TMEM (512 columns): pair 0 = S [0,64) dP [64,128); dK [128,256); dV [256,384); pair 1 = S [384,448) dP [448,512).
// 20 warps: TMA producer (and item counter), issuer of the first products, issuer of the accumulating products, store of
// dS, and 16 compute warps in two groups of 8, one per S / dP pair: while one group waits for its products, loads and
// stores tensor memory or arrives at a barrier, the other computes.
//
// What bounds it: before, one CTA per item with one group of 16 warps took 2850 clocks per 128 x 64 tile against about 1280
// that its MMAs take (S and dP are bound by the shared-memory reads of N = 64, 48 clocks per K step), and some 8000 clocks
// per item for its start and end; and dQ recomputed S, dP and the exponentials in a kernel as long.  Here dS costs its
// bytes once out and once in.  S and dP are handed over one by one, and so are P and dS: the exponentials run while dP is still
// being multiplied, dV's product while dS is computed (64 x 1024 nodes, 12 heads 601 -> 573 us, 8 x 2048, 4 heads 124 -> 115).
//
// Everything that is handed over once per tile has one barrier per S / dP pair: the next phase of a pair's barrier belongs
// to the tile two further on, which cannot start before the waiter of this phase has acted, so a parity test can never
// miss a phase.  Every wait is bounded; a give-up raises the status word.
#include "att_tc.cuh"
#include <type_traits>

namespace ts2 {

namespace {

constexpr int KV_THREADS = 640;
constexpr int KV_STAGES = 3;
constexpr int KV_STAGE_BYTES = 2 * KV_BYTES; // Q tile + dO tile, 64 rows each
constexpr int KV_G_BYTES = TC_BM * TC_BN * 2; // one dS^T tile
constexpr int KV_META_BYTES = ATT_NODE_BYTES + ATT_SPAN_BYTES;
constexpr int KV_STAGE_OFF = 2 * Q_BYTES;
constexpr int KV_G_OFF = KV_STAGE_OFF + KV_STAGES * KV_STAGE_BYTES;
constexpr int KV_META_OFF = KV_G_OFF + 2 * KV_G_BYTES;
constexpr int KV_BAR_OFF = KV_META_OFF + KV_STAGES * KV_META_BYTES;
constexpr int KV_SMEM = KV_BAR_OFF + 512;
static_assert(KV_SMEM <= 232448 && KV_BAR_OFF % 16 == 0, "shared memory budget");
constexpr int KV_RING = 4;

struct AttBwdKvParams {
    int T, H, Tpad, n_blocks;
    float slope;
    const float2 *meta;      // [H][Tpad]: {-lse, -dscale * c2} per node
    const uint8_t *spans;    // [Tpad / 64][ATT_SPAN_BYTES]
    const int4 *blocks;      // [n_blocks + 1]: see att_layout
    int *counter;            // next item, zero when the kernel starts
    uint8_t *ds;             // dS tiles, null: not wanted
    int ds_tiles;            // capacity
    int32_t *status;
};

// 16-byte piece c of row r of a tile with 128-byte rows in the 128-byte swizzle
__device__ __forceinline__ uint32_t piece128(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

// OUT16: dK and dV are written as fp16 (what the engine feeds its next kernel with) instead of fp32
template <bool OUT16>
__global__ void __launch_bounds__(KV_THREADS, 1)
    att_bwd_kv_tc_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                         const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                         const __grid_constant__ CUtensorMap tmDK, const __grid_constant__ CUtensorMap tmDV, const AttBwdKvParams p)
{
    extern __shared__ __align__(1024) uint8_t att_kv_smem[];
    uint8_t *smem = att_kv_smem;
    if (smem_u32(smem) & 1023) { // the swizzled tiles need a 1024-byte aligned base; refuse instead of computing garbage
        if (threadIdx.x == 0)
            atomicOr(p.status, TS2_STATUS_BAD_ARG);
        return;
    }
    const uint32_t sK = smem_u32(smem), sV = sK + Q_BYTES, sStage = sK + KV_STAGE_OFF, sG = sK + KV_G_OFF, sMeta = sK + KV_META_OFF;
    uint64_t *bars = (uint64_t *)(smem + KV_BAR_OFF);
    const uint32_t kv_full = smem_u32(bars), kv_empty = smem_u32(bars + 1), st_full0 = smem_u32(bars + 2), st_empty0 = smem_u32(bars + 5),
                   s_full0 = smem_u32(bars + 8), pair_free0 = smem_u32(bars + 10), g_full0 = smem_u32(bars + 12), g_free0 = smem_u32(bars + 14),
                   acc_done = smem_u32(bars + 16), acc_free = smem_u32(bars + 17), rfull0 = smem_u32(bars + 18), rempty0 = smem_u32(bars + 22),
                   mate0 = smem_u32(bars + 26), // [8]: the two warps that share a group's lane quarter
                   dp_full0 = smem_u32(bars + 34), p_full0 = smem_u32(bars + 36);
    uint32_t *tmem_slot = (uint32_t *)(bars + 38);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    volatile int *ring = (volatile int *)(tmem_slot + 2); // [KV_RING] item numbers, -1 = no more

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
    }
    if (threadIdx.x == 0) {
        mbar_init(kv_full, 1);
        mbar_init(kv_empty, 1);
        for (int s = 0; s < KV_STAGES; ++s) {
            mbar_init(st_full0 + 8 * s, 1);
            mbar_init(st_empty0 + 8 * s, 1);
        }
        for (int g = 0; g < 2; ++g) {
            mbar_init(s_full0 + 8 * g, 1);
            mbar_init(pair_free0 + 8 * g, 1);
            mbar_init(dp_full0 + 8 * g, 1);
            mbar_init(p_full0 + 8 * g, 8);
            mbar_init(g_full0 + 8 * g, 8);
            mbar_init(g_free0 + 8 * g, 2); // the MMAs that read the tile, and its store
        }
        mbar_init(acc_done, 1);
        mbar_init(acc_free, 16);
        for (int s = 0; s < KV_RING; ++s) {
            mbar_init(rfull0 + 8 * s, 1);
            mbar_init(rempty0 + 8 * s, 3 + 16);
        }
        for (int i = 0; i < 8; ++i)
            mbar_init(mate0 + 8 * i, 2);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmK);
        prefetch_tmap(&tmV);
        prefetch_tmap(&tmQ);
        prefetch_tmap(&tmDO);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tDK = tmem_base + 128, tDV = tmem_base + 256;
    const int n_items = p.n_blocks * p.H;

    // the next item of this CTA (-1: none, -2: a wait ran out)
    int rslot = 0;
    uint32_t rphase = 0;
    auto next_item = [&](bool leader) {
        if (!mbar_wait(rfull0 + 8 * rslot, rphase, abort_flag))
            return -2;
        const int item = ring[rslot];
        if (leader)
            mbar_arrive(rempty0 + 8 * rslot);
        if (++rslot == KV_RING) {
            rslot = 0;
            rphase ^= 1;
        }
        return item;
    };

    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            bool ok = true;
            int gt = 0, live = 0; // tiles so far; items with tiles so far
            int next = atomicAdd(p.counter, 1);
            while (ok) {
                const int item = next < n_items ? next : -1;
                if (!mbar_wait(rempty0 + 8 * rslot, rphase ^ 1, abort_flag))
                    break;
                ring[rslot] = item;
                mbar_arrive(rfull0 + 8 * rslot);
                if (++rslot == KV_RING) {
                    rslot = 0;
                    rphase ^= 1;
                }
                if (item < 0)
                    break;
                next = atomicAdd(p.counter, 1); // its latency hides behind this item's copies
                const int h = item / p.n_blocks, kb = item - h * p.n_blocks, col0 = h * TC_HD;
                const int4 tb = p.blocks[kb];
                if (tb.y == 0)
                    continue;
                if (!(ok = mbar_wait(kv_empty, (live & 1) ^ 1, abort_flag)))
                    break;
                ++live;
                mbar_arrive_expect_tx(kv_full, 2 * Q_BYTES);
                tma_load_2d(sK, &tmK, kv_full, col0, kb * TC_BM);
                tma_load_2d(sK + Q_BYTES / 2, &tmK, kv_full, col0 + 64, kb * TC_BM);
                tma_load_2d(sV, &tmV, kv_full, col0, kb * TC_BM);
                tma_load_2d(sV + Q_BYTES / 2, &tmV, kv_full, col0 + 64, kb * TC_BM);
                for (int j = 0; j < tb.y; ++j, ++gt) {
                    const int st = gt % KV_STAGES, tile = tb.x + j;
                    if (!(ok = mbar_wait(st_empty0 + 8 * st, ((gt / KV_STAGES) & 1) ^ 1, abort_flag)))
                        break;
                    const uint32_t fb = st_full0 + 8 * st, dq = sStage + st * KV_STAGE_BYTES, dd = dq + KV_BYTES, dm = sMeta + st * KV_META_BYTES;
                    mbar_arrive_expect_tx(fb, KV_STAGE_BYTES + KV_META_BYTES);
                    tma_load_2d(dq, &tmQ, fb, col0, tile * TC_BN);
                    tma_load_2d(dq + KV_BYTES / 2, &tmQ, fb, col0 + 64, tile * TC_BN);
                    tma_load_2d(dd, &tmDO, fb, col0, tile * TC_BN);
                    tma_load_2d(dd + KV_BYTES / 2, &tmDO, fb, col0 + 64, tile * TC_BN);
                    bulk_load(dm, p.meta + (size_t)h * p.Tpad + tile * TC_BN, ATT_NODE_BYTES, fb);
                    bulk_load(dm + ATT_NODE_BYTES, p.spans + (size_t)tile * ATT_SPAN_BYTES, ATT_SPAN_BYTES, fb);
                }
            }
            if (*abort_flag) { // copies in flight must land before the CTA gives its shared memory back (bounded)
                const long long t0 = clock64();
                for (int i = max(0, gt - KV_STAGES); i < gt; ++i)
                    while (!mbar_try_wait(st_full0 + 8 * (i % KV_STAGES), (i / KV_STAGES) & 1) && clock64() - t0 < 200000000ll) {
                    }
                while (live > 0 && !mbar_try_wait(kv_full, (live - 1) & 1) && clock64() - t0 < 200000000ll) {
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer A: S^T and dP^T ----------------
        // Two issuing threads on two schedulers: a thread is held for about as long as the MMAs it issues run, and while the
        // compute warps are busy its instructions wait for issue slots.  This one runs ahead with the first products;
        // issuer B (warp 2) follows the compute warps with the accumulating ones.
        if (lane == 0) {
            constexpr uint32_t idesc_s = umma_idesc_f16(TC_BN, false, false);
            const uint64_t dK = umma_smem_desc(sK, 16, 1024), dV = umma_smem_desc(sV, 16, 1024);
            int gt = 0, live = 0;
            bool ok = true;
            while (ok) {
                const int item = next_item(true);
                if (item < 0)
                    break;
                const int n = p.blocks[item % p.n_blocks].y;
                if (n == 0)
                    continue;
                ok = mbar_wait(kv_full, live & 1, abort_flag);
                ++live;
                for (int j = 0; j < n && ok; ++j, ++gt) { // S^T and dP^T of tile gt into pair gt & 1
                    // the pair's S block held P of tile gt - 2: the MMAs that read it must be complete before these write there
                    const int st = gt % KV_STAGES;
                    if ((gt >= 2 && !mbar_wait(pair_free0 + 8 * (gt & 1), ((gt - 2) >> 1) & 1, abort_flag)) ||
                        !mbar_wait(st_full0 + 8 * st, (gt / KV_STAGES) & 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t bq = sStage + st * KV_STAGE_BYTES, bd = bq + KV_BYTES;
                    const uint64_t dQ = umma_smem_desc(bq, 16, 1024), dD = umma_smem_desc(bd, 16, 1024);
                    const uint32_t tS = tmem_base + ((gt & 1) ? 384 : 0), tDP = tS + TC_BN;
                    // 8 steps of 16 head dims; operands are two 64-dim atoms each
                    umma_f16_x4(tS, dK, dQ, idesc_s, 0u, 2u, 2u);
                    umma_f16_x4(tS, dK + (Q_BYTES / 2 >> 4), dQ + (KV_BYTES / 2 >> 4), idesc_s, 1u, 2u, 2u);
                    tc_commit(s_full0 + 8 * (gt & 1));
                    // its dP block was last read by the compute warps on their way to dS of tile gt - 2
                    if (gt >= 2 && !mbar_wait(g_full0 + 8 * (gt & 1), ((gt - 2) >> 1) & 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    umma_f16_x4(tDP, dV, dD, idesc_s, 0u, 2u, 2u);
                    umma_f16_x4(tDP, dV + (Q_BYTES / 2 >> 4), dD + (KV_BYTES / 2 >> 4), idesc_s, 1u, 2u, 2u);
                    tc_commit(dp_full0 + 8 * (gt & 1));
                    if (j == n - 1)
                        tc_commit(kv_empty); // the next item's K and V may come in
                }
            }
        }
    } else if (warp == 2) {
        // ------------------------------ MMA issuer B: dV and dK -------------------
        if (lane == 0) {
            constexpr uint32_t idesc_acc = umma_idesc_f16(TC_HD, false, true);
            int gt = 0, live = 0;
            bool ok = true;
            while (ok) {
                const int item = next_item(true);
                if (item < 0)
                    break;
                const int n = p.blocks[item % p.n_blocks].y;
                if (n == 0)
                    continue;
                // the compute warps have read the previous item's accumulators
                ok = mbar_wait(acc_free, (live & 1) ^ 1, abort_flag);
                ++live;
                for (int j = 0; j < n && ok; ++j, ++gt) {
                    const int st = gt % KV_STAGES, pr = gt & 1;
                    if (!mbar_wait(p_full0 + 8 * pr, (gt >> 1) & 1, abort_flag) || !mbar_wait(st_full0 + 8 * st, (gt / KV_STAGES) & 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    // dV += P^T . dO, dK += dS^T . Q: 4 steps of 16 nodes.  P^T from tensor memory (16 nodes as 8 columns of fp16
                    // pairs at column 16 kk of the S block), dS^T from shared memory; the streamed tile is read MN-major (its
                    // 128 columns are the output columns), 16 rows = 2048 bytes per step
                    const uint32_t bq = sStage + st * KV_STAGE_BYTES, bd = bq + KV_BYTES;
                    const uint64_t dQm = umma_smem_desc(bq, KV_BYTES / 2, 1024), dDm = umma_smem_desc(bd, KV_BYTES / 2, 1024);
                    const uint64_t dG = umma_smem_desc(sG + pr * KV_G_BYTES, 16, 1024);
                    const uint32_t tS = tmem_base + (pr ? 384 : 0);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_f16_ts(tDV, tS + 16 * kk, dDm + (uint64_t)(kk * 128), idesc_acc, (j > 0 || kk > 0) ? 1u : 0u);
                    tc_commit(pair_free0 + 8 * pr);
                    if (!mbar_wait(g_full0 + 8 * pr, (gt >> 1) & 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    umma_f16_x4(tDK, dG, dQm, idesc_acc, j > 0 ? 1u : 0u, 2u, 128u);
                    tc_commit(st_empty0 + 8 * st);
                    tc_commit(g_free0 + 8 * pr);
                    if (j == n - 1)
                        tc_commit(acc_done);
                }
            }
        }
    } else if (warp == 3) {
        // ------------------------------ dS^T tiles -> global memory ---------------
        if (lane == 0) {
            int gt = 0;
            bool ok = true;
            while (ok) {
                const int item = next_item(true);
                if (item < 0)
                    break;
                const int h = item / p.n_blocks, kb = item - h * p.n_blocks;
                const int4 tb = p.blocks[kb];
                const long long first = (long long)h * p.blocks[p.n_blocks].z + tb.z;
                for (int j = 0; j < tb.y && ok; ++j, ++gt) {
                    const int pr = gt & 1;
                    if (!(ok = mbar_wait(g_full0 + 8 * pr, (gt >> 1) & 1, abort_flag)))
                        break;
                    if (p.ds && first + j < p.ds_tiles) {
                        bulk_store(p.ds + (first + j) * KV_G_BYTES, sG + pr * KV_G_BYTES, KV_G_BYTES);
                        bulk_commit();
                        bulk_wait_read<0>();
                    }
                    mbar_arrive(g_free0 + 8 * pr);
                }
            }
        }
    } else {
        // ------------------------------ compute warps -----------------------------
        const int quarter = warp & 3, half = ((warp - 4) & 7) >> 2, grp = (warp - 4) >> 3;
        const int row = quarter * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        const uint32_t tS = tmem_base + (grp ? 384 : 0) + lane_addr + half * 32, tDP = tS + TC_BN;
        const float ds = att_dot_scale_tc(), c2 = ds * 0.693147f, slope = p.slope;
        uint8_t *const gbuf = smem + KV_G_OFF + grp * KV_G_BYTES;
        const uint32_t s_full = s_full0 + 8 * grp, g_full = g_full0 + 8 * grp, g_free = g_free0 + 8 * grp, dp_full = dp_full0 + 8 * grp,
                       p_full = p_full0 + 8 * grp, mate = mate0 + 8 * (grp * 4 + quarter);
        int gt = 0, live = 0, last_gt = -1; // last_gt: this group's latest tile
        uint32_t mate_phase = 0;
        bool ok = true;
        while (ok) {
            int item = next_item(false);
            ok = __all_sync(0xffffffffu, item != -2);
            if (!ok)
                break;
            if (lane == 0)
                mbar_arrive(rempty0 + 8 * ((rslot + KV_RING - 1) % KV_RING)); // every lane has read the slot
            if (item < 0)
                break;
            const int h = item / p.n_blocks, kb = item - h * p.n_blocks;
            const int4 tb = p.blocks[kb];
            const int n = tb.y, r0 = kb * TC_BM, rr = r0 + row; // key of this thread
            for (int j = 0; j < n; ++j, ++gt) {
                if ((gt & 1) != grp)
                    continue;
                const int st = gt % KV_STAGES;
                // s_full says the product is done; the tile's per-node records came with the same stage by bulk copies, and
                // the threads that read them observe that stage's barrier themselves (it has long completed: the issuer
                // waited for it before the products), which is what orders the copies' writes before these reads
                ok = __all_sync(0xffffffffu, mbar_wait(s_full, (gt >> 1) & 1, abort_flag) &&
                                                 mbar_wait(st_full0 + 8 * st, (gt / KV_STAGES) & 1, abort_flag));
                if (!ok)
                    break;
                tc_fence_after();
                const uint8_t *mt = smem + KV_META_OFF + st * KV_META_BYTES;
                const float4 *node = (const float4 *)mt + half * 16; // {-lse, -dscale c2} of two nodes
                const int2 info = *(const int2 *)(mt + ATT_NODE_BYTES + TC_BN * 8); // {latest span start, earliest span end} of the tile
                const bool plain = slope == 0.f && info.x <= r0 && info.y >= r0 + TC_BM - 1; // every node sees every key
                // P from the scores, in time for its product while dP is still on its way
                uint32_t w[32]; // scores, then weights
                tmem_ld32(tS, w);
                tmem_ld_wait();
                auto weights = [&](auto plain_tag) {
                    constexpr bool PLAIN = decltype(plain_tag)::value;
#pragma unroll
                    for (int q16 = 0; q16 < 2; ++q16) {
                        uint32_t pv[8];
                        const int4 *span = (const int4 *)(mt + ATT_NODE_BYTES) + half * 16 + q16 * 8; // {start, length} of two nodes
                        const int c0 = (tb.x + j) * TC_BN + half * 32 + q16 * 16 - rr;               // node - key
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int e = 16 * q16 + 2 * i;
                            const float4 m = node[q16 * 8 + i];
                            float o0 = m.x, o1 = m.z, w0, w1;
                            if (!PLAIN && slope != 0.f) {
                                o0 -= slope * (float)(c0 + 2 * i);
                                o1 -= slope * (float)(c0 + 2 * i + 1);
                            }
                            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w0) : "f"(fmaf(__uint_as_float(w[e]), ds, o0)));
                            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w1) : "f"(fmaf(__uint_as_float(w[e + 1]), ds, o1)));
                            if (!PLAIN) {
                                const int4 sp = span[i];
                                w0 = (unsigned)(rr - sp.x) <= (unsigned)sp.y ? w0 : 0.f;
                                w1 = (unsigned)(rr - sp.z) <= (unsigned)sp.w ? w1 : 0.f;
                            }
                            w[e] = __float_as_uint(w0);
                            w[e + 1] = __float_as_uint(w1);
                            pv[i] = bits_from_h2(sat_half2(w0, w1));
                        }
                        tmem_st8(tS + q16 * 16, pv); // where this thread's own S values were
                    }
                };
                if (plain)
                    weights(std::true_type());
                else
                    weights(std::false_type());
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(p_full);
                // dS
                ok = __all_sync(0xffffffffu, mbar_wait(dp_full, (gt >> 1) & 1, abort_flag) &&
                                                 (gt < 2 || mbar_wait(g_free, ((gt - 2) >> 1) & 1, abort_flag)));
                if (!ok)
                    break;
                tc_fence_after();
                uint32_t rp[32];
                tmem_ld32(tDP, rp);
                tmem_ld_wait();
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t gk[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int e = 8 * c + 2 * i;
                        const float4 m = node[4 * c + i];
                        gk[i] = bits_from_h2(sat_half2(__uint_as_float(w[e]) * fmaf(__uint_as_float(rp[e]), c2, m.y),
                                                       __uint_as_float(w[e + 1]) * fmaf(__uint_as_float(rp[e + 1]), c2, m.w)));
                    }
                    *(uint4 *)(gbuf + piece128(row, half * 4 + c)) = make_uint4(gk[0], gk[1], gk[2], gk[3]);
                }
                last_gt = gt;
                fence_proxy_async(); // dS^T is read by MMAs and by its store
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(g_full);
            }
            if (!ok)
                break;
            // epilogue: 32 columns of this row of both accumulators -> registers, then through the group's dS buffer (4 KB per
            // lane quarter, half of it for each of the two warps that share the quarter) and TMA stores.  Rows past T are clipped.
            const int part = grp * 2 + half;
            uint32_t av[32], ak[32];
            if (n > 0) {
                // all MMAs of the item are done; and the store of this group's last tile has read the buffer
                ok = __all_sync(0xffffffffu, mbar_wait(acc_done, live & 1, abort_flag) &&
                                                 (last_gt < 0 || mbar_wait(g_free, (last_gt >> 1) & 1, abort_flag)));
                if (!ok)
                    break;
                ++live;
                tc_fence_after();
                tmem_ld32(tDV + lane_addr + part * 32, av);
                tmem_ld32(tDK + lane_addr + part * 32, ak);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(acc_free);
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    av[i] = ak[i] = 0u;
            }
            uint8_t *const blk = gbuf + quarter * 4096 + half * 2048, *const srow = blk + lane * 64;
            const int sw = (lane >> 1) & 3, col = h * TC_HD + part * 32;
            constexpr int ROUNDS = OUT16 ? 2 : 4;
#pragma unroll
            for (int rd = 0; rd < ROUNDS; ++rd) { // dV, then dK: 32 rows x 64 bytes per round
                const uint32_t *a = rd < ROUNDS / 2 ? av : ak;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint4 v;
                    if constexpr (OUT16) {
                        const __half2 h0 = sat_half2(__uint_as_float(a[8 * i]), __uint_as_float(a[8 * i + 1])),
                                      h1 = sat_half2(__uint_as_float(a[8 * i + 2]), __uint_as_float(a[8 * i + 3])),
                                      h2 = sat_half2(__uint_as_float(a[8 * i + 4]), __uint_as_float(a[8 * i + 5])),
                                      h3 = sat_half2(__uint_as_float(a[8 * i + 6]), __uint_as_float(a[8 * i + 7]));
                        v = make_uint4(*(const uint32_t *)&h0, *(const uint32_t *)&h1, *(const uint32_t *)&h2, *(const uint32_t *)&h3);
                    } else {
                        const int b = 16 * (rd & 1) + 4 * i;
                        v = make_uint4(a[b], a[b + 1], a[b + 2], a[b + 3]);
                    }
                    *(uint4 *)(srow + ((i ^ sw) << 4)) = v;
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    tma_store_2d(rd < ROUNDS / 2 ? (const void *)&tmDV : (const void *)&tmDK, smem_u32(blk), col + (OUT16 ? 0 : 16 * (rd & 1)), r0 + quarter * 32);
                    bulk_commit();
                    bulk_wait_read<0>();
                }
                __syncwarp();
            }
            // the next tile's dS rows of this quarter overlap both warps' blocks
            if (lane == 0)
                mbar_arrive(mate);
            ok = __all_sync(0xffffffffu, mbar_wait(mate, mate_phase, abort_flag));
            mate_phase ^= 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1)
        tmem_dealloc(tmem_base, 512);
    if (threadIdx.x == 0 && *abort_flag)
        atomicOr(p.status, TS2_STATUS_WAIT_TIMEOUT);
}

// {-lse, -dscale * c2} per (head, node), and the item counter back to zero
__global__ void att_pack_meta_kernel(const float *__restrict__ lse, const float *__restrict__ dscale, int T, int Tpad, int H, float c2,
                                     float2 *__restrict__ meta, int *__restrict__ counter)
{
    grid_dep_wait();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx == 0)
        *counter = 0;
    if (idx >= Tpad * H)
        return;
    const int h = idx / Tpad, t = idx - h * Tpad;
    meta[idx] = t < T ? make_float2(-lse[(size_t)t * H + h], -dscale[(size_t)t * H + h] * c2) : make_float2(0.f, 0.f);
}

// What the backward kernels need to know about a batch's spans, the same for every head and layer.  Block 0: per block of
// 128 keys the 64-node tiles that hold any node which may attend to it, {first tile, tiles, tiles of the blocks before it, 0},
// whole 128-node blocks (a dQ block then finds all or none of its nodes); the last entry's third number is the sum.
// The other blocks: per 64-node tile {start, length} of every node's span (no span: a start no key reaches), then
// {latest start, earliest end} over the tile.
__global__ void __launch_bounds__(1024) att_layout_kernel(const int *__restrict__ span_start, const int *__restrict__ span_finish,
                                                          const int *__restrict__ rev_first, const int *__restrict__ rev_last, int T,
                                                          int n_blocks, int4 *__restrict__ blocks, uint8_t *__restrict__ spans)
{
    grid_dep_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (blockIdx.x > 0) {
        const int tile = (blockIdx.x - 1) * 32 + warp;
        if (tile >= 2 * n_blocks)
            return;
        int late = -1, early = 0x7fffffff;
        int2 *out = (int2 *)(spans + (size_t)tile * ATT_SPAN_BYTES);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = tile * TC_BN + i * 32 + lane;
            int st = 0x40000000, len = 0, fin = -1;
            if (t < T && span_finish[t] >= span_start[t]) {
                st = span_start[t];
                fin = span_finish[t];
                len = fin - st;
            }
            out[i * 32 + lane] = make_int2(st, len);
            late = max(late, st);
            early = min(early, fin);
        }
        for (int o = 16; o > 0; o >>= 1) {
            late = max(late, __shfl_xor_sync(0xffffffffu, late, o));
            early = min(early, __shfl_xor_sync(0xffffffffu, early, o));
        }
        if (lane == 0)
            *(int4 *)(out + TC_BN) = make_int4(late, early, 0, 0);
        return;
    }
    __shared__ int sums[32];
    int carry = 0; // tiles of the key blocks of earlier rounds
    for (int kb0 = 0; kb0 < n_blocks; kb0 += 32) {
        const int kb = kb0 + warp;
        int first = 0x7fffffff, last = -1;
        if (kb < n_blocks)
            for (int i = lane; i < TC_BM; i += 32) {
                const int to = kb * TC_BM + i;
                if (to < T && rev_last[to] >= rev_first[to]) {
                    first = min(first, rev_first[to]);
                    last = max(last, rev_last[to]);
                }
            }
        for (int o = 16; o > 0; o >>= 1) {
            first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
            last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
        }
        const int tile0 = last >= 0 ? first / TC_BM * 2 : 0, n = last >= 0 ? last / TC_BM * 2 + 2 - tile0 : 0;
        if (lane == 0)
            sums[warp] = n;
        __syncthreads();
        int before = carry, total = carry;
        for (int w = 0; w < 32; ++w) {
            before += w < warp ? sums[w] : 0;
            total += sums[w];
        }
        if (lane == 0 && kb < n_blocks)
            blocks[kb] = make_int4(tile0, n, before, 0);
        carry = total;
        __syncthreads();
    }
    if (threadIdx.x == 0)
        blocks[n_blocks] = make_int4(0, 0, carry, 0);
}

} // namespace

size_t att_layout_bytes(int T)
{
    const size_t nb = ceil_div(T, TC_BM);
    return (nb + 1) * sizeof(int4) + 2 * nb * ATT_SPAN_BYTES;
}

int att_layout(const Ctx &c, const int *span_start, const int *span_finish, const int *rev_first, const int *rev_last, int T, void *layout)
{
    const int nb = (int)ceil_div(T, TC_BM);
    TS2_LAUNCH((att_layout_kernel), 1 + (int)ceil_div(2 * nb, 32), 1024, 0, c.stream, span_start, span_finish, rev_first, rev_last, T, nb,
               (int4 *)layout, (uint8_t *)layout + (nb + 1) * sizeof(int4));
    return TS2_OK;
}

size_t att_bwd_scratch_bytes(int T, int H) { return 256 + (size_t)ceil_div(T, TC_BM) * TC_BM * H * sizeof(float2); }

int attention_backward_kv_tc(const Ctx &c, const __half *q, const __half *k, const __half *v, const __half *dout, const float *lse,
                             const float *dscale, const AttBwdPlan &plan, int T, int H, float slope, void *dk, void *dv, bool out16)
{
    static bool configured[16] = {};
    if (!configured[c.device & 15]) {
        TS2_CUDA(cudaFuncSetAttribute(att_bwd_kv_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, KV_SMEM));
        TS2_CUDA(cudaFuncSetAttribute(att_bwd_kv_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, KV_SMEM));
        configured[c.device & 15] = true;
    }
    const int Q = H * TC_HD;
    CUtensorMap tK, tV, tQ, tDO, tDK, tDV;
    int rc;
    if ((rc = make_tensor_map(&tK, k, 2, Q, T, Q, TC_BM)) != TS2_OK)
        return rc;
    if ((rc = make_tensor_map(&tV, v, 2, Q, T, Q, TC_BM)) != TS2_OK)
        return rc;
    if ((rc = make_tensor_map(&tQ, q, 2, Q, T, Q, TC_BN)) != TS2_OK)
        return rc;
    if ((rc = make_tensor_map(&tDO, dout, 2, Q, T, Q, TC_BN)) != TS2_OK)
        return rc;
    // outputs: boxes of 64 bytes (16 fp32 or 32 fp16 columns) x 32 rows
    if ((rc = make_tensor_map(&tDK, dk, out16 ? 2 : 4, Q, T, Q, 32, 64)) != TS2_OK)
        return rc;
    if ((rc = make_tensor_map(&tDV, dv, out16 ? 2 : 4, Q, T, Q, 32, 64)) != TS2_OK)
        return rc;
    AttBwdKvParams p;
    p.T = T;
    p.H = H;
    p.n_blocks = (int)ceil_div(T, TC_BM);
    p.Tpad = p.n_blocks * TC_BM;
    p.slope = slope;
    p.counter = (int *)plan.scratch;
    p.meta = (const float2 *)((uint8_t *)plan.scratch + 256);
    p.blocks = (const int4 *)plan.layout;
    p.spans = (const uint8_t *)plan.layout + (p.n_blocks + 1) * sizeof(int4);
    p.ds = (uint8_t *)plan.ds;
    p.ds_tiles = (int)std::min<size_t>(plan.ds_bytes / KV_G_BYTES, 0x7fffffff);
    p.status = device_status_word(c.device);
    if (!p.status)
        return fail(TS2_ERR_CUDA, "attention: no device status word");
    TS2_LAUNCH((att_pack_meta_kernel), (unsigned)ceil_div((int64_t)p.Tpad * H, 256), 256, 0, c.stream, lse, dscale, T, p.Tpad, H,
               att_dot_scale_tc() * 0.693147f, (float2 *)p.meta, p.counter);
    const int grid = (int)std::min<long long>((long long)p.n_blocks * H, sm_count(c.device));
    if (out16)
        TS2_LAUNCH((att_bwd_kv_tc_kernel<true>), grid, KV_THREADS, KV_SMEM, c.stream, tK, tV, tQ, tDO, tDK, tDV, p);
    else
        TS2_LAUNCH((att_bwd_kv_tc_kernel<false>), grid, KV_THREADS, KV_SMEM, c.stream, tK, tV, tQ, tDO, tDK, tDV, p);
    return TS2_OK;
}

} // namespace ts2
