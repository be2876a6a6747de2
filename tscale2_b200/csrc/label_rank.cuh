// Inverse label index of a small batch: every entry finds its place by comparing itself with all others.
#pragma once
#include "common.cuh"

namespace ts2 {

// Up to this many entries the comparisons (n^2, spread over n / 16 blocks) cost less than the launches of a radix sort: 512
// entries under a microsecond, 4096 about three, in blocks that other work of the same launch hides.
constexpr uint32_t LABEL_RANK_MAX = 4096;
constexpr int LABEL_RANK_THREADS = 256, LABEL_RANK_PER_BLOCK = LABEL_RANK_THREADS / 16;
inline int label_rank_blocks(uint32_t n) { return (int)ceil_div(n, LABEL_RANK_PER_BLOCK); }

#ifdef __CUDACC__
// Block `block` of LABEL_RANK_THREADS threads: sixteen entries, sixteen threads each.  Equal labels keep their order.  key is
// 16-byte aligned and readable up to a multiple of four entries.
__device__ __forceinline__ void label_rank(const uint32_t *__restrict__ key, const uint32_t *__restrict__ val, uint32_t n, uint32_t *__restrict__ key_out,
                                           uint32_t *__restrict__ val_out, uint32_t block)
{
    const uint32_t i = block * LABEL_RANK_PER_BLOCK + threadIdx.x / 16, sub = threadIdx.x & 15;
    const uint32_t mine = i < n ? key[i] : 0;
    uint32_t rank = 0;
    for (uint32_t j = sub * 4; j < n; j += 64) {
        const uint4 k = *(const uint4 *)(key + j);
        const uint32_t kk[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
            rank += j + u < n && (j + u < i ? kk[u] <= mine : kk[u] < mine);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
        rank += __shfl_xor_sync(0xffffffffu, rank, o);
    if (sub == 0 && i < n) {
        key_out[rank] = mine;
        val_out[rank] = val[i];
    }
}
#endif

} // namespace ts2
