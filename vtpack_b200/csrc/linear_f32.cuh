// What the two fp32 Linear kernels on tensor cores share (linear_f32_tc.cu: fp32 operands, linear_f32_terms.cu: operands as
// terms): the sums are formed alike, so a row's bits do not depend on which of the two they come from.
#pragma once

#include "common.cuh"
#include "sm100.cuh"

namespace vtp {

using namespace sm100;

constexpr int FM = 128;                 // tile rows = TMEM lanes
constexpr int FK = 64;                  // k-block: one 128-byte row of bf16 per operand term
constexpr int F_TMEM = 4;               // in tile widths: two accumulators, two group sums

// Groups of k-blocks that are added up apart: at least three k-blocks each.  More splits would leave a CTA less work
// than the exchange costs.
inline int f32_groups_log2(int num_kb) { return num_kb >= 12 ? 2 : num_kb >= 6 ? 1 : 0; }

// acc (op) a sum kept in tensor memory, NR columns at a time
template <int CW>
__device__ __forceinline__ void stash_store(uint32_t taddr, const float (&acc)[CW]) {
    __syncwarp();
#pragma unroll
    for (int c0 = 0; c0 < CW; c0 += 16) {
        uint32_t r[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(acc[c0 + i]);
        tmem_st_32x16(taddr + c0, r);
    }
    tmem_st_wait();
}
template <int CW, int NR = 32>
__device__ __forceinline__ void stash_add(uint32_t taddr, float (&acc)[CW]) {
#pragma unroll
    for (int c0 = 0; c0 < CW; c0 += NR) {
        uint32_t r[NR];
        __syncwarp();
        if constexpr (NR == 16) tmem_ld_32x16(taddr + c0, r);
        else tmem_ld_32x32(taddr + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < NR; ++i) acc[c0 + i] += __uint_as_float(r[i]);
    }
}

}  // namespace vtp
