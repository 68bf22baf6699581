// What the bf16 tensor-core Linears (linear_tc.cu) and the MLP in one launch (mlp_tc.cu) share: tile constants, the GELU and the folded
// LayerNorm of their epilogues, operand maps.
#pragma once

#include <cuda_fp16.h>

#include "linear.h"
#include "runtime.h"
#include "sm100.cuh"

namespace vtp {

constexpr int TBM = 128;   // tile rows of one CTA = TMEM lanes
constexpr int TBK = 64;    // 64 bf16 = one 128-byte swizzle row
constexpr int SLAB = 64;   // columns a warp takes through its staging buffer at a time: 128-byte rows
constexpr int SLAB_BYTES = 32 * SLAB * 2;
constexpr int SMEM_MAX = 232448;

// erf-GELU of eight values, packed two per register in fp16, as 0.5 x (1 + tanh(x (k0 + k1 x^2))) with
// k0, k1 fitted to 0.5 x (1 + erf(x / sqrt 2)) (max abs error 2.7e-4); fp16 arithmetic adds an rms
// error of 5e-4, a fifth of the rounding of the bf16 result.  Six packed instructions and one
// tanh.approx per pair: the form with ex2 + rcp per value kept the special-function unit
// (16 results per clock per SM) busier than the tensor core.  Inputs beyond the fp16 range
// saturate; there x^2 overflows to +inf, tanh gives +-1 and the result is x or 0 as it should.
__device__ __forceinline__ uint32_t gelu_pair_f16(float lo, float hi) {
    uint32_t x, t;
    asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(x) : "f"(hi), "f"(lo));
    const __half2 xh = *reinterpret_cast<__half2*>(&x);
    const __half2 u = __hmul2(xh, xh);
    const __half2 p = __hfma2(u, __float2half2_rn(0.03470089f), __float2half2_rn(0.80015708f));
    const __half2 a = __hmul2(xh, p);
    asm("tanh.approx.f16x2 %0, %1;" : "=r"(t) : "r"(*reinterpret_cast<const uint32_t*>(&a)));
    const __half2 hx = __hmul2(xh, __float2half2_rn(0.5f));
    const __half2 g = __hfma2(hx, *reinterpret_cast<__half2*>(&t), hx);
    return *reinterpret_cast<const uint32_t*>(&g);
}
__device__ __forceinline__ void gelu8(float* v) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t g = gelu_pair_f16(v[2 * i], v[2 * i + 1]);
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&g));
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}

__device__ const __align__(16) float g_no_bias[8] = {};      // what a Linear without a bias adds, read up to 16 bytes at a time

// A row's folded LayerNorm, LN(a) W^T + b = ln_a * acc + (ln_b * s[n] + bias[n]), from its statistics.  The problem of a pair that
// folds none (mode 0; its s[n] are g_no_bias) gets 1 * acc + (-0 * 0 + bias[n]), which is acc + bias[n] to the last bit.
__device__ __forceinline__ void row_fold(const LnFold& ln, int m, float& ln_a, float& ln_b) {
    if (ln.mode == 2) {
        // (sum, sum of squares) of each 64-column slab of the row, left by the GEMM that produced it; added in order
        const float4* sp = reinterpret_cast<const float4*>(ln.stats + (size_t)m * ln.slots);
        const int used = ln.used;
        const float dim = (float)ln.dim, eps = ln.eps;
        float s1 = 0.f, s2 = 0.f;
        for (int i0 = 0; 2 * i0 < used; i0 += 4) {
            float4 v4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)                    // independent 16-byte loads, one latency
                v4[i] = (2 * (i0 + i) < used) ? sp[i0 + i] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s1 += v4[i].x; s2 += v4[i].y;
                if (2 * (i0 + i) + 1 < used) { s1 += v4[i].z; s2 += v4[i].w; }
            }
        }
        const float mean = s1 / dim;
        ln_a = rsqrtf(fmaxf(s2 / dim - mean * mean, 0.f) + eps);
        ln_b = -ln_a * mean;
    } else if (ln.mode == 0) {
        ln_a = 1.f;
        ln_b = -0.f;
    } else {
        const float2 st = ln.stats[m];
        ln_a = st.y;
        ln_b = -st.y * st.x;
    }
}

// A [m_max, K] in boxes of one k-block of a CTA's rows; W [N, K] in boxes of `rows` rows.
static inline int operand_maps(CUtensorMap* ta, CUtensorMap* tw, const LinearArgs& p, unsigned rows) {
    const unsigned long long da[2] = {(unsigned long long)p.K, (unsigned long long)p.m_max};
    const unsigned long long sa[1] = {(unsigned long long)p.lda * 2ull};
    const unsigned ba[2] = {TBK, TBM};
    if (ta) if (int rc = make_tmap_bf16(ta, p.a, 2, da, sa, ba)) return rc;
    const unsigned long long dw[2] = {(unsigned long long)p.K, (unsigned long long)p.N};
    const unsigned long long sw[1] = {(unsigned long long)p.K * 2ull};
    const unsigned bw[2] = {TBK, rows};
    return make_tmap_bf16(tw, p.w, 2, dw, sw, bw);
}

// Reserves the dynamic shared memory of a kernel once per device.
template <typename Kernel>
static int reserve_smem(Kernel kern, int bytes, bool (&done)[64]) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && done[dev]) return VTP_OK;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) {
        set_error("linear (tcgen05): cannot reserve %d bytes of shared memory: %s", bytes, cudaGetErrorString(e));
        return (int)e;
    }
    if (dev >= 0 && dev < 64) done[dev] = true;
    return VTP_OK;
}

static inline int launched(cudaError_t e) {
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("linear (tcgen05): %s", cudaGetErrorString(e));
        return (int)e;
    }
    return check_launch("linear (tcgen05)");
}

static inline int check_tc_args(const LinearArgs& p) {
    VTP_REQUIRE(p.dtype == VTP_BF16, VTP_ERR_DTYPE, "linear (tcgen05): bf16 operands only");
    VTP_REQUIRE(p.K % TBK == 0, VTP_ERR_SHAPE, "linear (tcgen05): K=%d must be a multiple of %d", p.K, TBK);
    VTP_REQUIRE(p.N % 8 == 0, VTP_ERR_SHAPE, "linear (tcgen05): N=%d must be a multiple of 8", p.N);
    VTP_REQUIRE(p.ln_mode == 0 || (p.ln_stats && p.ln_s && p.out_grp == 0 &&
                                   (p.ln_mode == 1 || (p.ln_dim > 0 && p.ln_slots >= ceil_div(p.ln_dim, SLAB) && p.ln_slots % 2 == 0))),
                VTP_ERR_NULL, "linear (tcgen05): folded LayerNorm needs row statistics and the column sums");
    VTP_REQUIRE(p.ln_mode == 0 || !p.res, VTP_ERR_UNSUPPORTED, "linear (tcgen05): a folded LayerNorm takes no residual");
    VTP_REQUIRE(p.lda % 8 == 0 && p.ldy % 8 == 0 && (!p.res || p.ldr % 8 == 0), VTP_ERR_ALIGN,
                "linear (tcgen05): row strides must be multiples of 16 bytes");
    return VTP_OK;
}

}  // namespace vtp
