// fp32 rows as three bf16 terms: the form in which the Linears and the attention of fp32 blocks take their operands (linear_f32_terms.cu,
// attention_f32_tc.cu).  linear_f32_tc.cu splits fp32 rows into the same terms on the way.
//
// 2^16 x = h + m + l with 8 significant bits each, so the three hold the 24 bits of an fp32 number.  The factor 2^16 takes the
// last bit of the smallest fp32 number, 2^-149, to that of the smallest bf16 number, 2^-133, so that the split is exact for
// every finite x that 2^16 x and h do not overflow for; it is decoded exactly too.  For the others (|x| of about 2^112 and
// more, infinities, NaN) h is infinite, so that every sum they enter comes out infinite or NaN and is worked out again, and m and
// l are the upper and lower half of x itself.
//
// A row of n values is laid out as [3][n] bf16: h, m, l.
#pragma once

#include "common.cuh"

namespace vtp {

constexpr float F_SCALE = 65536.f, F_UNSCALE = 1.f / (65536.f * 65536.f);     // of an operand, of a sum of products

// The terms in the upper halves of h, m, l (the lower half of l is zero, too).  h is rounded to nearest (half away), so what
// is left over has either sign and the products that are left out do not add up; m and l cut the rest in two.  All exact, in
// integer and fp32 adds (the bf16 conversion instruction has a fraction of their rate).
__device__ __forceinline__ void split_scaled(float x, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = (__float_as_uint(x) + 0x8000u) & 0xFFFF0000u;
    const float r = x - __uint_as_float(h);
    m = __float_as_uint(r) & 0xFFFF0000u;
    l = __float_as_uint(r - __uint_as_float(m));
}
__device__ __forceinline__ void split_terms(float v, uint32_t& h, uint32_t& m, uint32_t& l) {
    const float x = v * F_SCALE;
    split_scaled(x, h, m, l);
    constexpr uint32_t INF = 0x7F800000u;
    if ((h & INF) == INF || (__float_as_uint(x) & INF) == INF) {
        h = INF | (__float_as_uint(v) & 0x80000000u);
        m = __float_as_uint(v) & 0xFFFF0000u;
        l = __float_as_uint(v) << 16;
    }
}
__device__ __forceinline__ float join_terms(uint32_t h, uint32_t m, uint32_t l) {      // bf16 bits in the lower halves
    if ((h & 0x7F80u) == 0x7F80u) return __uint_as_float(m << 16 | l);
    return (__uint_as_float(h << 16) + (__uint_as_float(m << 16) + __uint_as_float(l << 16))) * (1.f / F_SCALE);
}

// Eight consecutive values of a row whose terms are n apart.
__device__ __forceinline__ void join8(const bf16* p, size_t n, float (&f)[8]) {
    uint4 t[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) t[i] = __ldg(reinterpret_cast<const uint4*>(p + i * n));
    const uint32_t* h = &t[0].x;
    const uint32_t* m = &t[1].x;
    const uint32_t* l = &t[2].x;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int s = (i & 1) * 16;
        f[i] = join_terms((h[i >> 1] >> s) & 0xFFFFu, (m[i >> 1] >> s) & 0xFFFFu, (l[i >> 1] >> s) & 0xFFFFu);
    }
}

// Four consecutive values, the h terms to `row` on, terms n apart.
__device__ __forceinline__ void store_terms4(bf16* row, size_t n, const float* v) {
    uint32_t t[3][4], most = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float x = v[i] * F_SCALE;
        most = max(most, __float_as_uint(x) & 0x7FFFFFFFu);
        split_scaled(x, t[0][i], t[1][i], t[2][i]);
    }
    if (most >= 0x7F7F8000u) {             // one whose h, rounded, is infinite
#pragma unroll
        for (int i = 0; i < 4; ++i) split_terms(v[i], t[0][i], t[1][i], t[2][i]);
    }
#pragma unroll
    for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint2*>(row + p * n) = make_uint2(__byte_perm(t[p][0], t[p][1], 0x7632), __byte_perm(t[p][2], t[p][3], 0x7632));
}
// 32 bytes to a 32-byte boundary.
__device__ __forceinline__ void stg_u8(void* p, const uint32_t (&r)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// Vec<T>::N values of element `col` on of row `row` of y: T as they are, or (T = float, terms) as terms.
template <typename T>
__device__ __forceinline__ void store_row_vec(T* y, size_t row, int C, int col, const float* o, bool terms) {
    if constexpr (sizeof(T) == 4) {
        if (terms) {
            store_terms4(reinterpret_cast<bf16*>(y) + row * 3 * C + col, C, o);
            return;
        }
    }
    Vec<T> v;
    v.from_float(o);
    v.store(y + row * C + col);
}

// The matrices of a block, split on every call: a forward then follows whatever was done to the parameters, and the terms of
// one block stay in L2 until its Linears read them.
struct TermSplit {
    static constexpr int MOST = 6, PER_THREAD = 2;     // units of eight values
    const float* src[MOST] = {}; bf16* dst[MOST] = {};
    int K[MOST] = {};                                  // values per row, a multiple of 8
    unsigned units[MOST] = {};
    int n = 0;
    void add(const void* s, void* d, int rows, int k) {
        src[n] = static_cast<const float*>(s); dst[n] = static_cast<bf16*>(d); K[n] = k;
        units[n++] = (unsigned)((long long)rows * k / 8);
    }
    int ctas(int threads) const {
        int c = 0;
        for (int i = 0; i < n; ++i) c += (int)((units[i] + PER_THREAD * threads - 1) / (PER_THREAD * threads));
        return c;
    }
};
// Share `cta` of the split: two units a thread, both loaded before the first is split.
template <int THREADS>
__device__ __forceinline__ void split_matrices(const TermSplit& s, int cta) {
    constexpr int PT = TermSplit::PER_THREAD;
#pragma unroll 1
    for (int i = 0; i < TermSplit::MOST; ++i) {
        const int ctas = (int)((s.units[i] + PT * THREADS - 1) / (PT * THREADS));
        if (cta >= ctas) { cta -= ctas; continue; }
        const float* src = s.src[i];
        bf16* dst = s.dst[i];
        const unsigned K8 = (unsigned)s.K[i] / 8, units = s.units[i], u0 = (unsigned)cta * (PT * THREADS) + threadIdx.x;
        float4 v[PT][2];
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            const unsigned u = u0 + j * THREADS;
            if (u < units) {
                v[j][0] = __ldg(reinterpret_cast<const float4*>(src + (size_t)u * 8));
                v[j][1] = __ldg(reinterpret_cast<const float4*>(src + (size_t)u * 8) + 1);
            }
        }
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            const unsigned u = u0 + j * THREADS;
            if (u >= units) return;
            const unsigned r = u / K8, c = u - r * K8;
            const float f[8] = {v[j][0].x, v[j][0].y, v[j][0].z, v[j][0].w, v[j][1].x, v[j][1].y, v[j][1].z, v[j][1].w};
            uint32_t t[3][8];
#pragma unroll
            for (int e = 0; e < 8; ++e) split_terms(f[e], t[0][e], t[1][e], t[2][e]);
            bf16* d = dst + ((size_t)r * 3 * K8 + c) * 8;
#pragma unroll
            for (int p = 0; p < 3; ++p)
                *reinterpret_cast<uint4*>(d + (size_t)p * K8 * 8) =
                    make_uint4(__byte_perm(t[p][0], t[p][1], 0x7632), __byte_perm(t[p][2], t[p][3], 0x7632),
                               __byte_perm(t[p][4], t[p][5], 0x7632), __byte_perm(t[p][6], t[p][7], 0x7632));
        }
        return;
    }
}

// vtp_layernorm with fp32 rows in and their terms out (pool_unpool.cu).
int layernorm_terms(const void* x, int rows_max, const int32_t* rows_dev, int C, const float* w, const float* b, float eps, void* y,
                    cudaStream_t st);
// Rows of the stride-sr convolution in front of a PVT block's keys, fp32 tokens in, terms out (patch_embed.cu).
int token_im2col_terms(const void* x, int B, int H, int W, int C, int sr, void* cols, cudaStream_t st);

}  // namespace vtp
