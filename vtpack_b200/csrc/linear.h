// Internal interface of the Linear (GEMM + epilogue) kernels.
#pragma once

#include "common.cuh"

namespace vtp {

// y[out_row(m), n] = act(sum_k a[m,k] w[n,k] + bias[n]) + res[res_row(m), n]
//   out_row(m) = m + (m / out_grp + 1) * out_skip   when out_grp > 0, else m
//   res_row(m) = m % res_mod + res_off              when res_mod > 0, else m
// The row maps exist for the patch embedding, whose GEMM rows (b, t) land on token
// rows (b, 1 + t) and add the position embedding of token 1 + t.
struct LinearArgs {
    const void* a = nullptr; long long lda = 0;
    const void* w = nullptr;
    const float* bias = nullptr;
    const void* res = nullptr; long long ldr = 0;
    void* y = nullptr; long long ldy = 0;
    int dtype = VTP_F32;
    int m_max = 0; const int32_t* m_dev = nullptr;
    int N = 0, K = 0;
    unsigned flags = 0;
    int out_grp = 0, out_skip = 0;
    int res_mod = 0, res_off = 0;
    // LayerNorm folded into the GEMM (tcgen05 kernel only): `a` holds the raw rows, `w` holds
    // W*diag(gamma), ln_s[n] = sum_k w[n,k], bias[n] = sum_k beta[k] W[n,k] + b[n]; then
    //   LN(a) W^T + b = rstd[m] * (acc[m,n] - mean[m] * ln_s[n]) + bias[n].
    // ln_mode 1: ln_stats[m] = (mean, rstd).  ln_mode 2: ln_stats[m * ln_slots + i], 64 i < ln_dim,
    // are (sum, sum of squares) over 64 of the row's ln_dim elements each (written by the GEMM that
    // produced the rows, see emit_stats); variance = E[x^2] - mean^2, rstd = rsqrt(var + ln_eps).
    const float2* ln_stats = nullptr; const float* ln_s = nullptr;
    int ln_mode = 0, ln_dim = 0, ln_slots = 0; float ln_eps = 0.f;
    // When set, every stored row leaves (sum, sum of squares) of its outputs here, one slot per 64 columns: plain
    // stores, so the result does not depend on timing, nor, the columns being added in a fixed order, on the tiles.
    // Slots of a row are linear_stat_slots(N) apart (an even number, for the consumer's 16-byte loads).
    float2* emit_stats = nullptr;
    // fp32 only: y takes the three bf16 terms of every row, [3][N], instead of fp32 values (f32_terms.cuh).
    bool out_terms = false;
};

int linear_stat_slots(int N);              // float2 slots a tcgen05 GEMM with N output columns takes per row

struct LnFold { const float2* stats; const float* s; int mode, dim; float eps; float2* emit; int slots, used; };

int linear_validate(const LinearArgs& p);
int linear_cuda_cores(const LinearArgs& p, cudaStream_t st);   // fp32 or bf16 inputs, CUDA cores
int linear_tcgen05(const LinearArgs& p, cudaStream_t st);      // bf16 inputs, tcgen05 + TMA
bool linear_f32_tc_supported(const LinearArgs& p);
int linear_f32_tcgen05(const LinearArgs& p, cudaStream_t st);  // fp32 inputs as three bf16 terms each, tcgen05
int linear_f32_terms(const LinearArgs& p, cudaStream_t st);    // fp32 with a and w as rows of terms (f32_terms.cuh), lda unused
int linear_f32_terms_pair(const LinearArgs& a, const LinearArgs& b, cudaStream_t st);    // two of them, in one launch if that is shorter
int linear(const LinearArgs& p, cudaStream_t st);              // picks by dtype / flags
bool linear_pair_supported(const LinearArgs& a, const LinearArgs& b);
int linear_tcgen05_pair(const LinearArgs& a, const LinearArgs& b, cudaStream_t st);   // two problems, one launch

bool mlp_tcgen05_supported(const LinearArgs& fc1, const LinearArgs& fc2);
bool mlp_tcgen05_pays(const LinearArgs& fc1);
int mlp_tcgen05(const LinearArgs& fc1, const LinearArgs& fc2, cudaStream_t st);       // both, the hidden rows on chip

// Unsigned division by a number the host knows: multiply by ceil(2^32 / d), then take back the one the estimate may
// be over (it is never under).  A runtime division is about forty dependent instructions on the way to a CTA's first load.
struct FastDiv { uint32_t d, magic; };
inline FastDiv make_fast_div(uint32_t d) { return FastDiv{d, d == 1 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d)}; }
__device__ __forceinline__ uint32_t fast_div(uint32_t n, const FastDiv& f) {
    if (f.d == 1) return n;
    uint32_t q = __umulhi(n, f.magic);
    if (q * f.d > n) --q;          // (n and d are below 2^31)
    return q;
}

struct RowMap { int out_grp, out_skip, res_mod, res_off; };
__device__ __forceinline__ long long map_out_row(const RowMap& r, int m) {
    return r.out_grp > 0 ? (long long)m + (long long)(m / r.out_grp + 1) * r.out_skip : (long long)m;
}
__device__ __forceinline__ long long map_res_row(const RowMap& r, int m) {
    return r.res_mod > 0 ? (long long)(m % r.res_mod + r.res_off) : (long long)m;
}

}  // namespace vtp
