// Variable-length-query attention on CUDA cores, fp32 arithmetic (fp32 or bf16 storage): fp32 of single calls and of fewer than 128 keys, and
// an independent check of the tcgen05 kernel.
//
// One CTA of four warps owns 32 packed queries of one (image, head) and walks the keys in chunks of up to 144 with an
// online softmax. A thread owns four query rows: of the scores it holds up to nine keys per row (keys tx, tx + 16,
// ...), of the output four channels, both in registers, so an inner step is 36 (or 16) fused multiply-adds per nine
// (five) shared-memory vectors; busiest are the issue slots and the shared-memory port (64 % each; FMA pipe 47 %, 256
// images). 257 keys are two chunks of 136 and 121. The sixteen threads that share a row exchange its maximum and sum
// with shuffles. Warps without live rows only stage K and V; images with fewer queries launch CTAs that exit. DeiT-S,
// 12 images in fp32: 71 us per launch for the form with one score per thread and step and the whole score row in shared
// memory, 42 us for this one with synchronous staging, 30 us with K and V copied asynchronously and unrolled steps.
//
// Replaces batched_sparse_attention_forward
// (vtpack/layers/csrc/batched_sparse_gemm/batched_sparse_gemm.cu:219-305): scale is applied
// to Q K^T before the softmax exactly as the reference passes it as the GEMM alpha (:275).
#include "attention.h"
#include "f32_terms.cuh"
#include "runtime.h"

namespace vtp {

constexpr int AQ = 32;              // queries per CTA
constexpr int AD = 64;              // head dim
constexpr int APITCH = AD + 4;      // row pitch of Q, K and V: consecutive rows start four banks apart
// J: keys per thread and chunk, 16 * J keys per chunk at most.  A template parameter, so that a step's loads are all
// issued before its multiply-adds (a branch per key left one shared-memory latency per key: 39 instead of 30 us).
constexpr int attn_simt_smem(int J) { return (AQ * APITCH + 2 * 16 * J * APITCH + AQ * (16 * J + 4)) * (int)sizeof(float); }

// fp32 rows are copied asynchronously, 16 bytes at a time; the caller commits and waits
__device__ __forceinline__ void copy_rows(float* dst, const float* __restrict__ src, long long stride, int n, int rows) {
    for (int e = threadIdx.x; e < rows * (AD / 4); e += 128) {
        const int r = e / (AD / 4), c = (e % (AD / 4)) * 4;
        float* d = dst + r * APITCH + c;
        if (r < n)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(d)),
                         "l"(src + (long long)r * stride + c) : "memory");
        else
            *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// rows of 64 elements -> fp32 rows of the shared-memory array `dst`; rows at or beyond `n` become zero
template <typename T>
__device__ __forceinline__ void stage_rows(float* dst, const T* __restrict__ src, long long stride, int n, int rows) {
    constexpr int VN = Vec<T>::N, CPR = AD / VN;
    for (int e = threadIdx.x; e < rows * CPR; e += 128) {
        const int r = e / CPR, c = (e % CPR) * VN;
        float f[VN];
#pragma unroll
        for (int i = 0; i < VN; ++i) f[i] = 0.f;
        if (r < n) {
            Vec<T> v;
            v.load(src + (long long)r * stride + c);
            v.to_float(f);
        }
#pragma unroll
        for (int i = 0; i < VN / 4; ++i)
            *reinterpret_cast<float4*>(dst + r * APITCH + c + 4 * i) = make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
    }
}
// the same for rows that do not start on 16-byte boundaries
template <typename T>
__device__ __forceinline__ void stage_rows_any(float* dst, const T* __restrict__ src, long long stride, int n, int rows) {
    for (int e = threadIdx.x; e < rows * AD; e += 128) {
        const int r = e / AD, c = e % AD;
        dst[r * APITCH + c] = r < n ? to_f32(src[(long long)r * stride + c]) : 0.f;
    }
}

template <typename T, bool VEC, int AKJ>
__global__ void __launch_bounds__(128, 2)
attn_simt_kernel(const T* __restrict__ q, long long q_rs, long long q_hs, const T* __restrict__ k,
                 const T* __restrict__ v, long long kv_bs, long long kv_rs, long long kv_hs,
                 T* __restrict__ out, long long o_rs, long long o_hs, int n_keys, int n_chunks, int kc,
                 const int32_t* __restrict__ offsets, int l_max, float scale, int* status, long long o_terms) {
    constexpr int AKC = 16 * AKJ, SPITCH = AKC + 4;      // chunk, row pitch of the probabilities
    pdl_begin();
    extern __shared__ float smem[];
    float* Qs = smem;                       // [AQ][APITCH]
    float* Ks = Qs + AQ * APITCH;           // [AKC][APITCH]
    float* Vs = Ks + AKC * APITCH;          // [AKC][APITCH]
    float* P = Vs + AKC * APITCH;           // [AQ][SPITCH]

    const int b = blockIdx.z, h = blockIdx.y;
    const int row0 = __ldg(offsets + b) + blockIdx.x * AQ;
    int row_end = __ldg(offsets + b + 1);
#if VTP_INDEX_GUARDS
    // caller-supplied offsets: rows outside [0, l_max) are not touched
    if (row0 < 0 || row_end > l_max) {
        if (threadIdx.x == 0 && status) atomicOr(status, STATUS_BAD_INDEX);
        if (row0 < 0) return;
        row_end = l_max;
    }
#endif
    if (row0 >= row_end) return;
    const int nq = min(AQ, row_end - row0);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;          // rows 4 * ty .. + 3
    const bool live = (threadIdx.x >> 5) * 8 < nq;                    // this warp's eight rows

    // every staging is one copy group (empty when the rows had to pass through registers): K of a chunk is on its way
    // while the chunk before multiplies P by V, its V while its scores are computed
    auto stage = [&](float* dst, const T* src, long long stride, int n, int rows) {
        if constexpr (VEC && sizeof(T) == 4) copy_rows(dst, src, stride, n, rows);
        else if constexpr (VEC) stage_rows<T>(dst, src, stride, n, rows);
        else stage_rows_any<T>(dst, src, stride, n, rows);
        copy_commit();
    };
    const T* kb = k + (long long)b * kv_bs + h * kv_hs;
    const T* vb = v + (long long)b * kv_bs + h * kv_hs;
    auto stage_chunk = [&](float* dst, const T* src, int c) {
        const int c0 = c * kc, n = min(kc, n_keys - c0);
        stage(dst, src + (long long)c0 * kv_rs, kv_rs, n, AKC);
    };
    stage(Qs, q + (long long)row0 * q_rs + h * q_hs, q_rs, nq, AQ);
    stage_chunk(Ks, kb, 0);
    stage_chunk(Vs, vb, 0);
    float o[4][4], m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) o[i][j] = 0.f;
    }
    for (int c = 0; c < n_chunks; ++c) {
        const int c0 = c * kc, n = min(kc, n_keys - c0), nr = (n + 3) & ~3;
        copy_wait<1>();                                              // this chunk's K (and Q) have landed, V may be on its way
        __syncthreads();
        if (live) {
            float s[4][AKJ];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < AKJ; ++j) s[i][j] = 0.f;
#pragma unroll 2
            for (int d = 0; d < AD; d += 4) {
                float4 qv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4*>(Qs + (ty * 4 + i) * APITCH + d);
#pragma unroll
                for (int j = 0; j < AKJ; ++j) {
                    const float4 kv = *reinterpret_cast<const float4*>(Ks + (tx + 16 * j) * APITCH + d);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        s[i][j] = fmaf(qv[i].x, kv.x, s[i][j]);
                        s[i][j] = fmaf(qv[i].y, kv.y, s[i][j]);
                        s[i][j] = fmaf(qv[i].z, kv.z, s[i][j]);
                        s[i][j] = fmaf(qv[i].w, kv.w, s[i][j]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float mx = -INFINITY;
#pragma unroll
                for (int j = 0; j < AKJ; ++j) {
                    s[i][j] = tx + 16 * j < n ? s[i][j] * scale : -INFINITY;
                    mx = fmaxf(mx, s[i][j]);
                }
#pragma unroll
                for (int w = 8; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
                const float m_new = fmaxf(m[i], mx);
                const float m_at = m_new == -INFINITY ? 0.f : m_new;  // (scores of -inf have weight zero, a chunk of them too)
                const float alpha = expf(m[i] - m_at);               // 0 while m is -inf
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < AKJ; ++j) {
                    const float p = expf(s[i][j] - m_at);            // keys beyond the chunk: exp(-inf) = 0
                    P[(ty * 4 + i) * SPITCH + tx + 16 * j] = p;
                    sum += p;
                }
#pragma unroll
                for (int w = 8; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
                l[i] = l[i] * alpha + sum;
                m[i] = m_new;
#pragma unroll
                for (int j = 0; j < 4; ++j) o[i][j] *= alpha;
            }
        }
        __syncthreads();                                             // K has been read
        if (c + 1 < n_chunks) stage_chunk(Ks, kb, c + 1);
        else copy_commit();
        copy_wait<1>();                                              // this chunk's V has landed
        __syncthreads();
        if (live) {
#pragma unroll 2
            for (int r = 0; r < nr; r += 4) {
                float4 pv[4], vv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) pv[i] = *reinterpret_cast<const float4*>(P + (ty * 4 + i) * SPITCH + r);
#pragma unroll
                for (int i = 0; i < 4; ++i) vv[i] = *reinterpret_cast<const float4*>(Vs + (r + i) * APITCH + tx * 4);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float pr[4] = {pv[i].x, pv[i].y, pv[i].z, pv[i].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        o[i][0] = fmaf(pr[j], vv[j].x, o[i][0]);
                        o[i][1] = fmaf(pr[j], vv[j].y, o[i][1]);
                        o[i][2] = fmaf(pr[j], vv[j].z, o[i][2]);
                        o[i][3] = fmaf(pr[j], vv[j].w, o[i][3]);
                    }
                }
            }
        }
        if (c + 1 < n_chunks) {
            __syncthreads();                                         // V has been read
            stage_chunk(Vs, vb, c + 1);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int qi = ty * 4 + i;
        if (qi >= nq) continue;
        const float inv = 1.f / l[i];
        if constexpr (sizeof(T) == 4) {
            if (o_terms) {
                const float v[4] = {o[i][0] * inv, o[i][1] * inv, o[i][2] * inv, o[i][3] * inv};
                store_terms4(reinterpret_cast<bf16*>(out) + (long long)(row0 + qi) * o_rs + h * o_hs + tx * 4, (size_t)o_terms, v);
                continue;
            }
        }
        T* p = out + (long long)(row0 + qi) * o_rs + h * o_hs + tx * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = from_f32<T>(o[i][j] * inv);
    }
}

template <typename T, int J>
static int launch_simt_j(const AttnArgs& p, cudaStream_t st) {
    constexpr int VN = Vec<T>::N;
    const bool vec = aligned16(p.q) && aligned16(p.k) && aligned16(p.v) && p.q_rs % VN == 0 && p.q_hs % VN == 0 &&
                     p.kv_bs % VN == 0 && p.kv_rs % VN == 0 && p.kv_hs % VN == 0;
    auto kern = vec ? attn_simt_kernel<T, true, J> : attn_simt_kernel<T, false, J>;
    constexpr int smem = attn_simt_smem(J);
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) {
        set_error("attention (CUDA cores): %s", cudaGetErrorString(e));
        return (int)e;
    }
    // equal chunks, each a multiple of 8 keys
    const int kc = (int)round_up(ceil_div(p.n_keys, ceil_div(p.n_keys, 16 * J)), 8);
    // a query tile never straddles images; images with fewer queries launch CTAs that exit
    launch_kernel(kern, false, 1, dim3(ceil_div(p.max_q, AQ), p.heads, p.B), dim3(128), (size_t)smem, st,
                  (const T*)p.q, p.q_rs, p.q_hs, (const T*)p.k, (const T*)p.v, p.kv_bs, p.kv_rs, p.kv_hs, (T*)p.out, p.o_rs,
                  p.o_hs, p.n_keys, ceil_div(p.n_keys, kc), kc, p.offsets, p.l_max, p.scale, device_status_ptr(), p.o_terms);
    return check_launch("attention (CUDA cores)");
}

// 64 keys (the spatially reduced keys of a pyramid block) are one chunk of four keys per thread, anything longer
// runs in chunks of up to 144 (257 keys: 136 + 121)
template <typename T>
static int launch_simt(const AttnArgs& p, cudaStream_t st) {
    return p.n_keys <= 64 ? launch_simt_j<T, 4>(p, st) : launch_simt_j<T, 9>(p, st);
}

int attention_cuda_cores(const AttnArgs& p, cudaStream_t st) {
    VTP_REQUIRE(p.head_dim == AD, VTP_ERR_UNSUPPORTED, "attention: head_dim %d (only %d)", p.head_dim, AD);
    VTP_REQUIRE(p.B <= 65535 && p.heads <= 65535, VTP_ERR_SHAPE, "attention (CUDA cores): %d images x %d heads exceed the grid", p.B, p.heads);
    return p.dtype == VTP_F32 ? launch_simt<float>(p, st) : launch_simt<bf16>(p, st);
}

}  // namespace vtp
