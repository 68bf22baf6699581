// Shared helpers for the vtpack_b200 kernels: element types, 16-byte vector access,
// warp reductions, argument checks and the per-thread error string.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/vtpack_b200.h"

namespace vtp {

typedef __nv_bfloat16 bf16;

// ---------------------------------------------------------------- host side errors
void set_error(const char* fmt, ...);
int fail(int code, const char* fmt, ...);
int check_launch(const char* what);

#define VTP_REQUIRE(cond, code, ...)            \
    do {                                        \
        if (!(cond)) return ::vtp::fail((code), __VA_ARGS__); \
    } while (0)

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline size_t elem_size(int dtype) { return dtype == VTP_BF16 ? 2 : 4; }
inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
inline long long round_up(long long a, long long b) { return (a + b - 1) / b * b; }

// Number of SMs of the current device (cached per device).
int sm_count();

// Launches `kernel`; with `early` it may start while the previous kernel on the stream is finishing (programmatic
// dependent launch; a programmatic edge when the stream is being captured into a graph).  Every kernel launched
// through here begins with pdl_begin(), or calls griddep_wait() before it touches anything an earlier kernel wrote
// (but for a first look at the status word, see launch_is_void) and griddep_launch() after that.  `cluster_x` > 1 cuts the grid into clusters.
template <typename... KArgs, typename... Args>
cudaError_t launch_kernel(void (*kernel)(KArgs...), bool early, int cluster_x, dim3 grid, dim3 block, size_t smem,
                          cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (early) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    if (cluster_x > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)cluster_x;
        attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
// Kernels with several CTAs per SM start early only when the grid is small.  CTAs that start early are placed on
// the SMs that have room first, as many as fit there, and stay packed on those: a latency-bound chain of small
// kernels gains (DeiT-Ti, one image: 790 -> 570 us launch by launch), a large grid would be left unevenly spread
// (DeiT-S, 12 images in fp32: 5.8 -> 8.2 ms with every kernel starting early).  The fp32 pool starts early whatever its grid, because of the
// matrices it splits (figures at pool_region_terms_kernel).
template <typename... KArgs, typename... Args>
cudaError_t launch_chain(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    const bool early = (long long)grid.x * grid.y * grid.z <= 2ll * sm_count();
    return launch_kernel(kernel, early, 1, grid, block, smem, st, static_cast<Args&&>(args)...);
}

// ---------------------------------------------------------------- device status word
// Bounded waits OR one of these codes into the device status word (see runtime.h)
// instead of hanging; vtp_device_status reads it back.
enum : int {
    STATUS_GEMM_PRODUCER = 1, STATUS_GEMM_MMA = 2, STATUS_GEMM_EPILOGUE = 4,
    STATUS_ATTN_LOAD = 8, STATUS_ATTN_MMA = 16, STATUS_ATTN_SOFTMAX = 32,
    STATUS_BAD_INDEX = 64,      // a caller-supplied patch row or row offset pointed outside the declared arrays
    STATUS_WAIT_MASK = 63,      // the bounded-wait codes: while one is set, tensor-core launches write nothing (launch_is_void)
};
// Whether an earlier launch gave up on a wait: nothing is written any more.  The word may be set by the kernel in front, so what
// decides about the stores is read behind the wait for that kernel; what is known in front of it saves the work too.  Launches
// on other streams may set the word at any time: ONE thread reads it and tells those that must decide alike (the roles of a
// CTA, the CTAs of a cluster) through shared memory.
__device__ __forceinline__ bool launch_is_void(const int* status) {
    return status && (*reinterpret_cast<const volatile int*>(status) & STATUS_WAIT_MASK) != 0;
}

// Index guards: kernels that follow caller-supplied indices (patch lists, packed-row offsets) check them
// against the declared shapes, skip what does not fit and OR STATUS_BAD_INDEX into the status word.
// Four integer compares per patch row; compile with -DVTP_INDEX_GUARDS=0 to leave them out.
#ifndef VTP_INDEX_GUARDS
#define VTP_INDEX_GUARDS 1
#endif

// ---------------------------------------------------------------- element vectors
// A Vec<T> is 16 bytes of T: 4 floats or 8 bf16.
template <typename T> struct Vec;
template <> struct Vec<float> {
    static constexpr int N = 4;
    float4 raw;
    __device__ __forceinline__ void load(const float* p) { raw = *reinterpret_cast<const float4*>(p); }
    __device__ __forceinline__ void store(float* p) const { *reinterpret_cast<float4*>(p) = raw; }
    __device__ __forceinline__ void to_float(float* f) const { f[0] = raw.x; f[1] = raw.y; f[2] = raw.z; f[3] = raw.w; }
    __device__ __forceinline__ void from_float(const float* f) { raw = make_float4(f[0], f[1], f[2], f[3]); }
};
template <> struct Vec<bf16> {
    static constexpr int N = 8;
    uint4 raw;
    __device__ __forceinline__ void load(const bf16* p) { raw = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ void store(bf16* p) const { *reinterpret_cast<uint4*>(p) = raw; }
    __device__ __forceinline__ void to_float(float* f) const {
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) { float2 t = __bfloat1622float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
    }
    __device__ __forceinline__ void from_float(const float* f) {
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    }
};

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(bf16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_f32<bf16>(float v) { return __float2bfloat16_rn(v); }

// Two values at once, each rounded as fmaf, a product and a difference are: half the issue slots.
#define VTP_PAIR_OP(OP, A, B, MORE, C)                                                                                  \
    float2 d;                                                                                                           \
    asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"        \
        OP ".rn.f32x2 d, a, b" MORE ";\n\tmov.b64 {%0, %1}, d;\n\t}"                                                    \
        : "=f"(d.x), "=f"(d.y)                                                                                          \
        : "f"(A.x), "f"(A.y), "f"(B.x), "f"(B.y), "f"(C.x), "f"(C.y));                                                  \
    return d;
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { VTP_PAIR_OP("fma", a, b, ", c", c) }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { VTP_PAIR_OP("mul", a, b, "", b) }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { VTP_PAIR_OP("add", a, b, "", b) }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { VTP_PAIR_OP("sub", a, b, "", b) }
#undef VTP_PAIR_OP
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
// channels 2i and 2i + 1 of a vector
__device__ __forceinline__ float2 pair_of(const Vec<bf16>& v, int i) {
    const uint32_t w = i == 0 ? v.raw.x : i == 1 ? v.raw.y : i == 2 ? v.raw.z : v.raw.w;
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
__device__ __forceinline__ void set_pair(Vec<bf16>& v, int i, float2 f) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
    (i == 0 ? v.raw.x : i == 1 ? v.raw.y : i == 2 ? v.raw.z : v.raw.w) = *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Programmatic dependent launch, device side.  griddep_wait() blocks until the kernel in front of this one on
// the stream has completed and its writes are visible; what stands before it overlaps that kernel's tail.
// griddep_launch() lets the kernel behind this one start once every CTA of this grid has called it.  It comes
// AFTER the wait: a kernel that has started then knows that everything up to the kernel before its
// predecessor has completed.  What stands before the wait reads no tensor, weights included: the predecessor may be
// the kernel that writes them.  (One kernel whose predecessor is always of the same call reads weights there:
// pool_region_terms_kernel.)
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() { griddep_wait(); griddep_launch(); }

__device__ __forceinline__ float gelu_erf(float x) {
    return 0.5f * x * (1.0f + erff(x * 0.70710678118654752440f));
}

}  // namespace vtp
