// Where the images' rows start in the operands of a ragged product.
#pragma once

#include <stdint.h>

namespace vtp {

// Host-side lengths travel with the launch: prefix sums of up to RG_INLINE_IMAGES images (4.1 KB of the 32 KB that a
// kernel's parameters may take) instead of a host-to-device copy in front of every product.  With more images, and
// for callers that have the offsets on the device, the kernels read them from memory.  One training-mode DeiT-S layer,
// forward and backward on 48 images, is bound by its host side: without the twelve copies of its six products, and with
// the region rows from the patch-list kernel instead of nine tensor operations, 3299 -> 2706 us.
constexpr int RG_INLINE_IMAGES = 512;
struct RaggedOffsets {
    const int32_t* a_dev;      // null: the arrays below
    const int32_t* b_dev;
    int32_t a[RG_INLINE_IMAGES + 1], b[RG_INLINE_IMAGES + 1];
    __device__ __forceinline__ int a_at(int i) const { return a_dev ? a_dev[i] : a[i]; }
    __device__ __forceinline__ int b_at(int i) const { return b_dev ? b_dev[i] : b[i]; }
};

// bf16: the tensor-core kernel (ragged_gemm_tc.cu)
int ragged_gemm_tcgen05(const void* a, const void* b, void* out, int heads, int n_images, long long a_rows,
                        int a_cols, long long b_rows, int b_cols, const RaggedOffsets& off,
                        int max_m, int max_n, int ta, int tb, long long out_rows, int out_cols, cudaStream_t st);

}  // namespace vtp
