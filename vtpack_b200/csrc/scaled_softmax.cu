// Softmax of scaled score rows and its gradient, for the attention of the training path between its two ragged products:
//   p = softmax(scale * s),   ds = scale * p * (dp - sum(p * dp))
// A warp per row, whose values it keeps in registers up to 1056 keys; sums in fp32, one rounding at the end (the separate
// operations round the scaled scores and the unscaled gradient as well).  Rows have n elements without padding, so that they may start
// on any element: a lane takes single ones, 64 (bf16) or 128 (fp32) consecutive bytes a warp and access.  Bound by HBM: in place,
// every value is read and written once.  A training step is bound by the host, which it spares two launches a block each way; with
// the layout changes around the products in one node of the graph, forward and backward of a layer (48 images, C = 384) went from 2.18 to 1.97 ms.
//
// Replaces "* scale" and softmax of vtpack/models/dge/deit_dge.py:90-91 and pvt_dge.py:77-114.
#include "common.cuh"

namespace vtp {

constexpr int SS_WARPS = 4;

// PER: elements of a lane; 0: more than registers hold, which are read again instead.
template <typename T, int PER, bool GRAD>
__global__ void __launch_bounds__(SS_WARPS * 32)
scaled_softmax_kernel(const T* p, const T* x, T* y, long long rows, int n, float scale) {
    const int lane = threadIdx.x & 31;
    for (long long row = (long long)blockIdx.x * SS_WARPS + (threadIdx.x >> 5); row < rows; row += (long long)gridDim.x * SS_WARPS) {
        const T* xr = x + row * n;
        const T* pr = GRAD ? p + row * n : nullptr;
        T* yr = y + row * n;
        constexpr int KEEP = PER > 0 ? PER : 1;
        float v[KEEP], w[GRAD ? KEEP : 1];
        if (PER > 0) {
#pragma unroll
            for (int i = 0; i < KEEP; ++i) {
                const int c = i * 32 + lane;
                v[i] = c < n ? to_f32(xr[c]) : GRAD ? 0.f : -INFINITY;
                if (GRAD) w[i] = c < n ? to_f32(pr[c]) : 0.f;
            }
        }
        // of element c = i * 32 + lane (kept, or read again)
        auto val = [&](int i, int c) { return PER > 0 ? v[i] : to_f32(xr[c]); };
        auto prob = [&](int i, int c) { return PER > 0 ? w[GRAD ? i : 0] : to_f32(pr[c]); };
        auto each = [&](auto f) {
            if constexpr (PER > 0) {
#pragma unroll
                for (int i = 0; i < KEEP; ++i)
                    if (i * 32 + lane < n) f(i, i * 32 + lane);
            } else {
                for (int c = lane; c < n; c += 32) f(0, c);
            }
        };
        if constexpr (GRAD) {
            // ds = scale * (p dp - p sum): with the products rounded alike inside the sum and in front of it, a probability near one cancels
            // them (fp32, 16 scores of spread 64: relative error 1.57e-7, of p (dp - sum) 1.76e-7)
            float dot = 0.f;
            each([&](int i, int c) { dot += __fmul_rn(prob(i, c), val(i, c)); });
            dot = warp_sum(dot);
            each([&](int i, int c) { yr[c] = from_f32<T>(scale * fmaf(-prob(i, c), dot, __fmul_rn(prob(i, c), val(i, c)))); });
        } else {
            // (a scale below zero turns the order of the scores round, so the largest scaled one is looked for)
            float most = -INFINITY, sum = 0.f;
            each([&](int i, int c) { most = fmaxf(most, scale * val(i, c)); });
            most = warp_max(most);
            each([&](int i, int c) {
                const float e = expf(scale * val(i, c) - most);
                if (PER > 0) v[i] = e;
                sum += e;
            });
            sum = warp_sum(sum);
            // (a quotient each: times the reciprocal of the sum is a rounding more, relative error 6.6e-8 -> 7.0e-8 in fp32 at 257 keys)
            each([&](int i, int c) { yr[c] = from_f32<T>(__fdiv_rn(PER > 0 ? v[i] : expf(scale * to_f32(xr[c]) - most), sum)); });
        }
    }
}

template <typename T, bool GRAD>
static void launch_softmax(const void* p, const void* x, void* y, long long rows, int n, float scale, cudaStream_t st) {
    const long long want = (rows + SS_WARPS - 1) / SS_WARPS, cap = 32ll * sm_count();
    const int grid = (int)(want < cap ? want : cap);
#define VTP_SS(PER) scaled_softmax_kernel<T, PER, GRAD><<<grid, SS_WARPS * 32, 0, st>>>((const T*)p, (const T*)x, (T*)y, rows, n, scale)
    if (n <= 64) VTP_SS(2);
    else if (n <= 160) VTP_SS(5);
    else if (n <= 288) VTP_SS(9);
    else if (n <= 608) VTP_SS(19);
    else if (n <= 1056) VTP_SS(33);
    else VTP_SS(0);
#undef VTP_SS
}

static int scaled_softmax(const void* p, const void* x, int dtype, long long rows, int n, float scale, void* y, bool grad, void* stream) {
    VTP_REQUIRE(x && y && (p || !grad), VTP_ERR_NULL, "scaled softmax: null pointer");
    VTP_REQUIRE(dtype == VTP_F32 || dtype == VTP_BF16, VTP_ERR_DTYPE, "scaled softmax: dtype %d", dtype);
    VTP_REQUIRE(rows >= 0 && n > 0, VTP_ERR_SHAPE, "scaled softmax: %lld rows of %d", rows, n);
    if (rows == 0) return VTP_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == VTP_F32) grad ? launch_softmax<float, true>(p, x, y, rows, n, scale, st) : launch_softmax<float, false>(p, x, y, rows, n, scale, st);
    else grad ? launch_softmax<bf16, true>(p, x, y, rows, n, scale, st) : launch_softmax<bf16, false>(p, x, y, rows, n, scale, st);
    return check_launch("scaled softmax");
}

}  // namespace vtp

extern "C" int vtp_scaled_softmax(const void* s, int dtype, long long rows, int n, float scale, void* p, void* stream) {
    return vtp::scaled_softmax(nullptr, s, dtype, rows, n, scale, p, false, stream);
}

extern "C" int vtp_scaled_softmax_grad(const void* p, const void* dp, int dtype, long long rows, int n, float scale, void* ds, void* stream) {
    return vtp::scaled_softmax(p, dp, dtype, rows, n, scale, ds, true, stream);
}
