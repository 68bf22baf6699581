// Bilinear-sampling attention of the deformable PVT (vtpack/models/standard/dpvt.py:92-115):
// every query position g of a feature map [B, H, W, C] looks at P sampling points given in pixel
// coordinates (x, y), reads the map there by bilinear interpolation (zero outside the map) and
//   "point"   mode: out[b,g,c] = sum_p weight[b,g,p] * sample(b, p, c)         weight [B,G,P]
//   "channel" mode: out[b,g,p] = sum_c weight[b,g,c] * sample(b, p, c)         weight [B,G,C]
// Replaces bilinear_attention_{pointwise,channelwise}_{forward,backward}
// (vtpack/layers/csrc/bilinear_attention/bilinear_attention.cu:88-132, :134-232, :234-268, :270-362).
//
// The reference runs one thread per (b, g) that walks the channels serially, so neighbouring threads read addresses
// C elements apart.  Here a group of LG lanes owns a (b, g) instance and each lane a 16-byte vector of its channels
// (8 bf16 / 4 fp32): 4 instances per warp at C = 64 in bf16.  A point's corner arithmetic and the reductions over
// the channels are then paid once per 16 bytes instead of once per channel pair, and the input gradient leaves as
// one vector red per corner.
// Measured on 32 maps of 64 x 64 x 64, 9 points, bf16, point mode: forward + backward 525 -> 245 us (71 + 163 us) against a
// warp per instance with a channel pair per lane, 203 (65 + 138) with the backward's derivatives formed from four dot products
// and taps outside the map as zeroed raw words.  Bound: the issue slots and, in the backward, the SM's request port to L2 (69 % at
// 163 us: 4 x 128 bytes of reds per point); DRAM 5 %.  Tried and not kept, with the sums as they were: contiguous query ranges per SM
// for the L1 (71 -> 76 / 163 -> 157 us), packed f32x2 arithmetic (70 / 163 us), a point's corners worked out by one lane and handed
// round by shuffles (78 / 159 us), no reds at all 136 us; and what is faster and less exact, relative errors in fp32: the corners' weights times
// the point's in front of the channels (forward 71 -> 69 us, 6.0e-8 -> 7.8e-8), derivatives from sums of taps (138 -> 120 us, point
// gradients of a map with an offset of 100 7.9e-8 -> 6.8e-6), weight gradients from one tap's sum and the differences' (138
// -> 130 us, 8.2e-8 -> 1.6e-7).
#include <initializer_list>

#include "common.cuh"

namespace vtp {

constexpr int BA_WARPS = 8;           // warps per block
constexpr int BA_MAXCH = 8;           // widest C of the backward / 32: a lane keeps its weight gradients in registers

struct Corner {
    int x0, y0;
    float w_lt, w_rt, w_lb, w_rb, tx, ty;
    bool in_lt, in_rt, in_lb, in_rb;
};

__device__ __forceinline__ Corner corners_of(float x, float y, int H, int W) {
    Corner c;
    const float fx = floorf(x), fy = floorf(y);
    c.x0 = (int)fx;
    c.y0 = (int)fy;
    c.tx = x - fx;
    c.ty = y - fy;
    c.w_lt = (1.f - c.tx) * (1.f - c.ty);
    c.w_rt = c.tx * (1.f - c.ty);
    c.w_lb = (1.f - c.tx) * c.ty;
    c.w_rb = c.tx * c.ty;
    const bool xl = c.x0 >= 0 && c.x0 < W, xr = c.x0 + 1 >= 0 && c.x0 + 1 < W;
    const bool yt = c.y0 >= 0 && c.y0 < H, yb = c.y0 + 1 >= 0 && c.y0 + 1 < H;
    c.in_lt = xl && yt; c.in_rt = xr && yt; c.in_lb = xl && yb; c.in_rb = xr && yb;
    return c;
}

// a coordinate far outside the map (or not finite) touches no pixel; clamp it so the int casts stay defined
__device__ __forceinline__ float sane(float v, int extent) {
    return (v > -4.f && v < (float)extent + 4.f) ? v : -4.f;
}

// V consecutive channels per lane: 16 bytes, or one pair / one channel where the rows are not made of 16-byte vectors
template <typename T, int V> struct Pack {
    static_assert(V == Vec<T>::N, "");
    static __device__ __forceinline__ void load(const T* p, float (&f)[V]) {
        Vec<T> v;
        v.load(p);
        v.to_float(f);
    }
    // zeros unless `in`
    static __device__ __forceinline__ void load_if(bool in, const T* p, float (&f)[V]) {
        Vec<T> v = {};
        if (in) v.load(p);
        v.to_float(f);
    }
    static __device__ __forceinline__ void store(T* p, const float (&f)[V]) {
        Vec<T> v;
        v.from_float(f);
        v.store(p);
    }
    static __device__ __forceinline__ void atomic_add(T* p, const float (&f)[V]) {
        Vec<T> v;
        v.from_float(f);
        const uint4 r = *reinterpret_cast<const uint4*>(&v.raw);
        if constexpr (sizeof(T) == 4)
            asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(f[0]), "f"(f[1]),
                         "f"(f[2]), "f"(f[3]));
        else
            asm volatile("red.relaxed.gpu.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(r.x),
                         "r"(r.y), "r"(r.z), "r"(r.w));
    }
};
template <> struct Pack<float, 1> {
    static __device__ __forceinline__ void load_if(bool in, const float* p, float (&f)[1]) {
        for (int v = 0; v < 1; ++v) f[v] = 0.f;
        if (in) load(p, f);
    }
    static __device__ __forceinline__ void load(const float* p, float (&f)[1]) { f[0] = *p; }
    static __device__ __forceinline__ void store(float* p, const float (&f)[1]) { *p = f[0]; }
    static __device__ __forceinline__ void atomic_add(float* p, const float (&f)[1]) { atomicAdd(p, f[0]); }
};
template <> struct Pack<float, 2> {
    static __device__ __forceinline__ void load_if(bool in, const float* p, float (&f)[2]) {
        for (int v = 0; v < 2; ++v) f[v] = 0.f;
        if (in) load(p, f);
    }
    static __device__ __forceinline__ void load(const float* p, float (&f)[2]) {
        const float2 v = *reinterpret_cast<const float2*>(p);
        f[0] = v.x; f[1] = v.y;
    }
    static __device__ __forceinline__ void store(float* p, const float (&f)[2]) {
        *reinterpret_cast<float2*>(p) = make_float2(f[0], f[1]);
    }
    static __device__ __forceinline__ void atomic_add(float* p, const float (&f)[2]) {
        atomicAdd(reinterpret_cast<float2*>(p), make_float2(f[0], f[1]));
    }
};
template <> struct Pack<bf16, 1> {
    static __device__ __forceinline__ void load_if(bool in, const bf16* p, float (&f)[1]) {
        for (int v = 0; v < 1; ++v) f[v] = 0.f;
        if (in) load(p, f);
    }
    static __device__ __forceinline__ void load(const bf16* p, float (&f)[1]) { f[0] = __bfloat162float(*p); }
    static __device__ __forceinline__ void store(bf16* p, const float (&f)[1]) { *p = __float2bfloat16_rn(f[0]); }
    static __device__ __forceinline__ void atomic_add(bf16* p, const float (&f)[1]) {
        atomicAdd(p, __float2bfloat16_rn(f[0]));
    }
};
template <> struct Pack<bf16, 2> {
    static __device__ __forceinline__ void load_if(bool in, const bf16* p, float (&f)[2]) {
        for (int v = 0; v < 2; ++v) f[v] = 0.f;
        if (in) load(p, f);
    }
    static __device__ __forceinline__ void load(const bf16* p, float (&f)[2]) {
        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
        f[0] = v.x; f[1] = v.y;
    }
    static __device__ __forceinline__ void store(bf16* p, const float (&f)[2]) {
        *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(f[0], f[1]);
    }
    static __device__ __forceinline__ void atomic_add(bf16* p, const float (&f)[2]) {
        atomicAdd(reinterpret_cast<__nv_bfloat162*>(p), __floats2bfloat162_rn(f[0], f[1]));
    }
};

template <typename T, int V>
struct Taps {
    float lt[V], rt[V], lb[V], rb[V];
    __device__ __forceinline__ void load(const T* __restrict__ img, const Corner& k, int W, int C, int c) {
        const size_t o = ((size_t)k.y0 * W + k.x0) * C + c;   // only dereferenced where in-bounds
        Pack<T, V>::load_if(k.in_lt, img + o, lt);
        Pack<T, V>::load_if(k.in_rt, img + o + C, rt);
        Pack<T, V>::load_if(k.in_lb, img + o + (size_t)W * C, lb);
        Pack<T, V>::load_if(k.in_rb, img + o + (size_t)W * C + C, rb);
    }
    __device__ __forceinline__ float value(const Corner& k, int v) const {
        return k.w_lt * lt[v] + k.w_rt * rt[v] + k.w_lb * lb[v] + k.w_rb * rb[v];
    }
};

template <typename T, int V>
__device__ __forceinline__ void scatter(T* __restrict__ gimg, const Corner& k, int W, int C, int c, const float (&up)[V], float sc) {
    const size_t o = ((size_t)k.y0 * W + k.x0) * C + c;
    float t[V];
#define VTP_BA_SCATTER(IN, OFF, WT)                              \
    if (IN) {                                                    \
        const float a = sc * (WT);                               \
        _Pragma("unroll") for (int v = 0; v < V; ++v) t[v] = up[v] * a; \
        Pack<T, V>::atomic_add(gimg + o + (OFF), t);             \
    }
    VTP_BA_SCATTER(k.in_lt, 0, k.w_lt)
    VTP_BA_SCATTER(k.in_rt, C, k.w_rt)
    VTP_BA_SCATTER(k.in_lb, (size_t)W * C, k.w_lb)
    VTP_BA_SCATTER(k.in_rb, (size_t)W * C + C, k.w_rb)
#undef VTP_BA_SCATTER
}

// sum over the LG lanes of a group
template <int LG> __device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int o = LG / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// a point's coordinates; one load where the caller checked that pairs are aligned
template <bool VEC> __device__ __forceinline__ float2 point_xy(const float* p) {
    if constexpr (VEC) return *reinterpret_cast<const float2*>(p);
    else return make_float2(p[0], p[1]);
}
template <bool VEC> __device__ __forceinline__ float2 point_xy(const bf16* p) {
    if constexpr (VEC) return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
    else return make_float2(__bfloat162float(p[0]), __bfloat162float(p[1]));
}

// ---------------------------------------------------------------------------- forward
template <typename T, bool POINT, int V, int LG>
__global__ void __launch_bounds__(BA_WARPS * 32)
bilinear_attention_fwd_kernel(const T* __restrict__ input, const T* __restrict__ grid, const T* __restrict__ weight,
                              T* __restrict__ out, int B, int H, int W, int C, int G, int P,
                              const long long* __restrict__ batch_of) {
    // batch_of == null: B * G instances, G per image; else G packed instances, instance i reads image batch_of[i]
    constexpr int PW = 32 / LG;                          // instances per warp
    constexpr bool VEC = V == Vec<T>::N;
    const int lane = threadIdx.x & 31, gl = lane % LG, sub = lane / LG;
    const long long n_inst = batch_of ? (long long)G : (long long)B * G;
    for (long long first = ((long long)blockIdx.x * BA_WARPS + (threadIdx.x >> 5)) * PW; first < n_inst;
         first += (long long)gridDim.x * BA_WARPS * PW) {
        const bool own = first + sub < n_inst;           // a group past the end goes along for the shuffles
        const long long inst = own ? first + sub : first;
        long long b = batch_of ? batch_of[inst] : inst / G;
        const bool image_ok = b >= 0 && b < B;           // an instance naming no image reads zeros
        if (!image_ok) b = 0;
        const int Hb = image_ok ? H : 0;                 // no pixel is in bounds
        const T* img = input + (size_t)b * H * W * C;
        const T* pts = grid + (size_t)inst * P * 2;
        if (POINT) {
            const T* wt = weight + (size_t)inst * P;
            for (int c = gl * V; c < C; c += LG * V) {
                float acc[V];
#pragma unroll
                for (int v = 0; v < V; ++v) acc[v] = 0.f;
#pragma unroll 3
                for (int p = 0; p < P; ++p) {
                    const float2 xy = point_xy<VEC>(pts + 2 * p);
                    const Corner k = corners_of(sane(xy.x, W), sane(xy.y, H), Hb, W);
                    Taps<T, V> t;
                    t.load(img, k, W, C, c);
                    const float wp = to_f32(wt[p]);
#pragma unroll
                    for (int v = 0; v < V; ++v) acc[v] = fmaf(t.value(k, v), wp, acc[v]);
                }
                if (own) Pack<T, V>::store(out + (size_t)inst * C + c, acc);
            }
        } else {
            const T* wt = weight + (size_t)inst * C;
            for (int p = 0; p < P; ++p) {
                const float2 xy = point_xy<VEC>(pts + 2 * p);
                const Corner k = corners_of(sane(xy.x, W), sane(xy.y, H), Hb, W);
                float acc = 0.f;
                for (int c = gl * V; c < C; c += LG * V) {
                    Taps<T, V> t;
                    t.load(img, k, W, C, c);
                    float wc[V];
                    Pack<T, V>::load(wt + c, wc);
#pragma unroll
                    for (int v = 0; v < V; ++v) acc = fmaf(t.value(k, v), wc[v], acc);
                }
                acc = group_sum<LG>(acc);
                if (gl == 0 && own) out[(size_t)inst * P + p] = from_f32<T>(acc);
            }
        }
    }
}

// --------------------------------------------------------------------------- backward
// grad_input must be zero on entry (the host wrapper clears it on the same stream).  It is a sum of reds, whose order, and with it the last
// bits, may change from call to call; the other two gradients repeat bit for bit.
template <typename T, bool POINT, int V, int LG>
__global__ void __launch_bounds__(BA_WARPS * 32)
bilinear_attention_bwd_kernel(const T* __restrict__ grad_out, const T* __restrict__ input, const T* __restrict__ grid,
                              const T* __restrict__ weight, T* __restrict__ grad_input, T* __restrict__ grad_grid,
                              T* __restrict__ grad_weight, int B, int H, int W, int C, int G, int P) {
    constexpr int J = LG == 32 && BA_MAXCH > V ? BA_MAXCH / V : 1;   // channel groups per lane
    constexpr int PW = 32 / LG;                                      // instances per warp
    constexpr bool VEC = V == Vec<T>::N;
    const int lane = threadIdx.x & 31, gl = lane % LG, sub = lane / LG;
    const long long n_inst = (long long)B * G;
    for (long long first = ((long long)blockIdx.x * BA_WARPS + (threadIdx.x >> 5)) * PW; first < n_inst;
         first += (long long)gridDim.x * BA_WARPS * PW) {
        const bool own = first + sub < n_inst;           // a group past the end goes along for the shuffles
        const long long inst = own ? first + sub : first;
        const int Hb = own ? H : 0;                      // and touches no pixel
        const int b = (int)(inst / G);
        const T* img = input + (size_t)b * H * W * C;
        T* gimg = grad_input + (size_t)b * H * W * C;
        const T* pts = grid + (size_t)inst * P * 2;
        // per lane and channel group: the upstream gradient (point mode) or the weight (channel mode),
        // read once, and in channel mode the weight gradient accumulated over the points
        float up[J][V], gw_c[J][V];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int c = (gl + LG * j) * V;
#pragma unroll
            for (int v = 0; v < V; ++v) up[j][v] = gw_c[j][v] = 0.f;
            if (c < C) Pack<T, V>::load((POINT ? grad_out : weight) + (size_t)inst * C + c, up[j]);
        }
        for (int p = 0; p < P; ++p) {
            const float2 xy = point_xy<VEC>(pts + 2 * p);
            const Corner k = corners_of(sane(xy.x, W), sane(xy.y, H), Hb, W);
            // scale turning up[] into g = d(loss) / d(sample(b, p, c))
            const float sc = POINT ? to_f32(weight[(size_t)inst * P + p]) : to_f32(grad_out[(size_t)inst * P + p]);
            // The derivatives are combinations of four sums over the channels, up times the difference of two taps.  (The differences are
            // formed per channel: sums of up times each tap cost four subtractions less, but where neighbouring pixels share most of
            // their value their difference has lost its digits; and each of the four has its own sum, because an edge in
            // the map or its border makes any one of them as small beside the others.)
            float d_xt = 0.f, d_xb = 0.f, d_yl = 0.f, d_yr = 0.f, giw = 0.f;
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const int c = (gl + LG * j) * V;
                if (c < C) {
                    Taps<T, V> t;
                    t.load(img, k, W, C, c);
                    scatter<T, V>(gimg, k, W, C, c, up[j], sc);
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        d_xt = fmaf(up[j][v], t.rt[v] - t.lt[v], d_xt);
                        d_xb = fmaf(up[j][v], t.rb[v] - t.lb[v], d_xb);
                        d_yl = fmaf(up[j][v], t.lb[v] - t.lt[v], d_yl);
                        d_yr = fmaf(up[j][v], t.rb[v] - t.rt[v], d_yr);
                        if (POINT) giw += t.value(k, v) * up[j][v];
                        if (!POINT) gw_c[j][v] += t.value(k, v) * sc;
                    }
                }
            }
            d_xt = group_sum<LG>(d_xt);
            d_xb = group_sum<LG>(d_xb);
            d_yl = group_sum<LG>(d_yl);
            d_yr = group_sum<LG>(d_yr);
            if (POINT) giw = group_sum<LG>(giw);
            // d(sample)/dx and d(sample)/dy of the bilinear form
            const float gix = sc * (d_xt * (1.f - k.ty) + d_xb * k.ty);
            const float giy = sc * (d_yl * (1.f - k.tx) + d_yr * k.tx);
            if (gl == 0 && own) {
                grad_grid[((size_t)inst * P + p) * 2] = from_f32<T>(gix);
                grad_grid[((size_t)inst * P + p) * 2 + 1] = from_f32<T>(giy);
                if (POINT) grad_weight[(size_t)inst * P + p] = from_f32<T>(giw);
            }
        }
        if (!POINT && own) {
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const int c = (gl + LG * j) * V;
                if (c < C) Pack<T, V>::store(grad_weight + (size_t)inst * C + c, gw_c[j]);
            }
        }
    }
}

static int ba_grid(long long instances, int per_warp) {
    const long long want = (instances + BA_WARPS * per_warp - 1) / (BA_WARPS * per_warp);
    const long long cap = (long long)sm_count() * 16;
    return (int)(want < 1 ? 1 : (want < cap ? want : cap));
}

static int ba_check(const char* what, int dtype, int mode, int B, int H, int W, int C, int G, int P) {
    VTP_REQUIRE(dtype == VTP_F32 || dtype == VTP_BF16, VTP_ERR_DTYPE, "%s: dtype %d", what, dtype);
    VTP_REQUIRE(mode == 0 || mode == 1, VTP_ERR_SHAPE, "%s: mode %d (0 = point, 1 = channel)", what, mode);
    VTP_REQUIRE(B > 0 && H > 0 && W > 0 && C > 0 && G > 0 && P > 0, VTP_ERR_SHAPE, "%s: bad shape", what);
    return VTP_OK;
}

struct BaLayout {
    int v, lanes;          // channels per lane, lanes per instance
};

// 16-byte vectors where every row of channels is made of them (C a multiple of 8 bf16 / 4 fp32, channel-indexed
// pointers on 16-byte boundaries, points on pair boundaries), as few lanes per instance as hold C; else pairs of
// channels (even C, pair-aligned pointers) or single channels, with a warp per instance.
static BaLayout ba_layout(int dtype, int C, const void* grid, std::initializer_list<const void*> ptrs) {
    const size_t e = elem_size(dtype);
    uintptr_t low = 0;
    for (const void* p : ptrs) low |= reinterpret_cast<uintptr_t>(p);
    const int v = (int)(16 / e);
    if (C % v == 0 && low % 16 == 0 && reinterpret_cast<uintptr_t>(grid) % (2 * e) == 0)
        return {v, C <= 4 * v ? 4 : C <= 8 * v ? 8 : C <= 16 * v ? 16 : 32};
    return {C % 2 == 0 && low % (2 * e) == 0 ? 2 : 1, 32};
}

// calls F<T, V, LG>() of the layout
#define VTP_BA_DISPATCH(T, NV, F)                                          \
    do {                                                                   \
        if (lay.v == NV && lay.lanes == 4) F(T, NV, 4);                    \
        else if (lay.v == NV && lay.lanes == 8) F(T, NV, 8);               \
        else if (lay.v == NV && lay.lanes == 16) F(T, NV, 16);             \
        else if (lay.v == NV) F(T, NV, 32);                                \
        else if (lay.v == 2) F(T, 2, 32);                                  \
        else F(T, 1, 32);                                                  \
    } while (0)

}  // namespace vtp

using namespace vtp;

static int ba_forward(const void* input, const void* grid, const void* weight, void* out, int dtype, int mode, int B,
                      int H, int W, int C, int G, int P, const long long* batch_of, void* stream) {
    VTP_REQUIRE(input && grid && weight && out, VTP_ERR_NULL, "bilinear_attention: null pointer");
    if (int rc = ba_check("bilinear_attention", dtype, mode, B, H, W, C, G, P)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const BaLayout lay = ba_layout(dtype, C, grid, {input, mode == 0 ? out : weight});
    const int blocks = ba_grid(batch_of ? (long long)G : (long long)B * G, 32 / lay.lanes);
#define VTP_BA_FWD(T, V, LG)                                                                                 \
    (mode == 0 ? bilinear_attention_fwd_kernel<T, true, V, LG> : bilinear_attention_fwd_kernel<T, false, V, LG>) \
        <<<blocks, BA_WARPS * 32, 0, st>>>((const T*)input, (const T*)grid, (const T*)weight, (T*)out, B, H, W, C, G, P, batch_of)
    if (dtype == VTP_F32) VTP_BA_DISPATCH(float, 4, VTP_BA_FWD);
    else VTP_BA_DISPATCH(bf16, 8, VTP_BA_FWD);
#undef VTP_BA_FWD
    return check_launch("bilinear_attention_forward");
}

extern "C" int vtp_bilinear_attention_forward(const void* input, const void* grid, const void* weight, void* out,
                                              int dtype, int mode, int B, int H, int W, int C, int G, int P,
                                              void* stream) {
    return ba_forward(input, grid, weight, out, dtype, mode, B, H, W, C, G, P, nullptr, stream);
}

extern "C" int vtp_sparse_bilinear_attention_forward(const void* input, const void* grid, const void* weight,
                                                     const long long* batches, void* out, int dtype, int B, int H,
                                                     int W, int C, int L, int P, void* stream) {
    VTP_REQUIRE(batches, VTP_ERR_NULL, "sparse_bilinear_attention: null batches");
    if (L == 0) return VTP_OK;
    return ba_forward(input, grid, weight, out, dtype, 0, B, H, W, C, L, P, batches, stream);
}

extern "C" int vtp_bilinear_attention_backward(const void* grad_out, const void* input, const void* grid,
                                               const void* weight, void* grad_input, void* grad_grid,
                                               void* grad_weight, int dtype, int mode, int B, int H, int W, int C,
                                               int G, int P, void* stream) {
    VTP_REQUIRE(grad_out && input && grid && weight && grad_input && grad_grid && grad_weight, VTP_ERR_NULL,
                "bilinear_attention_backward: null pointer");
    if (int rc = ba_check("bilinear_attention_backward", dtype, mode, B, H, W, C, G, P)) return rc;
    VTP_REQUIRE(C <= 32 * BA_MAXCH, VTP_ERR_SHAPE, "bilinear_attention_backward: C=%d above %d", C, 32 * BA_MAXCH);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemsetAsync(grad_input, 0, (size_t)B * H * W * C * elem_size(dtype), st);
    if (e != cudaSuccess) return fail((int)e, "bilinear_attention_backward: clearing grad_input: %s", cudaGetErrorString(e));
    const BaLayout lay = mode == 0 ? ba_layout(dtype, C, grid, {input, grad_input, grad_out})
                                   : ba_layout(dtype, C, grid, {input, grad_input, weight, grad_weight});
    const int blocks = ba_grid((long long)B * G, 32 / lay.lanes);
#define VTP_BA_BWD(T, V, LG)                                                                                 \
    (mode == 0 ? bilinear_attention_bwd_kernel<T, true, V, LG> : bilinear_attention_bwd_kernel<T, false, V, LG>) \
        <<<blocks, BA_WARPS * 32, 0, st>>>((const T*)grad_out, (const T*)input, (const T*)grid, (const T*)weight, \
                                           (T*)grad_input, (T*)grad_grid, (T*)grad_weight, B, H, W, C, G, P)
    if (dtype == VTP_F32) VTP_BA_DISPATCH(float, 4, VTP_BA_BWD);
    else VTP_BA_DISPATCH(bf16, 8, VTP_BA_BWD);
#undef VTP_BA_BWD
    return check_launch("bilinear_attention_backward");
}
