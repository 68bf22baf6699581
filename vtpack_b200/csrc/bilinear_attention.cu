// Bilinear-sampling attention of the deformable PVT (vtpack/models/standard/dpvt.py:92-115):
// every query position g of a feature map [B, H, W, C] looks at P sampling points given in pixel
// coordinates (x, y), reads the map there by bilinear interpolation (zero outside the map) and
//   "point"   mode: out[b,g,c] = sum_p weight[b,g,p] * sample(b, p, c)         weight [B,G,P]
//   "channel" mode: out[b,g,p] = sum_c weight[b,g,c] * sample(b, p, c)         weight [B,G,C]
// Replaces bilinear_attention_{pointwise,channelwise}_{forward,backward}
// (vtpack/layers/csrc/bilinear_attention/bilinear_attention.cu:88-132, :134-232, :234-268, :270-362).
//
// The reference runs one thread per (b, g) that walks the channels serially, so neighbouring threads read addresses
// C elements apart.  Here, where rows are made of 16-byte vectors (8 bf16 / 4 fp32 channels), a group of lanes owns a (b, g) instance
// and each lane one to three vectors of its channels (bilinear_vectors_*_kernel); else a warp owns it and a lane takes pairs of channels or single ones
// (bilinear_attention_*_kernel).  A point's corner arithmetic and the reductions over the channels are then paid once per lane instead of
// once per channel pair, and the input gradient leaves as one vector red per corner and vector.
//
// Measured on 32 maps of 64 x 64 x 64, 9 points, bf16, point mode, forward / backward us: a warp per instance with a channel pair per lane, forward and
// backward together 525; a vector a lane 71 / 163; with derivatives from four dot products and taps outside the map as zeroed raw words
// 65 / 141 (issue slots 80 % busy in both).  Then, with the same sums: arithmetic on pairs of channels, taps outside the map read from
// a vector of zeros instead of conditional loads, no 64-bit division, tiles of pixels, launch bounds for 20 warps a SM and more:
// 56 / 124; two vectors a lane 45 / 134 (the rule for it is at bv_shape); 50 forward without the tiles.
// Bound: forward the issue slots; backward the reds, 604 MB that L2 takes at 5.6 TB/s (108 us when nothing else runs; bulk reductions of 256 bytes
// from shared memory arrive at the same rate); DRAM 5 %.
// Tried and not kept: contiguous query ranges per SM (71 -> 76 / 163 -> 157), a point's corners worked out by one lane and handed round by
// shuffles (78 / 159), two points at a time (45 -> 47), 8 or 2 warps a block (49 / 137, 47 / 137); and what is faster and less
// exact, relative errors in fp32: the corners' weights times the point's in front of the channels (6.0e-8 -> 7.8e-8), derivatives from sums of
// taps (point gradients of a map with an offset of 100 7.9e-8 -> 6.8e-6), weight gradients from one tap's sum and the differences' (8.2e-8
// -> 1.6e-7).
#include <initializer_list>

#include "bilinear_attention.cuh"

namespace vtp {

constexpr int BA_WARPS = 8;           // warps per block
constexpr int BA_MAXCH = 8;           // widest C of the backward / 32: a lane keeps its weight gradients in registers

// V consecutive channels per lane: 16 bytes (forward, rows wider than the vector kernels take), or one pair / one channel where the rows are
// not made of 16-byte vectors
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

// ---------------------------------------------------------------------------- forward
template <typename T, bool POINT, int V>
__global__ void __launch_bounds__(BA_WARPS * 32)
bilinear_attention_fwd_kernel(const T* __restrict__ input, const T* __restrict__ grid, const T* __restrict__ weight,
                              T* __restrict__ out, int B, int H, int W, int C, int G, int P,
                              const long long* __restrict__ batch_of) {
    // batch_of == null: B * G instances, G per image; else G packed instances, instance i reads image batch_of[i]
    constexpr bool VEC = V == Vec<T>::N;
    const int lane = threadIdx.x & 31;
    const long long n_inst = batch_of ? (long long)G : (long long)B * G;
    for (long long inst = (long long)blockIdx.x * BA_WARPS + (threadIdx.x >> 5); inst < n_inst; inst += (long long)gridDim.x * BA_WARPS) {
        long long b = batch_of ? batch_of[inst] : inst / G;
        const bool image_ok = b >= 0 && b < B;           // an instance naming no image reads zeros
        if (!image_ok) b = 0;
        const int Hb = image_ok ? H : 0;                 // no pixel is in bounds
        const T* img = input + (size_t)b * H * W * C;
        const T* pts = grid + (size_t)inst * P * 2;
        if (POINT) {
            const T* wt = weight + (size_t)inst * P;
            for (int c = lane * V; c < C; c += 32 * V) {
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
                Pack<T, V>::store(out + (size_t)inst * C + c, acc);
            }
        } else {
            const T* wt = weight + (size_t)inst * C;
            for (int p = 0; p < P; ++p) {
                const float2 xy = point_xy<VEC>(pts + 2 * p);
                const Corner k = corners_of(sane(xy.x, W), sane(xy.y, H), Hb, W);
                float acc = 0.f;
                for (int c = lane * V; c < C; c += 32 * V) {
                    Taps<T, V> t;
                    t.load(img, k, W, C, c);
                    float wc[V];
                    Pack<T, V>::load(wt + c, wc);
#pragma unroll
                    for (int v = 0; v < V; ++v) acc = fmaf(t.value(k, v), wc[v], acc);
                }
                acc = warp_sum(acc);
                if (lane == 0) out[(size_t)inst * P + p] = from_f32<T>(acc);
            }
        }
    }
}

// --------------------------------------------------------------------------- backward
// grad_input must be zero on entry (the host wrapper clears it on the same stream).  It is a sum of reds, whose order, and with it the last
// bits, may change from call to call; the other two gradients repeat bit for bit.
template <typename T, bool POINT, int V>
__global__ void __launch_bounds__(BA_WARPS * 32)
bilinear_attention_bwd_kernel(const T* __restrict__ grad_out, const T* __restrict__ input, const T* __restrict__ grid,
                              const T* __restrict__ weight, T* __restrict__ grad_input, T* __restrict__ grad_grid,
                              T* __restrict__ grad_weight, int B, int H, int W, int C, int G, int P) {
    constexpr int J = BA_MAXCH > V ? BA_MAXCH / V : 1;               // channel groups per lane
    constexpr bool VEC = V == Vec<T>::N;
    const int lane = threadIdx.x & 31;
    const long long n_inst = (long long)B * G;
    for (long long inst = (long long)blockIdx.x * BA_WARPS + (threadIdx.x >> 5); inst < n_inst; inst += (long long)gridDim.x * BA_WARPS) {
        const int b = (int)(inst / G);
        const T* img = input + (size_t)b * H * W * C;
        T* gimg = grad_input + (size_t)b * H * W * C;
        const T* pts = grid + (size_t)inst * P * 2;
        // per lane and channel group: the upstream gradient (point mode) or the weight (channel mode),
        // read once, and in channel mode the weight gradient accumulated over the points
        float up[J][V], gw_c[J][V];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int c = (lane + 32 * j) * V;
#pragma unroll
            for (int v = 0; v < V; ++v) up[j][v] = gw_c[j][v] = 0.f;
            if (c < C) Pack<T, V>::load((POINT ? grad_out : weight) + (size_t)inst * C + c, up[j]);
        }
        for (int p = 0; p < P; ++p) {
            const float2 xy = point_xy<VEC>(pts + 2 * p);
            const Corner k = corners_of(sane(xy.x, W), sane(xy.y, H), H, W);
            // scale turning up[] into g = d(loss) / d(sample(b, p, c))
            const float sc = POINT ? to_f32(weight[(size_t)inst * P + p]) : to_f32(grad_out[(size_t)inst * P + p]);
            // The derivatives are combinations of four sums over the channels, up times the difference of two taps.  (The differences are
            // formed per channel: sums of up times each tap cost four subtractions less, but where neighbouring pixels share most of
            // their value their difference has lost its digits; and each of the four has its own sum, because an edge in
            // the map or its border makes any one of them as small beside the others.)
            float d_xt = 0.f, d_xb = 0.f, d_yl = 0.f, d_yr = 0.f, giw = 0.f;
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const int c = (lane + 32 * j) * V;
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
            d_xt = warp_sum(d_xt);
            d_xb = warp_sum(d_xb);
            d_yl = warp_sum(d_yl);
            d_yr = warp_sum(d_yr);
            if (POINT) giw = warp_sum(giw);
            // d(sample)/dx and d(sample)/dy of the bilinear form
            const float gix = sc * (d_xt * (1.f - k.ty) + d_xb * k.ty);
            const float giy = sc * (d_yl * (1.f - k.tx) + d_yr * k.tx);
            if (lane == 0) {
                grad_grid[((size_t)inst * P + p) * 2] = from_f32<T>(gix);
                grad_grid[((size_t)inst * P + p) * 2 + 1] = from_f32<T>(giy);
                if (POINT) grad_weight[(size_t)inst * P + p] = from_f32<T>(giw);
            }
        }
        if (!POINT) {
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const int c = (lane + 32 * j) * V;
                if (c < C) Pack<T, V>::store(grad_weight + (size_t)inst * C + c, gw_c[j]);
            }
        }
    }
}

static int ba_grid(long long instances, int sms) {
    const long long want = (instances + BA_WARPS - 1) / BA_WARPS;
    const long long cap = (long long)sms * 16;
    return (int)(want < 1 ? 1 : (want < cap ? want : cap));
}

static int ba_check(const char* what, int dtype, int mode, int B, int H, int W, int C, int G, int P) {
    VTP_REQUIRE(dtype == VTP_F32 || dtype == VTP_BF16, VTP_ERR_DTYPE, "%s: dtype %d", what, dtype);
    VTP_REQUIRE(mode == 0 || mode == 1, VTP_ERR_SHAPE, "%s: mode %d (0 = point, 1 = channel)", what, mode);
    VTP_REQUIRE(B > 0 && H > 0 && W > 0 && C > 0 && G > 0 && P > 0, VTP_ERR_SHAPE, "%s: bad shape", what);
    return VTP_OK;
}

// Channels of a load: 16 bytes where every row of channels is made of them (C a multiple of 8 bf16 / 4 fp32, channel-indexed
// pointers on 16-byte boundaries, points on pair boundaries); else a pair (even C, pair-aligned pointers) or one.
static int channels_of_a_load(int dtype, int C, const void* grid, std::initializer_list<const void*> ptrs) {
    const size_t e = elem_size(dtype);
    uintptr_t low = 0;
    for (const void* p : ptrs) low |= reinterpret_cast<uintptr_t>(p);
    const int v = (int)(16 / e);
    if (C % v == 0 && low % 16 == 0 && reinterpret_cast<uintptr_t>(grid) % (2 * e) == 0) return v;
    return C % 2 == 0 && low % (2 * e) == 0 ? 2 : 1;
}

// Lanes of a group and vectors of a lane; lanes == 0: not for bilinear_vectors_*_kernel.
// One vector where queries are few (a lane's chain is shorter, and there are more warps: below 16 a SM).  Else the fewest slots, as a
// slot without channels costs like any other, and of these two vectors a lane, in the backward only where a group still covers 128 bytes: its reds of
// 64 bytes are slower than its arithmetic is quicker.  In fp32, where a vector is half as much arithmetic, the backward takes several
// a lane in groups of eight lanes and more only, two a lane for rows of more than 12 (in groups of eight from a hundred warps a SM on); a forward of
// rows of four keeps one a lane.
// us, forward / backward, point mode, of 32 maps of 64 x 64, 9 points (in brackets backward of 24 of 22 x 48, 5 points):
//   bf16   4 vectors   2 x 2   25.7 /             4 x 1   29.0 /  72 (13)
//          8           4 x 2   43.9 / 131 (22)    8 x 1   54.6 / 120 (18)
//         12           4 x 3   63.3 / 194 (30)    8 x 2   83.5 / 210 (29)   16 x 1  106.4 / 240 (30)
//         24           8 x 3  133   / 339 (42)   16 x 2  174   / 426 (50)   32 x 1  210   / 478 (55)
//   fp32   4 vectors   2 x 2   27.3 /             4 x 1   23.8 /  73 (12)
//         12           4 x 3   57.0 / 194 (35)    8 x 2   70.3 / 184 (25)   16 x 1   84.4 / 189 (24)
//         16           8 x 2   74.3 / 208 (27)   16 x 1   85.6 / 222 (26)
//         24           8 x 3  111   / 304 (42)   16 x 2  133   / 331 (39)   32 x 1  169   / 362 (42)
// 4 maps of 28 x 28, 8 vectors in bf16, 5 points 8 x 1 3.9 / 7.0, 4 x 2 4.8 / 8.5; 64 of 14 x 14, 16 vectors in fp32, 4 points, channel mode
// 16 x 1 6.6 / 13.3, 8 x 2 5.7 / 14.1.
static BvShape bv_shape(int v, int dtype, int C, int H, int W, long long n_inst, bool grads, int sms) {
    const int n = C / v;
    if (v * elem_size(dtype) != 16 || n > BV_MAXVEC || n_inst > (1ll << 30) || (long long)H * W > (1ll << 30)) return {0, 0};
    BvShape best{4, 1};
    while (best.lanes < n && best.lanes < 32) best.lanes *= 2;
    if (best.lanes < n) return {32, 2};
    const bool f32 = dtype == VTP_F32;
    for (int j = 2; j <= 3; ++j) {
        int lanes = !grads ? 2 : f32 ? 8 : 4;
        while (lanes * j < n) lanes *= 2;
        const long long warps = n_inst * lanes / 32;
        if (n < 3 || lanes > 16 || warps < 16ll * sms) continue;
        const int slots = lanes * j, least = best.lanes * best.vecs;
        const bool pays = !grads ? !f32 || n > 4 : !f32 ? lanes >= 8 : n > 12 && (lanes > 8 || warps >= 100ll * sms);
        if (slots < least || (slots == least && best.vecs == 1 && pays)) best = {lanes, j};
    }
    return best;
}

static void bv_run(const BvArgs& a, const BvShape& s, int dtype, int mode, bool grads, cudaStream_t st) {
    if (dtype == VTP_F32) bilinear_vectors<float>(a, s, mode == 0, grads, st);
    else bilinear_vectors<bf16>(a, s, mode == 0, grads, st);
}
static BvArgs bv_args(const void* input, const void* grid, const void* weight, int dtype, int B, int H, int W, int C, int G, int P, long long n,
                      int sms) {
    BvArgs a{};
    a.input = (const char*)input; a.grid = (const char*)grid; a.weight = (const char*)weight;
    a.B = B; a.H = H; a.W = W; a.G = G; a.P = P; a.n_inst = (int)n; a.most_blocks = 32 * sms;
    a.row = (int)(C * elem_size(dtype)); a.vecs = a.row / 16;
    a.per_image = make_fast_div((uint32_t)G);
    return a;
}

}  // namespace vtp

using namespace vtp;

static int ba_forward(const void* input, const void* grid, const void* weight, void* out, int dtype, int mode, int B,
                      int H, int W, int C, int G, int P, const long long* batch_of, void* stream) {
    VTP_REQUIRE(input && grid && weight && out, VTP_ERR_NULL, "bilinear_attention: null pointer");
    if (int rc = ba_check("bilinear_attention", dtype, mode, B, H, W, C, G, P)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int v = channels_of_a_load(dtype, C, grid, {input, mode == 0 ? out : weight}), sms = sm_count();
    const long long n_inst = batch_of ? (long long)G : (long long)B * G;
    if (const BvShape shape = bv_shape(v, dtype, C, H, W, n_inst, false, sms); shape.lanes) {
        BvArgs a = bv_args(input, grid, weight, dtype, B, H, W, C, G, P, n_inst, sms);
        a.out = (char*)out;
        a.batch_of = batch_of;
        bv_run(a, shape, dtype, mode, false, st);
        return check_launch("bilinear_attention_forward");
    }
    const int blocks = ba_grid(n_inst, sms);
#define VTP_BA_FWD(T, V)                                                                                 \
    (mode == 0 ? bilinear_attention_fwd_kernel<T, true, V> : bilinear_attention_fwd_kernel<T, false, V>) \
        <<<blocks, BA_WARPS * 32, 0, st>>>((const T*)input, (const T*)grid, (const T*)weight, (T*)out, B, H, W, C, G, P, batch_of)
#define VTP_BA_TYPED(F, T, N) v == N ? F(T, N) : v == 2 ? F(T, 2) : F(T, 1)
    if (dtype == VTP_F32) VTP_BA_TYPED(VTP_BA_FWD, float, 4);
    else VTP_BA_TYPED(VTP_BA_FWD, bf16, 8);
#undef VTP_BA_TYPED
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
    const int v = mode == 0 ? channels_of_a_load(dtype, C, grid, {input, grad_input, grad_out})
                            : channels_of_a_load(dtype, C, grid, {input, grad_input, weight, grad_weight}), sms = sm_count();
    if (const BvShape shape = bv_shape(v, dtype, C, H, W, (long long)B * G, true, sms); shape.lanes) {
        BvArgs a = bv_args(input, grid, weight, dtype, B, H, W, C, G, P, (long long)B * G, sms);
        a.grad_out = (const char*)grad_out;
        a.grad_input = (char*)grad_input; a.grad_grid = (char*)grad_grid; a.grad_weight = (char*)grad_weight;
        bv_run(a, shape, dtype, mode, true, st);
        return check_launch("bilinear_attention_backward");
    }
    const int blocks = ba_grid((long long)B * G, sms);
#define VTP_BA_BWD(T, V)                                                                                 \
    (mode == 0 ? bilinear_attention_bwd_kernel<T, true, V> : bilinear_attention_bwd_kernel<T, false, V>) \
        <<<blocks, BA_WARPS * 32, 0, st>>>((const T*)grad_out, (const T*)input, (const T*)grid, (const T*)weight, \
                                           (T*)grad_input, (T*)grad_grid, (T*)grad_weight, B, H, W, C, G, P)
    // (whole vectors only come here beyond 2^30 queries or pixels: as pairs)
    if (dtype == VTP_F32) v == 1 ? VTP_BA_BWD(float, 1) : VTP_BA_BWD(float, 2);
    else v == 1 ? VTP_BA_BWD(bf16, 1) : VTP_BA_BWD(bf16, 2);
#undef VTP_BA_BWD
    return check_launch("bilinear_attention_backward");
}
