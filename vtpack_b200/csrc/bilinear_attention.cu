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

#include "common.cuh"
#include "linear.h"

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

// ------------------------------------------------------------- rows of 16-byte vectors
// A group of LG lanes owns an instance, a lane J vectors of its channels: the arithmetic of a point's corners, which every lane of a
// group repeats, is paid once per J of them.
constexpr int BV_WARPS = 4;

template <typename T> struct Quad;                  // 16 bytes as pairs of channels
template <> struct Quad<float> {
    static constexpr int NP = 2;
    uint4 raw;
    __device__ __forceinline__ float2 pair(int i) const {
        return i ? make_float2(__uint_as_float(raw.z), __uint_as_float(raw.w)) : make_float2(__uint_as_float(raw.x), __uint_as_float(raw.y));
    }
    __device__ __forceinline__ void set(const float2 (&f)[NP]) {
        raw = make_uint4(__float_as_uint(f[0].x), __float_as_uint(f[0].y), __float_as_uint(f[1].x), __float_as_uint(f[1].y));
    }
};
template <> struct Quad<bf16> {
    static constexpr int NP = 4;
    uint4 raw;
    __device__ __forceinline__ float2 pair(int i) const {
        const uint32_t v = i == 0 ? raw.x : i == 1 ? raw.y : i == 2 ? raw.z : raw.w;
        return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    }
    static __device__ __forceinline__ uint32_t word(float2 f) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
    __device__ __forceinline__ void set(const float2 (&f)[NP]) { raw = make_uint4(word(f[0]), word(f[1]), word(f[2]), word(f[3])); }
};
template <typename T> __device__ __forceinline__ Quad<T> quad_at(const char* p) { return Quad<T>{*reinterpret_cast<const uint4*>(p)}; }
__device__ __forceinline__ void red_quad(char* p, const Quad<float>& v) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.pair(0).x), "f"(v.pair(0).y), "f"(v.pair(1).x),
                 "f"(v.pair(1).y));
}
__device__ __forceinline__ void red_quad(char* p, const Quad<bf16>& v) {
    asm volatile("red.relaxed.gpu.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.raw.x), "r"(v.raw.y), "r"(v.raw.z),
                 "r"(v.raw.w));
}

// What a corner outside the map is read from: the loads need no condition, and no zeros in front of them.
constexpr int BV_MAXVEC = 64;
__device__ const __align__(16) uint4 g_no_pixel[BV_MAXVEC] = {};

struct BvArgs {
    const char *input, *grid, *weight, *grad_out;
    char *out, *grad_input, *grad_grid, *grad_weight;
    const long long* batch_of;
    int B, H, W, G, P, n_inst;
    int row, vecs;                                  // bytes and 16-byte vectors of a row of channels
    FastDiv per_image;                              // G
    FastDiv tile_rows, tiles;                       // tiles of a row of tiles (d = 0: no tiles) and of a map
    int units;                                      // pieces of work, one block each
};

// Which of its J vectors a lane takes j-th: groups that read less than the 128 bytes of all banks at a time start on different ones.
template <int LG, int J>
__device__ __forceinline__ int bv_turn(int j, int sub) { return LG < 8 ? (j + sub) % J : j; }

// A lane's query.  Where the queries are the pixels of the map (as many of them, in order), a block takes a tile of them, PW wide and
// a row a warp, because their points are near them and what they read is then near too; else it takes PW consecutive ones a warp.
template <int PW>
struct BvPlace {
    int inst, Hb;
    bool own;
    long long map;                                  // byte of the map in input
    __device__ __forceinline__ BvPlace(const BvArgs& a, int unit, int sub, bool grads) {
        const int warp = (int)threadIdx.x >> 5;
        long long b;
        if (a.tile_rows.d) {
            const uint32_t img = fast_div((uint32_t)unit, a.tiles), t = unit - img * a.tiles.d;
            const uint32_t ty = fast_div(t, a.tile_rows), tx = t - ty * a.tile_rows.d;
            const int x = (int)tx * PW + sub, y = (int)ty * BV_WARPS + warp;
            own = x < a.W && y < a.H;               // a group past the end goes along for the shuffles
            b = img;
            inst = (int)img * a.G + (own ? y * a.W + x : 0);
        } else {
            const int i = (unit * BV_WARPS + warp) * PW + sub;
            own = i < a.n_inst;
            inst = own ? i : 0;
            b = a.batch_of ? a.batch_of[inst] : (long long)fast_div((uint32_t)inst, a.per_image);
        }
        const bool ok = b >= 0 && b < a.B;          // an instance naming no image reads zeros
        if (!ok) b = 0;
        Hb = ok && (own || !grads) ? a.H : 0;       // no pixel is in bounds
        map = b * a.H * a.W * a.row;
    }
};

struct BvTaps {
    const char* at[4];                              // lt, rt, lb, rb
    __device__ __forceinline__ BvTaps(const char* px, const Corner& k, int W, int row, const char* none) {
        const char* lt = px + (long long)(k.y0 * W + k.x0) * row;
        const long long down = (long long)W * row;
        at[0] = k.in_lt ? lt : none;
        at[1] = k.in_rt ? lt + row : none;
        at[2] = k.in_lb ? lt + down : none;
        at[3] = k.in_rb ? lt + down + row : none;
    }
};

template <typename T, bool POINT, int LG, int J>
__global__ void __launch_bounds__(BV_WARPS * 32, J == 1 ? 8 : J == 2 ? 7 : 6)
bilinear_vectors_fwd_kernel(const __grid_constant__ BvArgs a) {
    constexpr int PW = 32 / LG, NP = Quad<T>::NP;
    const int lane = threadIdx.x & 31, gl = lane % LG, sub = lane / LG;
    int c[J];
    bool has[J];
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const int v = bv_turn<LG, J>(j, sub) * LG + gl;
        c[j] = v * 16;
        has[j] = v < a.vecs;
    }
    const char* none = reinterpret_cast<const char*>(g_no_pixel);
    for (int unit = blockIdx.x; unit < a.units; unit += gridDim.x) {
        const BvPlace<PW> at(a, unit, sub, false);
        const char* px = a.input + at.map;
        const T* pts = reinterpret_cast<const T*>(a.grid) + (size_t)at.inst * a.P * 2;
        const T* wt = reinterpret_cast<const T*>(a.weight) + (size_t)at.inst * a.P;        // (point mode)
        float2 sum[J][NP];                          // point: the output; channel: the weights
#pragma unroll
        for (int j = 0; j < J; ++j) {
            Quad<T> w{};
            if (!POINT && has[j]) w = quad_at<T>(a.weight + (size_t)at.inst * a.row + c[j]);
#pragma unroll
            for (int i = 0; i < NP; ++i) sum[j][i] = w.pair(i);
        }
#pragma unroll 1
        for (int p = 0; p < a.P; ++p) {
            const float2 xy = point_xy<true>(pts + 2 * p);
            const Corner k = corners_of(sane(xy.x, a.W), sane(xy.y, a.H), at.Hb, a.W);
            const BvTaps t(px, k, a.W, a.row, none);
            const float2 wp = both(POINT ? to_f32(wt[p]) : 0.f);
            float2 dot = both(0.f);
#pragma unroll
            for (int j = 0; j < J; ++j) {
                if (!has[j]) continue;
                Quad<T> q[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) q[i] = quad_at<T>(t.at[i] + c[j]);
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    const float2 v = fma2(both(k.w_rb), q[3].pair(i), fma2(both(k.w_lb), q[2].pair(i),
                                          fma2(both(k.w_rt), q[1].pair(i), mul2(both(k.w_lt), q[0].pair(i)))));
                    if (POINT) sum[j][i] = fma2(v, wp, sum[j][i]);
                    else dot = fma2(v, sum[j][i], dot);
                }
            }
            if (!POINT) {
                const float s = group_sum<LG>(dot.x + dot.y);
                if (gl == 0 && at.own) reinterpret_cast<T*>(a.out)[(size_t)at.inst * a.P + p] = from_f32<T>(s);
            }
        }
        if (POINT && at.own) {
#pragma unroll
            for (int j = 0; j < J; ++j) {
                Quad<T> o;
                o.set(sum[j]);
                if (has[j]) *reinterpret_cast<uint4*>(a.out + (size_t)at.inst * a.row + c[j]) = o.raw;
            }
        }
    }
}

// (see bilinear_attention_bwd_kernel)
template <typename T, bool POINT, int LG, int J>
__global__ void __launch_bounds__(BV_WARPS * 32, J == 3 ? 4 : 5)
bilinear_vectors_bwd_kernel(const __grid_constant__ BvArgs a) {
    constexpr int PW = 32 / LG, NP = Quad<T>::NP;
    const int lane = threadIdx.x & 31, gl = lane % LG, sub = lane / LG;
    int c[J];
    bool has[J];
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const int v = bv_turn<LG, J>(j, sub) * LG + gl;
        c[j] = v * 16;
        has[j] = v < a.vecs;
    }
    const char* none = reinterpret_cast<const char*>(g_no_pixel);
    for (int unit = blockIdx.x; unit < a.units; unit += gridDim.x) {
        const BvPlace<PW> at(a, unit, sub, true);
        const char* px = a.input + at.map;
        char* gpx = a.grad_input + at.map;
        const T* pts = reinterpret_cast<const T*>(a.grid) + (size_t)at.inst * a.P * 2;
        const T* per_point = reinterpret_cast<const T*>(POINT ? a.weight : a.grad_out) + (size_t)at.inst * a.P;
        float2 up[J][NP], gw[POINT ? 1 : J][NP];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            Quad<T> u{};
            if (has[j]) u = quad_at<T>((POINT ? a.grad_out : a.weight) + (size_t)at.inst * a.row + c[j]);
#pragma unroll
            for (int i = 0; i < NP; ++i) up[j][i] = u.pair(i);
        }
#pragma unroll
        for (int j = 0; j < (POINT ? 1 : J); ++j)
#pragma unroll
            for (int i = 0; i < NP; ++i) gw[j][i] = both(0.f);
#pragma unroll 1
        for (int p = 0; p < a.P; ++p) {
            const float2 xy = point_xy<true>(pts + 2 * p);
            const Corner k = corners_of(sane(xy.x, a.W), sane(xy.y, a.H), at.Hb, a.W);
            const BvTaps t(px, k, a.W, a.row, none);
            const float sc = to_f32(per_point[p]);
            float2 d_xt = both(0.f), d_xb = both(0.f), d_yl = both(0.f), d_yr = both(0.f), giw = both(0.f);
            char* g = gpx + (long long)(k.y0 * a.W + k.x0) * a.row;
            const long long down = (long long)a.W * a.row;
#pragma unroll
            for (int j = 0; j < J; ++j) {
                if (!has[j]) continue;
                Quad<T> q[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) q[i] = quad_at<T>(t.at[i] + c[j]);
#define BV_RED(IN, OFF, WT)                                                               \
                if (IN) {                                                                 \
                    float2 s[NP];                                                         \
                    const float w = sc * (WT);                                            \
                    _Pragma("unroll") for (int i = 0; i < NP; ++i) s[i] = mul2(up[j][i], both(w)); \
                    Quad<T> r;                                                            \
                    r.set(s);                                                             \
                    red_quad(g + (OFF) + c[j], r);                                        \
                }
                BV_RED(k.in_lt, 0, k.w_lt)
                BV_RED(k.in_rt, a.row, k.w_rt)
                BV_RED(k.in_lb, down, k.w_lb)
                BV_RED(k.in_rb, down + a.row, k.w_rb)
#undef BV_RED
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    const float2 lt = q[0].pair(i), rt = q[1].pair(i), lb = q[2].pair(i), rb = q[3].pair(i), u = up[j][i];
                    d_xt = fma2(u, sub2(rt, lt), d_xt);
                    d_xb = fma2(u, sub2(rb, lb), d_xb);
                    d_yl = fma2(u, sub2(lb, lt), d_yl);
                    d_yr = fma2(u, sub2(rb, rt), d_yr);
                    const float2 v = fma2(both(k.w_rb), rb, fma2(both(k.w_lb), lb, fma2(both(k.w_rt), rt, mul2(both(k.w_lt), lt))));
                    if (POINT) giw = fma2(v, u, giw);
                    else gw[j][i] = fma2(v, both(sc), gw[j][i]);
                }
            }
            const float xt = group_sum<LG>(d_xt.x + d_xt.y), xb = group_sum<LG>(d_xb.x + d_xb.y);
            const float yl = group_sum<LG>(d_yl.x + d_yl.y), yr = group_sum<LG>(d_yr.x + d_yr.y);
            const float gi = POINT ? group_sum<LG>(giw.x + giw.y) : 0.f;
            const float gix = sc * (xt * (1.f - k.ty) + xb * k.ty);
            const float giy = sc * (yl * (1.f - k.tx) + yr * k.tx);
            if (gl == 0 && at.own) {
                T* gg = reinterpret_cast<T*>(a.grad_grid) + ((size_t)at.inst * a.P + p) * 2;
                gg[0] = from_f32<T>(gix);
                gg[1] = from_f32<T>(giy);
                if (POINT) reinterpret_cast<T*>(a.grad_weight)[(size_t)at.inst * a.P + p] = from_f32<T>(gi);
            }
        }
        if (!POINT && at.own) {
#pragma unroll
            for (int j = 0; j < J; ++j) {
                Quad<T> o;
                o.set(gw[POINT ? 0 : j]);
                if (has[j]) *reinterpret_cast<uint4*>(a.grad_weight + (size_t)at.inst * a.row + c[j]) = o.raw;
            }
        }
    }
}

static int ba_grid(long long instances) {
    const long long want = (instances + BA_WARPS - 1) / BA_WARPS;
    const long long cap = (long long)sm_count() * 16;
    return (int)(want < 1 ? 1 : (want < cap ? want : cap));
}

static int ba_check(const char* what, int dtype, int mode, int B, int H, int W, int C, int G, int P) {
    VTP_REQUIRE(dtype == VTP_F32 || dtype == VTP_BF16, VTP_ERR_DTYPE, "%s: dtype %d", what, dtype);
    VTP_REQUIRE(mode == 0 || mode == 1, VTP_ERR_SHAPE, "%s: mode %d (0 = point, 1 = channel)", what, mode);
    VTP_REQUIRE(B > 0 && H > 0 && W > 0 && C > 0 && G > 0 && P > 0, VTP_ERR_SHAPE, "%s: bad shape", what);
    return VTP_OK;
}

struct BaLayout { int v; };          // channels of a load

// 16-byte vectors where every row of channels is made of them (C a multiple of 8 bf16 / 4 fp32, channel-indexed
// pointers on 16-byte boundaries, points on pair boundaries); else pairs of
// channels (even C, pair-aligned pointers) or single channels.
static BaLayout ba_layout(int dtype, int C, const void* grid, std::initializer_list<const void*> ptrs) {
    const size_t e = elem_size(dtype);
    uintptr_t low = 0;
    for (const void* p : ptrs) low |= reinterpret_cast<uintptr_t>(p);
    const int v = (int)(16 / e);
    if (C % v == 0 && low % 16 == 0 && reinterpret_cast<uintptr_t>(grid) % (2 * e) == 0) return {v};
    return {C % 2 == 0 && low % (2 * e) == 0 ? 2 : 1};
}

// calls F<T, V>() of the layout, a warp per instance
#define VTP_BA_DISPATCH(T, NV, F)                                          \
    do {                                                                   \
        if (lay.v == NV) F(T, NV);                                         \
        else if (lay.v == 2) F(T, 2);                                      \
        else F(T, 1);                                                      \
    } while (0)

// Lanes of a group and vectors of a lane; lanes == 0: not for bilinear_vectors_*_kernel.
// One vector where queries are few (a lane's chain is shorter, and there are more warps: below 16 a SM).  Else the fewest slots, as a
// slot without channels costs like any other, and of these two vectors a lane, in the backward only where a group still covers 128 bytes: its reds of
// 64 bytes are slower than its arithmetic is quicker.  us, forward / backward of 32 maps of 64 x 64, 9 points, point mode, one | two vectors:
// bf16 C = 64 56 / 124 | 45 / 134, C = 32 31 / 75 | 27 / 105, fp32 C = 64 86 / 224 | 74 / 209; 16 maps, C = 96 bf16, 5 points 35 / 74 | three vectors
// 23 / 61; 4 maps of 28 x 28, C = 64 bf16 6.4 / 13.4 | 8.5 / 15.2, 16 maps in fp32 12.6 / 29.9 | 11.5 / 29.5.
struct BvShape { int lanes, vecs; };
static BvShape bv_shape(const BaLayout& lay, int dtype, int C, int H, int W, long long n_inst, bool grads) {
    const int n = C / lay.v;
    if (lay.v * elem_size(dtype) != 16 || n > BV_MAXVEC || n_inst > (1ll << 30) || (long long)H * W > (1ll << 30)) return {0, 0};
    BvShape best{4, 1};
    while (best.lanes < n && best.lanes < 32) best.lanes *= 2;
    if (best.lanes < n) return {32, 2};
    for (int j = 2; j <= 3; ++j) {
        int lanes = grads ? 4 : 2;
        while (lanes * j < n) lanes *= 2;
        if (n < 3 || lanes > 16 || n_inst * lanes < 16ll * 32 * sm_count()) continue;
        const int slots = lanes * j, least = best.lanes * best.vecs;
        if (slots < least || (slots == least && best.vecs == 1 && (!grads || lanes >= 8))) best = {lanes, j};
    }
    return best;
}

template <typename T, bool POINT, bool GRAD>
static void bv_launch(BvArgs a, const BvShape& s, cudaStream_t st) {
    const int pw = 32 / s.lanes;
    const long long tx = (a.W + pw - 1) / pw, ty = (a.H + BV_WARPS - 1) / BV_WARPS, in_tiles = tx * pw * ty * BV_WARPS;
    // (a tile's lanes beyond the map are idle: not where they would be more than a fifth)
    if (!a.batch_of && a.G == (long long)a.H * a.W && in_tiles * 4 <= a.G * 5ll) {
        a.tile_rows = make_fast_div((uint32_t)tx);
        a.tiles = make_fast_div((uint32_t)(tx * ty));
        a.units = (int)(a.B * tx * ty);
    } else
        a.units = (int)(((long long)a.n_inst + BV_WARPS * pw - 1) / (BV_WARPS * pw));
    const int blocks = a.units < 32 * sm_count() ? a.units : 32 * sm_count();
#define VTP_BV(LG, J)                                                                       \
    if (s.lanes == LG && s.vecs == J) {                                                     \
        if constexpr (!GRAD) bilinear_vectors_fwd_kernel<T, POINT, LG, J><<<blocks, BV_WARPS * 32, 0, st>>>(a); \
        else if constexpr (LG >= 4) bilinear_vectors_bwd_kernel<T, POINT, LG, J><<<blocks, BV_WARPS * 32, 0, st>>>(a); \
    }
    VTP_BV(4, 1) VTP_BV(8, 1) VTP_BV(16, 1) VTP_BV(32, 1)
    VTP_BV(2, 2) VTP_BV(4, 2) VTP_BV(8, 2) VTP_BV(16, 2) VTP_BV(32, 2)
    VTP_BV(2, 3) VTP_BV(4, 3) VTP_BV(8, 3) VTP_BV(16, 3)
#undef VTP_BV
}
template <bool GRAD>
static void bv_run(const BvArgs& a, const BvShape& s, int dtype, int mode, cudaStream_t st) {
    if (dtype == VTP_F32) mode == 0 ? bv_launch<float, true, GRAD>(a, s, st) : bv_launch<float, false, GRAD>(a, s, st);
    else mode == 0 ? bv_launch<bf16, true, GRAD>(a, s, st) : bv_launch<bf16, false, GRAD>(a, s, st);
}
static BvArgs bv_args(const void* input, const void* grid, const void* weight, int dtype, int B, int H, int W, int C, int G, int P, long long n) {
    BvArgs a{};
    a.input = (const char*)input; a.grid = (const char*)grid; a.weight = (const char*)weight;
    a.B = B; a.H = H; a.W = W; a.G = G; a.P = P; a.n_inst = (int)n;
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
    const BaLayout lay = ba_layout(dtype, C, grid, {input, mode == 0 ? out : weight});
        const long long n_inst = batch_of ? (long long)G : (long long)B * G;
    if (const BvShape shape = bv_shape(lay, dtype, C, H, W, n_inst, false); shape.lanes) {
        BvArgs a = bv_args(input, grid, weight, dtype, B, H, W, C, G, P, n_inst);
        a.out = (char*)out;
        a.batch_of = batch_of;
        bv_run<false>(a, shape, dtype, mode, st);
        return check_launch("bilinear_attention_forward");
    }
    const int blocks = ba_grid(n_inst);
#define VTP_BA_FWD(T, V)                                                                                 \
    (mode == 0 ? bilinear_attention_fwd_kernel<T, true, V> : bilinear_attention_fwd_kernel<T, false, V>) \
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
    if (const BvShape shape = bv_shape(lay, dtype, C, H, W, (long long)B * G, true); shape.lanes) {
        BvArgs a = bv_args(input, grid, weight, dtype, B, H, W, C, G, P, (long long)B * G);
        a.grad_out = (const char*)grad_out;
        a.grad_input = (char*)grad_input; a.grad_grid = (char*)grad_grid; a.grad_weight = (char*)grad_weight;
        bv_run<true>(a, shape, dtype, mode, st);
        return check_launch("bilinear_attention_backward");
    }
    const int blocks = ba_grid((long long)B * G);
#define VTP_BA_BWD(T, V)                                                                                 \
    (mode == 0 ? bilinear_attention_bwd_kernel<T, true, V> : bilinear_attention_bwd_kernel<T, false, V>) \
        <<<blocks, BA_WARPS * 32, 0, st>>>((const T*)grad_out, (const T*)input, (const T*)grid, (const T*)weight, \
                                           (T*)grad_input, (T*)grad_grid, (T*)grad_weight, B, H, W, C, G, P)
    if (dtype == VTP_F32) VTP_BA_DISPATCH(float, 4, VTP_BA_BWD);
    else VTP_BA_DISPATCH(bf16, 8, VTP_BA_BWD);
#undef VTP_BA_BWD
    return check_launch("bilinear_attention_backward");
}
