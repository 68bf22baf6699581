// Bilinear attention over rows of 16-byte vectors, forward and gradients; what was measured stands in bilinear_attention.cu.
// A group of LG lanes owns an instance, a lane J vectors of its channels: the arithmetic of a point's corners, which every lane of a
// group repeats, is paid once per J of them.
#include "bilinear_attention.cuh"

namespace vtp {

constexpr int BV_WARPS = 4;

// 16 bytes as pairs of channels (bf16: common.cuh)
__device__ __forceinline__ float2 pair_of(const Vec<float>& v, int i) { return i ? make_float2(v.raw.z, v.raw.w) : make_float2(v.raw.x, v.raw.y); }
__device__ __forceinline__ void set_pair(Vec<float>& v, int i, float2 f) {
    if (i) { v.raw.z = f.x; v.raw.w = f.y; }
    else { v.raw.x = f.x; v.raw.y = f.y; }
}
__device__ __forceinline__ void red_vec(char* p, const Vec<float>& v) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.raw.x), "f"(v.raw.y), "f"(v.raw.z), "f"(v.raw.w));
}
__device__ __forceinline__ void red_vec(char* p, const Vec<bf16>& v) {
    asm volatile("red.relaxed.gpu.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.raw.x), "r"(v.raw.y), "r"(v.raw.z),
                 "r"(v.raw.w));
}

// What a corner outside the map is read from: the loads need no condition, and no zeros in front of them.
__device__ const __align__(16) uint4 g_no_pixel[BV_MAXVEC] = {};

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
            own = true;
            b = img;
            inst = (int)img * a.G + ((int)ty * BV_WARPS + warp) * a.W + (int)tx * PW + sub;
        } else {
            const int i = (unit * BV_WARPS + warp) * PW + sub;
            own = i < a.n_inst;                     // a group past the end goes along for the shuffles
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
    constexpr int PW = 32 / LG, NP = Vec<T>::N / 2;
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
            Vec<T> w{};
            if (!POINT && has[j]) w.load(reinterpret_cast<const T*>(a.weight + (size_t)at.inst * a.row + c[j]));
#pragma unroll
            for (int i = 0; i < NP; ++i) sum[j][i] = pair_of(w, i);
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
                Vec<T> q[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) q[i].load(reinterpret_cast<const T*>(t.at[i] + c[j]));
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    const float2 v = fma2(both(k.w_rb), pair_of(q[3], i), fma2(both(k.w_lb), pair_of(q[2], i),
                                          fma2(both(k.w_rt), pair_of(q[1], i), mul2(both(k.w_lt), pair_of(q[0], i)))));
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
                Vec<T> o;
#pragma unroll
                for (int i = 0; i < NP; ++i) set_pair(o, i, sum[j][i]);
                if (has[j]) o.store(reinterpret_cast<T*>(a.out + (size_t)at.inst * a.row + c[j]));
            }
        }
    }
}

// (see bilinear_attention_bwd_kernel)
template <typename T, bool POINT, int LG, int J>
__global__ void __launch_bounds__(BV_WARPS * 32, J == 3 ? 4 : 5)
bilinear_vectors_bwd_kernel(const __grid_constant__ BvArgs a) {
    constexpr int PW = 32 / LG, NP = Vec<T>::N / 2;
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
            Vec<T> u{};
            if (has[j]) u.load(reinterpret_cast<const T*>((POINT ? a.grad_out : a.weight) + (size_t)at.inst * a.row + c[j]));
#pragma unroll
            for (int i = 0; i < NP; ++i) up[j][i] = pair_of(u, i);
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
                Vec<T> q[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) q[i].load(reinterpret_cast<const T*>(t.at[i] + c[j]));
#define BV_RED(IN, OFF, WT)                                                               \
                if (IN) {                                                                 \
                    const float w = sc * (WT);                                            \
                    Vec<T> r;                                                             \
                    _Pragma("unroll") for (int i = 0; i < NP; ++i) set_pair(r, i, mul2(up[j][i], both(w))); \
                    red_vec(g + (OFF) + c[j], r);                                         \
                }
                BV_RED(k.in_lt, 0, k.w_lt)
                BV_RED(k.in_rt, a.row, k.w_rt)
                BV_RED(k.in_lb, down, k.w_lb)
                BV_RED(k.in_rb, down + a.row, k.w_rb)
#undef BV_RED
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    const float2 lt = pair_of(q[0], i), rt = pair_of(q[1], i), lb = pair_of(q[2], i), rb = pair_of(q[3], i), u = up[j][i];
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
                Vec<T> o;
#pragma unroll
                for (int i = 0; i < NP; ++i) set_pair(o, i, gw[POINT ? 0 : j][i]);
                if (has[j]) o.store(reinterpret_cast<T*>(a.grad_weight + (size_t)at.inst * a.row + c[j]));
            }
        }
    }
}

template <typename T, bool POINT, bool GRAD>
static void bv_launch(BvArgs a, const BvShape& s, cudaStream_t st) {
    const int pw = 32 / s.lanes;
    const long long tx = (a.W + pw - 1) / pw, ty = (a.H + BV_WARPS - 1) / BV_WARPS, in_tiles = tx * pw * ty * BV_WARPS;
    // Whole tiles only: idle lanes beyond the map cost more than the tiles save.  260 maps of 5 to 64 pixels a side, mean time over that without tiles'
    // lanes beyond the map allowed: up to a quarter of them 1.03 (forward) and 1.02 (backward), a twentieth 1.005 and 1.004.
    if (!a.batch_of && a.G == (long long)a.H * a.W && in_tiles == a.G) {
        a.tile_rows = make_fast_div((uint32_t)tx);
        a.tiles = make_fast_div((uint32_t)(tx * ty));
        a.units = (int)(a.B * tx * ty);
    } else
        a.units = (int)(((long long)a.n_inst + BV_WARPS * pw - 1) / (BV_WARPS * pw));
    const int blocks = a.units < a.most_blocks ? a.units : a.most_blocks;
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

template <typename T>
void bilinear_vectors(const BvArgs& a, const BvShape& s, bool point, bool grad, cudaStream_t st) {
    if (grad) point ? bv_launch<T, true, true>(a, s, st) : bv_launch<T, false, true>(a, s, st);
    else point ? bv_launch<T, true, false>(a, s, st) : bv_launch<T, false, false>(a, s, st);
}

}  // namespace vtp
