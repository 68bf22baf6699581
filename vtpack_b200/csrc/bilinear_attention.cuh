// What the kernels of the bilinear attention share: a point's four corners, and what the host hands to the vector kernels
// (bilinear_vectors.cuh), which are compiled once for each element type in a file of its own: a program pays for loading the module of
// the type it uses (a process's first forward and backward: both types in one module 4.3 ms, apart 1.5 in fp32 and 2.0 in bf16).
#pragma once
#include "common.cuh"
#include "linear.h"

namespace vtp {

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

constexpr int BV_MAXVEC = 64;                      // 16-byte vectors of the widest row of channels

struct BvArgs {
    const char *input, *grid, *weight, *grad_out;
    char *out, *grad_input, *grad_grid, *grad_weight;
    const long long* batch_of;
    int B, H, W, G, P, n_inst;
    int row, vecs;                                  // bytes and 16-byte vectors of a row of channels
    FastDiv per_image;                              // G
    FastDiv tile_rows, tiles;                       // tiles of a row of tiles (d = 0: no tiles) and of a map
    int units, most_blocks;                         // pieces of work, one block each at a time
};

struct BvShape { int lanes, vecs; };                // lanes of a group, vectors of a lane
template <typename T> void bilinear_vectors(const BvArgs& a, const BvShape& s, bool point, bool grad, cudaStream_t st);

}  // namespace vtp
