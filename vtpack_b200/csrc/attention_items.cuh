// The work items of the tensor-core attention kernels: 128 packed queries of one (image, head), listed on the device from the
// per-image offsets, so that images with few queries cost nothing and nothing is read back to the host.
#pragma once

#include "common.cuh"

namespace vtp {

constexpr int QT = 128;            // queries per item = TMEM lanes
constexpr int HD = 64;             // head dim

struct AttnItem { int b, h, row0, nq; };

// tile_prefix[b] = number of 128-query tiles of the images in front of b, b <= B, in shared memory; offs: a copy of the offsets, or
// null.  All threads fetch the per-image tile counts at once (one global-load latency), then warp 0 scans them, a run of images
// per lane.  (The offsets come from the caller: a count outside [0, max_q] is clamped, so the item list always fits the grid's
// bound.)  A barrier of the CTA has to follow.
__device__ __forceinline__ void list_tiles(const int32_t* __restrict__ offsets, int B, int max_q, int l_max, int* status,
                                           int* tile_prefix, int32_t* offs) {
    for (int b = threadIdx.x; b < B; b += blockDim.x) {
        const int o0 = offsets[b], o1 = offsets[b + 1];
        int cnt = o1 - o0;
#if VTP_INDEX_GUARDS
        if (cnt < 0 || cnt > max_q || o0 < 0 || o1 > l_max) {
            if (status && blockIdx.x == 0) atomicOr(status, STATUS_BAD_INDEX);
            cnt = (o0 < 0) ? 0 : min(max(cnt, 0), max_q);
        }
#endif
        tile_prefix[b] = (cnt + QT - 1) / QT;
        if (offs) {
            offs[b] = o0;
            if (b + 1 == B) offs[B] = o1;
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        const int per = (B + 31) / 32, b0 = min(lane * per, B), b1 = min(b0 + per, B);
        int sum = 0;
        for (int b = b0; b < b1; ++b) sum += tile_prefix[b];
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int nb = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += nb;
        }
        int run = incl - sum;
        for (int b = b0; b < b1; ++b) {
            const int tiles = tile_prefix[b];
            tile_prefix[b] = run;
            run += tiles;
        }
        if (lane == 31) tile_prefix[B] = incl;
    }
}

// item w -> (image, head, first packed row, valid rows); tile_prefix is in shared memory, so are the offsets of a moderate batch
__device__ __forceinline__ AttnItem attn_item(int w, int heads, int B, const int* tile_prefix, const int32_t* offsets) {
    const int tg = w / heads;
    int lo = 0, hi = B;                        // largest b with tile_prefix[b] <= tg
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (tile_prefix[mid] <= tg) lo = mid; else hi = mid;
    }
    AttnItem it;
    it.b = lo;
    it.h = w - tg * heads;
    const int t = tg - tile_prefix[lo];
    it.row0 = offsets[lo] + t * QT;
    it.nq = min(QT, offsets[lo + 1] - it.row0);
    return it;
}

// The same for up to 32 images by one warp alone, which also works out item `w`, so that its loads are under way before the other
// warps know the list: o0, o1 are offsets[lane] and offsets[lane + 1] (lane < B, else 0).  Returns the number of tiles; `it` holds only if
// w is below that times heads.
constexpr int FEW_IMAGES = 32;
__device__ __forceinline__ int list_few_tiles(int o0, int o1, int B, int max_q, int l_max, int* status, int* tile_prefix, int32_t* offs,
                                              int w, int heads, AttnItem& it) {
    const int lane = threadIdx.x & 31;
    int cnt = o1 - o0;
#if VTP_INDEX_GUARDS
    if (cnt < 0 || cnt > max_q || o0 < 0 || o1 > l_max) {
        if (status && blockIdx.x == 0) atomicOr(status, STATUS_BAD_INDEX);
        cnt = (o0 < 0) ? 0 : min(max(cnt, 0), max_q);
    }
#endif
    const int tiles = lane < B ? (cnt + QT - 1) / QT : 0;
    int incl = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int nb = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += nb;
    }
    const int excl = incl - tiles, total = __shfl_sync(0xffffffffu, incl, 31);
    if (lane < B) {
        tile_prefix[lane] = excl;
        offs[lane] = o0;
        if (lane + 1 == B) { tile_prefix[B] = total; offs[B] = o1; }
    }
    const int tg = w / heads;
    // the last image whose first tile is not behind tile tg (as attn_item finds it)
    const int b = 31 - __clz(__ballot_sync(0xffffffffu, lane < B && excl <= tg));
    const int first = __shfl_sync(0xffffffffu, o0, b), end = __shfl_sync(0xffffffffu, o1, b);
    it.b = b;
    it.h = w - tg * heads;
    it.row0 = first + (tg - __shfl_sync(0xffffffffu, excl, b)) * QT;
    it.nq = min(QT, end - it.row0);
    return total;
}

}  // namespace vtp
