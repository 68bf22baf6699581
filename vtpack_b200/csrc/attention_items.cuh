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

// The same for up to 32 * PER images by one warp alone, a run of up to PER images per lane, which also works out item `w`, so that
// its loads are under way before the other warps know the list.  Two steps, so that the caller can look at other memory while the
// offsets are under way.  Batches of up to 32 images have a form and kernels of
// their own (DeiT-Ti, 12 images: 519 us with list_tiles, 516 with eight images per lane, 513 with both forms in one kernel, 509
// apart; DeiT-B, 8 images: 937, 935, 934 and 927).
constexpr int FEW_PER = 8, FEW_IMAGES = 32 * FEW_PER;
template <int PER>
struct FewImages {
    int o[PER + 1];                // offsets of the lane's images b0 .. b0 + n - 1 and of the one behind them
    int b0, n;

    __device__ __forceinline__ void load(const int32_t* __restrict__ offsets, int B) {
        const int lane = threadIdx.x & 31, per = PER == 1 ? 1 : (B + 31) / 32;
        b0 = min(lane * per, B);
        n = min(per, B - b0);
#pragma unroll
        for (int i = 0; i <= PER; ++i) o[i] = (n > 0 && i <= n) ? offsets[b0 + i] : 0;
    }

    // Returns the number of tiles; `it` holds only if w is below that times heads.
    __device__ __forceinline__ int list(int B, int max_q, int l_max, int* status, int* tile_prefix, int32_t* offs, int w, int heads,
                                        AttnItem& it) const {
        const int lane = threadIdx.x & 31;
        int before[PER], sum = 0;              // tiles of the lane's images in front of an image
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            int cnt = i < n ? o[i + 1] - o[i] : 0;
#if VTP_INDEX_GUARDS
            if (i < n && (cnt < 0 || cnt > max_q || o[i] < 0 || o[i + 1] > l_max)) {
                if (status && blockIdx.x == 0) atomicOr(status, STATUS_BAD_INDEX);
                cnt = (o[i] < 0) ? 0 : min(max(cnt, 0), max_q);
            }
#endif
            before[i] = sum;
            sum += (cnt + QT - 1) / QT;
        }
        int incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int nb = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += nb;
        }
        const int excl = incl - sum, total = __shfl_sync(0xffffffffu, incl, 31);
        // the last image whose first tile is not behind tile tg (as attn_item finds it): the last of the lane's and the lane that has it
        const int tg = w / heads;
        int b = 0, row0 = 0, end = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            if (i >= n) continue;
            const int first = excl + before[i];
            tile_prefix[b0 + i] = first;
            offs[b0 + i] = o[i];
            if (first <= tg) { b = b0 + i; row0 = o[i] + (tg - first) * QT; end = o[i + 1]; }
            if (b0 + i + 1 == B) { tile_prefix[B] = total; offs[B] = o[i + 1]; }
        }
        const int from = 31 - __clz(__ballot_sync(0xffffffffu, n > 0 && excl <= tg));
        it.b = __shfl_sync(0xffffffffu, b, from);
        it.h = w - tg * heads;
        it.row0 = __shfl_sync(0xffffffffu, row0, from);
        it.nq = min(QT, __shfl_sync(0xffffffffu, end, from) - it.row0);
        return total;
    }
};

}  // namespace vtp
