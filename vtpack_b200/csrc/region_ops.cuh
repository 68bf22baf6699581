// Region-parallel token movers used by the fused block forward: router gate, multi-grain
// pooling (with LayerNorm statistics or explicit LayerNorm rows) and replicate-unpool with
// residual.  One CTA (one warp, where there are many: pool_warp_kernel, unpool_warp_kernel) owns one 4x4 region of the token grid, whatever grain
// the gate picked for it.  A token row is spread over a GROUP of G lanes, each lane holding CPL chunks of 16
// bytes (C = G * CPL * 16 bytes exactly, e.g. 16 lanes x 3 chunks at C=384 bf16), so no lane
// idles and no access needs a bounds check; a group owns TPG neighbouring tokens of a grid
// row.  All 16 rows of a region are requested before any arithmetic, every region costs the
// same, and nothing depends on walking the patch list.
// Sums that span tokens go through shared memory: each group sums its own tokens in order,
// then the partial sums of a patch are added top-left to bottom-right (the reference adds
// the same tokens in one sequential chain; results differ by fp32 rounding only).
//
// Replaces DynamicRouter.forward (vtpack/layers/dge.py:145-150), grained_sample_compress /
// grained_sample_decompress (vtpack/layers/csrc/grained_sample/grained_sample.cu:31-69,
// 107-144) and the nn.LayerNorm norm1 calls of Block.forward
// (vtpack/models/dge/deit_dge.py:127) on the fused path.
//
// Compiled by element type and kind of mover (region_pool_*.cu, region_unpool_*.cu, region_gated.cu): a program pays for loading the modules
// of the kernels it launches, and they build side by side (a process's first forward, all in one module / apart, ms: DeiT-Ti, one image, 59 / 37,
// an fp32 layer 54 / 28; build 124 -> 50 s on eight cores).
#pragma once
#include "region_ops.h"
#include "runtime.h"

namespace vtp {

constexpr int RG = 4;              // tokens per region side

// bf16: four warps, one per grid row, so a group owns 1, 2 or 4 tokens.  fp32: a token per group, 4, 8 or 16 warps.  What a region
// takes is its longest chain, and an fp32 batch has few regions: DeiT-S, 12 images, pool 16.0 -> 8.0 us, unpool 10.7 -> 6.1 (gate,
// pool and unpool of bf16 in the same form: DeiT-S, 256 images, 19.6 / 17.1 / 38.5 -> 35 / 26 / 45, DeiT-B, 33 images, pool 7.6 ->
// 11.0, unpool 14.8 -> 15.1, 7 images no faster: there regions in flight count, and each warp of theirs moves fewer bytes).
template <typename T, int G, int CPL>
struct Lay {
    static constexpr int VN = Vec<T>::N;
    static constexpr int GROUPS = 32 / G;                                  // groups of a warp
    static constexpr int TPG = sizeof(T) == 4 ? 1 : RG / GROUPS;           // tokens of a group
    static constexpr int THREADS = RG * RG / TPG * G;
    // Sums that span tokens go through rows of C floats in shared memory: the two halves of each grid row, or (TPG == 4) whole
    // grid rows too; groups of a whole warp with one token each leave that.
    static constexpr bool BY_TOKEN = TPG == 1 && G == 32;
    static constexpr int SLOTS = BY_TOKEN ? RG * RG : RG * 2;
};

// group-wide sum over the G lanes that share a row
template <int G>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <typename T, int CPL>
__device__ __forceinline__ void load_row(Vec<T> (&r)[CPL], const T* src, int sub, int G) {
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch) r[ch].load(src + (sub + G * ch) * Vec<T>::N);
}
template <typename T, int CPL>
__device__ __forceinline__ void store_row(const Vec<T> (&r)[CPL], T* dst, int sub, int G) {
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch) r[ch].store(dst + (sub + G * ch) * Vec<T>::N);
}
template <typename T, int CPL>
__device__ __forceinline__ void to_f(float (&f)[CPL][Vec<T>::N], const Vec<T> (&r)[CPL]) {
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch) r[ch].to_float(f[ch]);
}
template <typename T, int CPL>
__device__ __forceinline__ void zero_f(float (&f)[CPL][Vec<T>::N]) {
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
        for (int i = 0; i < Vec<T>::N; ++i) f[ch][i] = 0.f;
}
// shared-memory row of C floats, accessed as float4 (a lane's chunk is VN consecutive floats)
template <typename T, int CPL>
__device__ __forceinline__ void smem_store(float* row, const float (&f)[CPL][Vec<T>::N], int sub, int G) {
    constexpr int VN = Vec<T>::N;
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
        for (int i = 0; i < VN / 4; ++i)
            reinterpret_cast<float4*>(row + (sub + G * ch) * VN)[i] =
                make_float4(f[ch][4 * i], f[ch][4 * i + 1], f[ch][4 * i + 2], f[ch][4 * i + 3]);
}
template <typename T, int CPL>
__device__ __forceinline__ void smem_add(float (&f)[CPL][Vec<T>::N], const float* row, int sub, int G) {
    constexpr int VN = Vec<T>::N;
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
        for (int i = 0; i < VN / 4; ++i) {
            const float4 v = reinterpret_cast<const float4*>(row + (sub + G * ch) * VN)[i];
            f[ch][4 * i] += v.x; f[ch][4 * i + 1] += v.y; f[ch][4 * i + 2] += v.z; f[ch][4 * i + 3] += v.w;
        }
}

// (sum, sum of squares) of a row held across a group
template <typename T, int G, int CPL>
__device__ __forceinline__ float2 row_sums(const float (&f)[CPL][Vec<T>::N]) {
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
        for (int i = 0; i < Vec<T>::N; ++i) { s1 += f[ch][i]; s2 = fmaf(f[ch][i], f[ch][i], s2); }
    return make_float2(group_sum<G>(s1), group_sum<G>(s2));
}
// (mean, rstd) from (sum, sum of squares): exact enough for bf16 rows (8 significant bits)
__device__ __forceinline__ float2 mean_rstd(float2 s, int C, float eps) {
    const float mean = s.x / (float)C;
    return make_float2(mean, rsqrtf(fmaxf(s.y / (float)C - mean * mean, 0.f) + eps));
}

// explicit LayerNorm of a row (two-pass), stored in one place or two
template <typename T, int G, int CPL>
__device__ __forceinline__ void ln_store(const float (&f)[CPL][Vec<T>::N], int sub, int C,
                                         const float* __restrict__ lnw, const float* __restrict__ lnb, float eps,
                                         T* y, size_t row, bool terms, T* y2 = nullptr, size_t row2 = 0, bool terms2 = false) {
    constexpr int VN = Vec<T>::N;
    float s = 0.f;
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
        for (int i = 0; i < VN; ++i) s += f[ch][i];
    const float mean = group_sum<G>(s) / (float)C;
    float v = 0.f;
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
        for (int i = 0; i < VN; ++i) { const float d = f[ch][i] - mean; v = fmaf(d, d, v); }
    const float rstd = rsqrtf(group_sum<G>(v) / (float)C + eps);
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch) {
        const int c0 = (sub + G * ch) * VN;
        float o[VN];
#pragma unroll
        for (int i = 0; i < VN; ++i) o[i] = (f[ch][i] - mean) * rstd * __ldg(lnw + c0 + i) + __ldg(lnb + c0 + i);
        store_row_vec<T>(y, row, C, c0, o, terms);
        if (y2) store_row_vec<T>(y2, row2, C, c0, o, terms2);
    }
}

// round a row to T (what the consumer GEMM will read), store it, keep the rounded values
template <typename T, int CPL>
__device__ __forceinline__ void round_store(float (&f)[CPL][Vec<T>::N], T* dst, int sub, int G) {
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch) {
        Vec<T> ov;
        ov.from_float(f[ch]);
        ov.store(dst + (sub + G * ch) * Vec<T>::N);
        ov.to_float(f[ch]);
    }
}

// packed row of a region's first query, from the per-image counts and the grain indices of
// the image's earlier regions (executed redundantly by every warp)
__device__ __forceinline__ int derive_first(const int32_t* __restrict__ counts, const int32_t* __restrict__ idx, int b,
                                            int rr, int R, const Splits& sp, int num_extra, int lane, int* img_base) {
    int part_sum = 0, own = 0;
    for (int j = lane; j < b; j += 32) part_sum += counts[j];
    for (int r = lane; r < rr; r += 32) {
        const int kk = min(max(idx[b * R + r], 0), sp.n - 1);
        own += sp.v[kk] * sp.v[kk];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        part_sum += __shfl_xor_sync(0xffffffffu, part_sum, o);
        own += __shfl_xor_sync(0xffffffffu, own, o);
    }
    *img_base = part_sum;
    return part_sum + num_extra + own;
}

// Each group `gi` leaves the in-order sum `acc` of its tokens in shared memory.  Slot layout: part[(w * 2 + half) * C], half 0 = left
// two tokens of grid row w, 1 = right two.  A group that owns a whole row (TPG == 4) fills slot (w, 0) only, unless it was told to
// split.  Groups that own a single token are paired through shared memory, or (BY_TOKEN) leave it in a slot of its own.
// Ends with the CTA barrier.
template <typename T, int G, int CPL>
__device__ __forceinline__ void publish_partials(float* part, float (&acc)[CPL][Vec<T>::N], int gi, int sub, int C) {
    using L = Lay<T, G, CPL>;
    if (L::TPG == 4) {
        smem_store<T, CPL>(part + (size_t)(gi * 2) * C, acc, sub, G);
    } else if (L::TPG == 2 || L::BY_TOKEN) {
        smem_store<T, CPL>(part + (size_t)gi * C, acc, sub, G);
    } else {
        float* slot = part + (size_t)(gi >> 1) * C;
        if ((gi & 1) == 0) smem_store<T, CPL>(slot, acc, sub, G);
        __syncwarp();
        if ((gi & 1) == 1) {
            float tmp[CPL][Vec<T>::N];
            zero_f<T, CPL>(tmp);
            smem_add<T, CPL>(tmp, slot, sub, G);          // even token first, then the odd one
#pragma unroll
            for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
                for (int i = 0; i < Vec<T>::N; ++i) tmp[ch][i] += acc[ch][i];
            smem_store<T, CPL>(slot, tmp, sub, G);
        }
    }
    __syncthreads();
}
// acc += the left or right half (tokens) of grid row w, or (HALVES == 2) the whole row.  The order in which a region's tokens are
// added does not depend on TPG where G does not.
template <typename T, int G, int CPL, int HALVES>
__device__ __forceinline__ void add_row(float (&acc)[CPL][Vec<T>::N], const float* part, int w, int half, int sub, int C) {
    using L = Lay<T, G, CPL>;
    if (L::BY_TOKEN) {
        float sum[CPL][Vec<T>::N];
        zero_f<T, CPL>(sum);
#pragma unroll
        for (int j = 0; j < 2 * HALVES; ++j) smem_add<T, CPL>(sum, part + (size_t)(w * RG + 2 * half + j) * C, sub, G);
#pragma unroll
        for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
            for (int i = 0; i < Vec<T>::N; ++i) acc[ch][i] += sum[ch][i];
    } else {
        smem_add<T, CPL>(acc, part + (size_t)(w * 2 + half) * C, sub, G);
        if (HALVES == 2 && L::TPG != 4) smem_add<T, CPL>(acc, part + (size_t)(w * 2 + 1) * C, sub, G);
    }
}

// ------------------------------------------------------------------------------- pool
// POOL_STATS: comp rows + (mean, rstd) of every comp row (and of every token row unless
//             they are already known), for the GEMMs that apply LayerNorm in their
//             epilogue; zeroes the stats_acc rows.
// POOL_LN:    comp rows + explicit LN(x) rows and LN(comp) rows.
// POOL_PLAIN: comp rows only, as means or (sum_only) as sums: the latter is the gradient of the
//             replicate-unpool with respect to its packed rows (vtpack/layers/grained_sample.py:61-72).
// Seven CTAs per SM (at most 73 registers, a few spilled words): the kernel is bound by how many
// regions are in flight, and measured faster over the whole forward than at the 88 registers / five
// CTAs the compiler picks on its own (six: +0.5 %, seven: +0.9 %, eight: +0.8 %).
// POOL_COLS:  POOL_STATS, and LayerNorm(x) as the rows of the strided convolution in front of the keys (a block with a spatial
//             reduction): token (y, x) is element (y % sr, x % sr) of window (y / sr, x / sr).  The tokens are in registers
//             here; a gather of its own read them again (PVT-small, 96 images: 2678 -> 2640 us, PVT-tiny, 3 images, 450 -> 444).
constexpr int POOL_LN = 0, POOL_STATS = 1, POOL_PLAIN = 2, POOL_COLS = 3;
// (A thread of a narrow-row layout holds one or two 16-byte vectors of a region: such kernels run with 16 or 12 CTAs per SM
// (a few spilled words in the unpool; measured faster all the same), and the kernel is bound by how many regions are in flight.)
template <typename T, int G, int CPL>
constexpr int pool_ctas() {
    if (Lay<T, G, CPL>::THREADS != 128) return G == 16 ? (CPL <= 2 ? 6 : 4) : CPL <= 2 ? 3 : CPL <= 3 ? 2 : 1;
    return Lay<T, G, CPL>::TPG * CPL <= 1 ? 16 : Lay<T, G, CPL>::TPG * CPL <= 2 ? 12 : 7;
}
// LayerNorm(x) of token (ty, tx) as a part of its window's row (POOL_COLS)
template <typename T, int G, int CPL>
__device__ __forceinline__ void cols_row(const float (&f)[CPL][Vec<T>::N], float2 st, int b, int ty, int tx, const RegionGeom& g, int sr, int sub,
                                         const float* __restrict__ lnw, const float* __restrict__ lnb, T* __restrict__ xn) {
    constexpr int VN = Vec<T>::N;
    const int wy = ty / sr, wx = tx / sr;
    const size_t win = ((size_t)b * (g.Hr * RG / sr) + wy) * (g.W / sr) + wx;
    T* dst = xn + ((win * sr + (ty - wy * sr)) * sr + (tx - wx * sr)) * g.C;
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch) {
        const int c0 = (sub + G * ch) * VN;
        float o[VN];
#pragma unroll
        for (int i4 = 0; i4 < VN / 4; ++i4) {
            const float4 w4 = __ldg(reinterpret_cast<const float4*>(lnw + c0) + i4);
            const float4 b4 = __ldg(reinterpret_cast<const float4*>(lnb + c0) + i4);
            const float gw[4] = {w4.x, w4.y, w4.z, w4.w}, gb[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) o[4 * i4 + i] = (f[ch][4 * i4 + i] - st.x) * st.y * gw[i] + gb[i];
        }
        Vec<T> ov;
        ov.from_float(o);
        ov.store(dst + c0);
    }
}
// the e-th extra (cls) token, copied, by a group
template <typename T, int G, int CPL, int MODE>
__device__ __forceinline__ void pool_extra(int e, int sub, const T* __restrict__ x, const RegionGeom& g, const int32_t* __restrict__ region_first,
                                           const int32_t* __restrict__ offsets, const int32_t* __restrict__ counts,
                                           int32_t* __restrict__ counts_next, T* __restrict__ comp, float2* __restrict__ stats_x,
                                           float2* __restrict__ stats_q, float2* __restrict__ stats_acc, int write_stats_x,
                                           const float* __restrict__ lnw, const float* __restrict__ lnb, float eps, T* __restrict__ xn,
                                           T* __restrict__ qn, int* status, int terms) {
    constexpr bool STATS = MODE == POOL_STATS || MODE == POOL_COLS, EXPLICIT_LN = MODE == POOL_LN;
    constexpr int VN = Vec<T>::N;
    if (e >= g.B * g.num_extra) return;
    const int b = e / g.num_extra, t = e % g.num_extra;
    const size_t src_row = (size_t)b * g.N + t;
    int dst_row;
    if (region_first) {
        dst_row = offsets[b] + t;
        if (VTP_INDEX_GUARDS && g.l_max > 0 && (dst_row < 0 || dst_row >= g.l_max)) {   // caller's offsets
            if (sub == 0 && status) atomicOr(status, STATUS_BAD_INDEX);
            return;
        }
    } else {
        int base = 0;
        for (int j = sub; j < b; j += G) base += counts[j];
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) base += __shfl_xor_sync(0xffffffffu, base, o);
        dst_row = base + t;
    }
    // start the next block's per-image count at the extra tokens; its gate adds the rest
    if (t == 0 && sub == 0 && counts_next) counts_next[b] = g.num_extra;
    Vec<T> row[CPL];
    load_row<T, CPL>(row, x + src_row * g.C, sub, G);
    store_row<T, CPL>(row, comp + (size_t)dst_row * g.C, sub, G);
    float f[CPL][VN];
    to_f<T, CPL>(f, row);
    if (STATS) {
        float2 st;
        if (write_stats_x) {
            st = mean_rstd(row_sums<T, G, CPL>(f), g.C, eps);
            if (sub == 0) stats_x[src_row] = st;
        } else {
            st = stats_x[src_row];
        }
        if (sub == 0) { stats_q[dst_row] = st; if (stats_acc) stats_acc[dst_row] = make_float2(0.f, 0.f); }
    } else if (EXPLICIT_LN) {
        ln_store<T, G, CPL>(f, sub, g.C, lnw, lnb, eps, xn, src_row, terms & 1);
        ln_store<T, G, CPL>(f, sub, g.C, lnw, lnb, eps, qn, (size_t)dst_row, terms & 2);
    }
}
// (terms: POOL_LN of fp32 rows only; 1: xn, 2: qn as terms)
template <typename T, int G, int CPL, int MODE>
__device__ __forceinline__ void
pool_region(const int rid, const T* __restrict__ x, RegionGeom g, const int32_t* __restrict__ idx,
                   const int32_t* __restrict__ region_first, const int32_t* __restrict__ offsets,
                   const int32_t* __restrict__ counts, int32_t* __restrict__ offsets_out,
                   int32_t* __restrict__ region_first_out, int32_t* __restrict__ counts_next, Splits sp,
                   T* __restrict__ comp, float2* __restrict__ stats_x, float2* __restrict__ stats_q,
                   float2* __restrict__ stats_acc, int write_stats_x, const float* __restrict__ lnw,
                   const float* __restrict__ lnb, float eps, T* __restrict__ xn, T* __restrict__ qn, int sum_only,
                   int sr, int* status, int terms) {
    constexpr bool COLS = MODE == POOL_COLS, STATS = MODE == POOL_STATS || COLS, EXPLICIT_LN = MODE == POOL_LN;
    using L = Lay<T, G, CPL>;
    constexpr int VN = L::VN, GROUPS = L::GROUPS, TPG = L::TPG;
    extern __shared__ float part[];          // [SLOTS][C] partial sums
    __shared__ int first_s;
    const int lane = threadIdx.x & 31, sub = lane % G;
    const int gi = (int)(threadIdx.x >> 5) * GROUPS + lane / G;      // the group, its tokens: row w, columns col0 .. col0 + TPG - 1
    const int w = gi * TPG / RG, col0 = gi * TPG % RG;
    const int R = g.Hr * g.Wr;

    if (rid >= g.B * R) {
        pool_extra<T, G, CPL, MODE>((rid - g.B * R) * (RG * RG / TPG) + gi, sub, x, g, region_first, offsets, counts, counts_next, comp, stats_x, stats_q,
                                    stats_acc, write_stats_x, lnw, lnb, eps, xn, qn, status, terms);
        return;
    }

    const int b = rid / R, rr = rid % R;
    const int ry = rr / g.Wr, rx = rr % g.Wr;
    const int k = min(max(idx[rid], 0), sp.n - 1);
    const int s = sp.v[k];                     // sub-patches per region side: 4, 2 or 1
    const int step = RG / s;
    const size_t tok0 = (size_t)b * g.N + g.num_extra + (size_t)(ry * RG + w) * g.W + rx * RG + col0;

    Vec<T> rows[TPG][CPL];
#pragma unroll
    for (int j = 0; j < TPG; ++j) load_row<T, CPL>(rows[j], x + (tok0 + j) * g.C, sub, G);

    int first;
    if (region_first) {
        first = region_first[rid];
        // a caller-supplied first row whose patches would not fit the packed array: skip the region
        if (VTP_INDEX_GUARDS && g.l_max > 0 && (first < 0 || first + s * s > g.l_max)) {
            if (threadIdx.x == 0 && status) atomicOr(status, STATUS_BAD_INDEX);
            return;
        }
    } else {
        // One warp adds up the counts in front while the rows are on their way: with every warp doing it PVT-small's stage 1, 96
        // images, takes 65.8 us instead of 57.5 (DeiT-B, 33 images: 1443 / 1433 us); of two tokens a group, where the barrier
        // costs more (DeiT-S, 256 images: 16.5 / 17.0 us), each warp does.
        constexpr bool EACH = TPG == 2;
        if (EACH || threadIdx.x < 32) {
            int img_base;
            const int at = derive_first(counts, idx, b, rr, R, sp, g.num_extra, lane, &img_base);
            first = at;
            if (threadIdx.x == 0) {
                first_s = at;
                region_first_out[rid] = at;
                if (rr == 0) {
                    offsets_out[b] = img_base;
                    if (b == g.B - 1) offsets_out[g.B] = img_base + counts[b];
                }
            }
        }
        if (!EACH) {
            __syncthreads();
            first = first_s;
        }
    }
    // a grid without extra tokens has no extra-token CTA to start the next block's count
    if (rr == 0 && threadIdx.x == 0 && counts_next && g.num_extra == 0) counts_next[b] = 0;

    // per token: statistics / explicit LayerNorm, and at the finest grain the token is its own patch
    float acc[CPL][VN];                          // in-order sum of this group's tokens (of the current half)
    zero_f<T, CPL>(acc);
#pragma unroll
    for (int j = 0; j < TPG; ++j) {
        float f[CPL][VN];
        to_f<T, CPL>(f, rows[j]);
        const int col = col0 + j;                             // column inside the grid row
        const int prow = first + w * RG + col;                // packed row if step == 1
        if (STATS) {
            float2 st = make_float2(0.f, 1.f);
            if (write_stats_x) {
                st = mean_rstd(row_sums<T, G, CPL>(f), g.C, eps);
                if (sub == 0) stats_x[tok0 + j] = st;
            } else if (COLS || step == 1) {
                st = stats_x[tok0 + j];
            }
            if (step == 1 && sub == 0) { stats_q[prow] = st; if (stats_acc) stats_acc[prow] = make_float2(0.f, 0.f); }
            if (COLS) {
                cols_row<T, G, CPL>(f, st, b, ry * RG + w, rx * RG + col, g, sr, sub, lnw, lnb, xn);
            }
        } else if (EXPLICIT_LN) {
            ln_store<T, G, CPL>(f, sub, g.C, lnw, lnb, eps, xn, tok0 + j, terms & 1, step == 1 ? qn : nullptr, (size_t)prow, terms & 2);
        }
        if (step == 1) {
            store_row<T, CPL>(rows[j], comp + (size_t)prow * g.C, sub, G);
        } else {
#pragma unroll
            for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
                for (int i = 0; i < VN; ++i) acc[ch][i] += f[ch][i];
            // a group that owns the whole grid row closes the left half after two tokens (2x2 patches)
            if (TPG == 4 && step == 2 && j == 1) {
                smem_store<T, CPL>(part + (size_t)(w * 2) * g.C, acc, sub, G);
                zero_f<T, CPL>(acc);
            }
        }
    }
    if (step == 1) return;

    if (TPG == 4 && step == 2) {
        smem_store<T, CPL>(part + (size_t)(w * 2 + 1) * g.C, acc, sub, G);
        __syncthreads();
    } else {
        publish_partials<T, G, CPL>(part, acc, gi, sub, g.C);
    }

    // finishing: group gi takes patch gi.  step 2: four patches (dy, dx); step 4: one.
    if (gi >= s * s) return;
    const int dy = (step == 2) ? (gi >> 1) : 0;
    const int dx = (step == 2) ? (gi & 1) : 0;
    zero_f<T, CPL>(acc);
    if (step == 2) {
        add_row<T, G, CPL, 1>(acc, part, 2 * dy, dx, sub, g.C);
        add_row<T, G, CPL, 1>(acc, part, 2 * dy + 1, dx, sub, g.C);
    } else {
#pragma unroll 1
        for (int r2 = 0; r2 < RG; ++r2) add_row<T, G, CPL, 2>(acc, part, r2, 0, sub, g.C);
    }
    // step * step is 4 or 16: multiplying by its reciprocal is the division, bit for bit
    const float inv_denom = sum_only ? 1.0f : 1.0f / (float)(step * step);
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
        for (int i = 0; i < VN; ++i) acc[ch][i] = acc[ch][i] * inv_denom;
    const int row = first + dy * s + dx;
    if (STATS) {
        round_store<T, CPL>(acc, comp + (size_t)row * g.C, sub, G);
        const float2 st = mean_rstd(row_sums<T, G, CPL>(acc), g.C, eps);
        if (sub == 0) { stats_q[row] = st; if (stats_acc) stats_acc[row] = make_float2(0.f, 0.f); }
    } else {
        if (EXPLICIT_LN) ln_store<T, G, CPL>(acc, sub, g.C, lnw, lnb, eps, qn, (size_t)row, terms & 2);
        round_store<T, CPL>(acc, comp + (size_t)row * g.C, sub, G);
    }
}

template <typename T, int G, int CPL, int MODE>
__global__ void __launch_bounds__((Lay<T, G, CPL>::THREADS), (pool_ctas<T, G, CPL>()))
pool_region_kernel(const T* __restrict__ x, RegionGeom g, const int32_t* __restrict__ idx,
                   const int32_t* __restrict__ region_first, const int32_t* __restrict__ offsets,
                   const int32_t* __restrict__ counts, int32_t* __restrict__ offsets_out,
                   int32_t* __restrict__ region_first_out, int32_t* __restrict__ counts_next, Splits sp,
                   T* __restrict__ comp, float2* __restrict__ stats_x, float2* __restrict__ stats_q,
                   float2* __restrict__ stats_acc, int write_stats_x, const float* __restrict__ lnw,
                   const float* __restrict__ lnb, float eps, T* __restrict__ xn, T* __restrict__ qn, int sum_only,
                   int sr, int* status) {
    pdl_begin();
    pool_region<T, G, CPL, MODE>((int)blockIdx.x, x, g, idx, region_first, offsets, counts, offsets_out, region_first_out, counts_next, sp, comp,
                                 stats_x, stats_q, stats_acc, write_stats_x, lnw, lnb, eps, xn, qn, sum_only, sr, status, 0);
}
// The same with a warp per region, for many bf16 regions (POOL_STATS and POOL_COLS), bit for bit: see unpool_warp_kernel, whose reasons are the same
// (a block per region, C = 384, 256 images: 30 % of DRAM's rate, half of the issue slots).  us of a launch, block -> warp: POOL_STATS C = 384, 4096 regions
// 17.1 -> 13.6, 1536 regions 8.9 -> 7.1, C = 192, 4096 regions 14.7 -> 10.9; POOL_COLS (PVT-small, 96 images) C = 64, 24576 regions 58.2 -> 45.5,
// C = 128, 6144 21.8 -> 19.0, C = 320, 1536 16.2 -> 13.3.
constexpr int PW_WARPS = 4;
template <int G, int CPL, int MODE>
constexpr int pool_warp_ctas() { return G * CPL >= 40 ? (MODE == POOL_COLS ? 3 : 4) : G * CPL > 16 ? 4 : G * CPL == 16 ? 6 : 8; }

template <int G, int CPL, bool COLS, int STEP>
__device__ __forceinline__ void pool_rows(const bf16* __restrict__ x, const RegionGeom& g, int b, int ry, int rx, int first, bf16* __restrict__ comp,
                                          float2* __restrict__ stats_x, float2* __restrict__ stats_q, float2* __restrict__ stats_acc,
                                          bool write_stats_x, const float* __restrict__ lnw, const float* __restrict__ lnb, float eps,
                                          bf16* __restrict__ xn, int sr, int sub, int grp) {
    constexpr int VN = 8, GROUPS = 32 / G, TPG = RG / GROUPS, S = RG / STEP;
    const size_t tok0 = (size_t)b * g.N + g.num_extra + (size_t)ry * RG * g.W + rx * RG + grp * TPG;
    auto leave_stats = [&](int row, float2 st) {         // of a packed row
        if (sub == 0) { stats_q[row] = st; if (stats_acc) stats_acc[row] = make_float2(0.f, 0.f); }
    };
    Vec<bf16> cur[TPG][CPL], next[TPG][CPL];
#pragma unroll
    for (int j = 0; j < TPG; ++j) load_row<bf16, CPL>(cur[j], x + (tok0 + j) * g.C, sub, G);
    float acc[CPL][VN];                                  // of a patch
    zero_f<bf16, CPL>(acc);
#pragma unroll 1
    for (int w = 0; w < RG; ++w) {
        const size_t tok = tok0 + (size_t)w * g.W;
        if (w + 1 < RG)
#pragma unroll
            for (int j = 0; j < TPG; ++j) load_row<bf16, CPL>(next[j], x + (tok + g.W + j) * g.C, sub, G);
        float half[CPL][VN];                             // sum of this group's tokens of the row
#pragma unroll
        for (int j = 0; j < TPG; ++j) {
            const int col = grp * TPG + j;
            float f[CPL][VN];
            to_f<bf16, CPL>(f, cur[j]);
            float2 st = make_float2(0.f, 1.f);
            if (write_stats_x) {
                st = mean_rstd(row_sums<bf16, G, CPL>(f), g.C, eps);
                if (sub == 0) stats_x[tok + j] = st;
            } else if (COLS || STEP == 1) {
                st = stats_x[tok + j];
            }
            if (COLS) cols_row<bf16, G, CPL>(f, st, b, ry * RG + w, rx * RG + col, g, sr, sub, lnw, lnb, xn);
            if (STEP == 1) {
                const int row = first + w * RG + col;
                leave_stats(row, st);
                store_row<bf16, CPL>(cur[j], comp + (size_t)row * g.C, sub, G);
            }
#pragma unroll
            for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
                for (int i = 0; i < VN; ++i) half[ch][i] = j == 0 ? f[ch][i] : half[ch][i] + f[ch][i];
        }
        if (STEP > 1) {
#pragma unroll
            for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
                for (int i = 0; i < VN; ++i) {
                    float v = half[ch][i];
                    if (GROUPS == 4) v += __shfl_xor_sync(0xffffffffu, v, G);      // two neighbours
                    acc[ch][i] += v;
                    if (STEP == 4) acc[ch][i] += __shfl_xor_sync(0xffffffffu, v, 16);     // (right for the left half only, which stores)
                }
            if (w % STEP == STEP - 1) {
                const bool mine = STEP == 4 ? grp == 0 : grp % (GROUPS / 2) == 0;
                const int row = first + (w / STEP) * S + (STEP == 2 ? grp / (GROUPS / 2) : 0);
#pragma unroll
                for (int ch = 0; ch < CPL; ++ch) {
#pragma unroll
                    for (int i = 0; i < VN; ++i) acc[ch][i] *= 1.0f / (float)(STEP * STEP);
                    Vec<bf16> o;
                    o.from_float(acc[ch]);
                    if (mine) o.store(comp + (size_t)row * g.C + (sub + G * ch) * VN);
                    o.to_float(acc[ch]);
                }
                const float2 st = mean_rstd(row_sums<bf16, G, CPL>(acc), g.C, eps);
                if (mine) leave_stats(row, st);
                zero_f<bf16, CPL>(acc);
            }
        }
#pragma unroll
        for (int j = 0; j < TPG; ++j)
#pragma unroll
            for (int ch = 0; ch < CPL; ++ch) cur[j][ch] = next[j][ch];
    }
}

template <int G, int CPL, int MODE>
__global__ void __launch_bounds__(PW_WARPS * 32, (pool_warp_ctas<G, CPL, MODE>()))
pool_warp_kernel(const bf16* __restrict__ x, RegionGeom g, const int32_t* __restrict__ idx, const int32_t* __restrict__ region_first,
                 const int32_t* __restrict__ offsets, const int32_t* __restrict__ counts, int32_t* __restrict__ offsets_out,
                 int32_t* __restrict__ region_first_out, int32_t* __restrict__ counts_next, Splits sp, bf16* __restrict__ comp,
                 float2* __restrict__ stats_x, float2* __restrict__ stats_q, float2* __restrict__ stats_acc, int write_stats_x,
                 const float* __restrict__ lnw, const float* __restrict__ lnb, float eps, bf16* __restrict__ xn, int sr) {
    pdl_begin();
    constexpr int GROUPS = 32 / G;
    const int lane = threadIdx.x & 31, sub = lane % G, grp = lane / G, warp = threadIdx.x >> 5;
    const int R = g.Hr * g.Wr, regions = g.B * R, blocks = (regions + PW_WARPS - 1) / PW_WARPS;
    if ((int)blockIdx.x >= blocks) {
        const int e = (((int)blockIdx.x - blocks) * PW_WARPS + warp) * GROUPS + grp;
        if (e - grp < g.B * g.num_extra)                 // (a group past the end does the last one again: sums are the whole warp's)
            pool_extra<bf16, G, CPL, MODE>(min(e, g.B * g.num_extra - 1), sub, x, g, region_first, offsets, counts, counts_next, comp, stats_x,
                                           stats_q, stats_acc, write_stats_x, lnw, lnb, eps, xn, nullptr, nullptr, 0);
        return;
    }
    const int rid = (int)blockIdx.x * PW_WARPS + warp;
    if (rid >= regions) return;
    const int b = rid / R, rr = rid % R;
    const int ry = rr / g.Wr, rx = rr % g.Wr;
    const int step = RG / sp.v[min(max(idx[rid], 0), sp.n - 1)];
    int first;
    if (region_first) {
        first = region_first[rid];
    } else {
        int img_base;
        first = derive_first(counts, idx, b, rr, R, sp, g.num_extra, lane, &img_base);
        if (lane == 0) {
            region_first_out[rid] = first;
            if (rr == 0) {
                offsets_out[b] = img_base;
                if (b == g.B - 1) offsets_out[g.B] = img_base + counts[b];
            }
        }
    }
    // a grid without extra tokens has none to start the next block's count
    if (rr == 0 && lane == 0 && counts_next && g.num_extra == 0) counts_next[b] = 0;
#define VTP_POOL_ROWS(STEP) \
    pool_rows<G, CPL, MODE == POOL_COLS, STEP>(x, g, b, ry, rx, first, comp, stats_x, stats_q, stats_acc, write_stats_x != 0, lnw, lnb, eps, xn, sr, sub, grp)
    if (step == 1) VTP_POOL_ROWS(1);
    else if (step == 2) VTP_POOL_ROWS(2);
    else VTP_POOL_ROWS(4);
#undef VTP_POOL_ROWS
}
// The pool of an fp32 block whose Linears take terms.  The CTAs in front of the pool's split the block's matrices, and do not wait
// for the kernel in front: that is always one of the same call (the gate, or the unpool of the block before), which let this one start
// only once everything before itself had completed, whatever wrote the parameters and the Linears that read the last
// block's terms among it.  So the split runs beside the end of that kernel (behind the pool's CTAs, in a kernel that
// started late: DeiT-S, 12 images, 17.3 us a block instead of 16.0).  It starts early whatever its grid: early / late, us a block, DeiT-S, 12
// images 98.2 / 99.4, 128 images 503.8 / 504.3, DeiT-B, 40 images 650.1 / 650.6, DeiT-Ti, 200 images 341.2 / 340.5.
// The split is most of what few images move, and still less than splitting in every Linear took (terms / fp32 rows): DeiT-B, 1
// image, pool 24.6 / 21.9 us by itself and the block 104 / 131, 2 images 30.8 / 22.5 and 148 / 199.
template <int G, int CPL>
__global__ void __launch_bounds__((Lay<float, G, CPL>::THREADS), (pool_ctas<float, G, CPL>()))
pool_region_terms_kernel(const float* __restrict__ x, RegionGeom g, const int32_t* __restrict__ idx,
                         const int32_t* __restrict__ region_first, const int32_t* __restrict__ offsets,
                         const int32_t* __restrict__ counts, int32_t* __restrict__ offsets_out,
                         int32_t* __restrict__ region_first_out, int32_t* __restrict__ counts_next, Splits sp,
                         float* __restrict__ comp, const float* __restrict__ lnw, const float* __restrict__ lnb, float eps,
                         float* __restrict__ xn, float* __restrict__ qn, int terms, int split_grid, TermSplit split) {
    if ((int)blockIdx.x < split_grid) {
        split_matrices<Lay<float, G, CPL>::THREADS>(split, (int)blockIdx.x);
        return;
    }
    pdl_begin();
    pool_region<float, G, CPL, POOL_LN>((int)blockIdx.x - split_grid, x, g, idx, region_first, offsets, counts, offsets_out, region_first_out, counts_next, sp,
                                        comp, nullptr, nullptr, nullptr, 0, lnw, lnb, eps, xn, qn, 0, 1, nullptr, terms);
}

// ------------------------------------------------------------------------ router gate
// Region mean of the raw tokens (/ 16), n_splits fp32 dot products, argmax with the lowest
// index winning ties.  acc: the sum of the region's tokens across group 0 of G lanes, of which the lane with `writes` stores.
template <typename T, int G, int CPL>
__device__ __forceinline__ void gate_of_sum(float (&acc)[CPL][Vec<T>::N], int C, int sub, bool writes, const float* __restrict__ gw,
                                            const float* __restrict__ gb, int S, float* __restrict__ logits_out,
                                            int32_t* __restrict__ idx_out, int rid, int32_t* counts_img,
                                            const Splits& sp, const float* __restrict__ img_bias) {
    constexpr int VN = Vec<T>::N;
    // the region mean: 1/16 is a power of two, so the product equals the quotient
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
        for (int i = 0; i < VN; ++i) acc[ch][i] *= 1.0f / (float)(RG * RG);
    float best = 0.f;
    int best_i = 0;
    for (int sI = 0; sI < S; ++sI) {
        float pdot = 0.f;
#pragma unroll
        for (int ch = 0; ch < CPL; ++ch) {
            const float4* wp = reinterpret_cast<const float4*>(gw + (size_t)sI * C + (sub + G * ch) * VN);
#pragma unroll
            for (int i4 = 0; i4 < VN / 4; ++i4) {
                const float4 w4 = __ldg(wp + i4);
                pdot = fmaf(acc[ch][4 * i4 + 0], w4.x, pdot);
                pdot = fmaf(acc[ch][4 * i4 + 1], w4.y, pdot);
                pdot = fmaf(acc[ch][4 * i4 + 2], w4.z, pdot);
                pdot = fmaf(acc[ch][4 * i4 + 3], w4.w, pdot);
            }
        }
        pdot = group_sum<G>(pdot) + __ldg(gb + sI);
        if (img_bias) pdot += __ldg(img_bias + sI);          // per-image offset of the logits (forced grain mixes)
        if (writes && logits_out) logits_out[(size_t)rid * S + sI] = pdot;
        if (sI == 0 || pdot > best) { best = pdot; best_i = sI; }
    }
    if (writes) {
        idx_out[rid] = best_i;
        // queries this region contributes to its image (the image's slot starts at num_extra)
        if (counts_img) atomicAdd(counts_img, sp.v[min(best_i, sp.n - 1)] * sp.v[min(best_i, sp.n - 1)]);
    }
}
// `part` holds the partial row sums published by publish_partials; executed by one group of G lanes.
template <typename T, int G, int CPL>
__device__ __forceinline__ void gate_from_partials(const float* part, int C, int sub, const float* __restrict__ gw,
                                                   const float* __restrict__ gb, int S, float* __restrict__ logits_out,
                                                   int32_t* __restrict__ idx_out, int rid, int32_t* counts_img,
                                                   const Splits& sp, const float* __restrict__ img_bias) {
    float acc[CPL][Vec<T>::N];
    zero_f<T, CPL>(acc);
#pragma unroll 1
    for (int r2 = 0; r2 < RG; ++r2) add_row<T, G, CPL, 2>(acc, part, r2, 0, sub, C);
    gate_of_sum<T, G, CPL>(acc, C, sub, sub == 0, gw, gb, S, logits_out, idx_out, rid, counts_img, sp, img_bias);
}

// ----------------------------------------------------------------------------- unpool
// out[b,tok] = ref[b,tok] + (q[p] - comp[p]) for the patch p that covers the token; optionally
// also the next block's token statistics, router gate decisions and per-image counts.
// an extra (cls) token: its own patch, row p of the packed ones
template <typename T, int G, int CPL>
__device__ __forceinline__ void unpool_extra(const T* __restrict__ q, const T* __restrict__ comp, const T* ref, T* out, const RegionGeom& g,
                                             int b, int t, size_t p, int sub, const NextBlock& nx) {
    constexpr int VN = Vec<T>::N;
    const size_t tok = (size_t)b * g.N + t;
    Vec<T> qv[CPL], cv[CPL], rv[CPL];
    load_row<T, CPL>(qv, q + p * g.C, sub, G);
    load_row<T, CPL>(cv, comp + p * g.C, sub, G);
    load_row<T, CPL>(rv, ref + tok * g.C, sub, G);
    float qf[CPL][VN], cf[CPL][VN], rf[CPL][VN];
    to_f<T, CPL>(qf, qv); to_f<T, CPL>(cf, cv); to_f<T, CPL>(rf, rv);
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
        for (int i = 0; i < VN; ++i) rf[ch][i] = (qf[ch][i] - cf[ch][i]) + rf[ch][i];
    round_store<T, CPL>(rf, out + tok * g.C, sub, G);
    if (nx.stats_x) {
        const float2 st = mean_rstd(row_sums<T, G, CPL>(rf), g.C, nx.eps);
        if (sub == 0) nx.stats_x[tok] = st;
    }
}
template <typename T, int G, int CPL>
constexpr int unpool_ctas() {
    if (Lay<T, G, CPL>::THREADS != 128) return G == 16 ? (CPL <= 2 ? 6 : 3) : CPL <= 2 ? 3 : CPL <= 3 ? 2 : 1;
    return Lay<T, G, CPL>::TPG * CPL <= 1 ? 16 : Lay<T, G, CPL>::TPG * CPL <= 2 ? 12 : 4;
}
template <typename T, int G, int CPL>
__global__ void __launch_bounds__((Lay<T, G, CPL>::THREADS), (unpool_ctas<T, G, CPL>()))
unpool_region_kernel(const T* __restrict__ q, const T* __restrict__ comp, const T* ref, T* out, RegionGeom g,
                     const int32_t* __restrict__ idx, const int32_t* __restrict__ region_first,
                     const int32_t* __restrict__ offsets, Splits sp, NextBlock nx) {
    pdl_begin();
    using L = Lay<T, G, CPL>;
    constexpr int VN = L::VN, GROUPS = L::GROUPS, TPG = L::TPG;
    extern __shared__ float part[];          // [SLOTS][C] sums of the output (next gate)
    const int lane = threadIdx.x & 31, sub = lane % G;
    const int gi = (int)(threadIdx.x >> 5) * GROUPS + lane / G;
    const int w = gi * TPG / RG, col0 = gi * TPG % RG;
    const int R = g.Hr * g.Wr;
    const int rid = blockIdx.x;

    if (rid >= g.B * R) {
        const int e = (rid - g.B * R) * (RG * RG / TPG) + gi;
        if (e >= g.B * g.num_extra) return;
        const int b = e / g.num_extra, t = e % g.num_extra;
        unpool_extra<T, G, CPL>(q, comp, ref, out, g, b, t, (size_t)(offsets[b] + t), sub, nx);
        return;
    }
    const int b = rid / R, rr = rid % R;
    const int ry = rr / g.Wr, rx = rr % g.Wr;
    const int k = min(max(idx[rid], 0), sp.n - 1);
    const int s = sp.v[k];
    const int step = RG / s;
    const int first = region_first[rid];
    const size_t tok0 = (size_t)b * g.N + g.num_extra + (size_t)(ry * RG + w) * g.W + rx * RG + col0;
    const int prow = first + (w / step) * s;            // packed row of this grid row's first patch

    // every row this group needs, requested up front: TPG reference rows and the patch rows they map to.
    // At the finest grain a token is its own patch and comp[p] is a copy of ref[tok], so
    // ref + (q - comp) is q: neither ref nor comp is read (a third of the regions on average; the
    // grain is the same for the whole CTA, so nothing diverges)
    const bool fine = step == 1;
    Vec<T> rrow[TPG][CPL], qrow[TPG][CPL], crow[TPG][CPL];
#pragma unroll
    for (int j = 0; j < TPG; ++j) {
        const int col = col0 + j;
        if (!fine) load_row<T, CPL>(rrow[j], ref + (tok0 + j) * g.C, sub, G);
        if (j == 0 || (col % step) == 0) {               // a new patch starts at this column
            const int p = prow + col / step;
            load_row<T, CPL>(qrow[j], q + (size_t)p * g.C, sub, G);
            if (!fine) load_row<T, CPL>(crow[j], comp + (size_t)p * g.C, sub, G);
        }
    }
    float acc[CPL][VN];                                  // in-order sum of this group's output tokens
    zero_f<T, CPL>(acc);
    float d[CPL][VN];
    zero_f<T, CPL>(d);
#pragma unroll
    for (int j = 0; j < TPG; ++j) {
        const int col = col0 + j;
        if (j == 0 || (col % step) == 0) {
            to_f<T, CPL>(d, qrow[j]);
            if (!fine) {
                float cf[CPL][VN];
                to_f<T, CPL>(cf, crow[j]);
#pragma unroll
                for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
                    for (int i = 0; i < VN; ++i) d[ch][i] -= cf[ch][i];
            }
        }
        float o[CPL][VN];
        if (fine) {
#pragma unroll
            for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
                for (int i = 0; i < VN; ++i) o[ch][i] = d[ch][i];
        } else {
            to_f<T, CPL>(o, rrow[j]);
#pragma unroll
            for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
                for (int i = 0; i < VN; ++i) o[ch][i] = d[ch][i] + o[ch][i];
        }
        round_store<T, CPL>(o, out + (tok0 + j) * g.C, sub, G);       // o now holds the rounded values
        if (nx.stats_x) {
            const float2 st = mean_rstd(row_sums<T, G, CPL>(o), g.C, nx.eps);
            if (sub == 0) nx.stats_x[tok0 + j] = st;
        }
        if (nx.gw) {
#pragma unroll
            for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
                for (int i = 0; i < VN; ++i) acc[ch][i] += o[ch][i];
        }
    }
    if (!nx.gw) return;
    // ---- the next block's router gate on the region this CTA has just written
    publish_partials<T, G, CPL>(part, acc, gi, sub, g.C);
    if (gi != 0) return;
    gate_from_partials<T, G, CPL>(part, g.C, sub, nx.gw, nx.gb, nx.S, nx.logits, nx.idx, rid,
                                  nx.counts ? nx.counts + b : nullptr, sp,
                                  nx.image_bias ? nx.image_bias + (size_t)b * nx.S : nullptr);
}

// The same with a warp per region, for many bf16 regions, bit for bit.  With a block per region 41 us of DeiT-S, 256 images, were 20 % of DRAM's rate and
// 42 % of the issue slots: 16 warps a SM, of which three wait while one works out the gate.  Here no barrier is left, arithmetic is on pairs
// of channels and the code is the grain's own; a warp walks down the four grid rows, the next one's values on their way.
// us of a launch, block -> warp: C = 384, 4096 regions (256 images) 37.7 -> 25.8, 1536 regions 17.0 -> 11.1; C = 64, 24576 regions (PVT-small, 96
// images) 50.6 -> 33; C = 128, 6144 22.0 -> 15.3; C = 320, 1536 15.2 -> 11.0.  Without the next row's loads 24.0 / 12.2 (C = 384); with a row's vectors
// loaded one chunk after the other, 24 warps a SM, 31.1 / 16.5.  112 MB in 25.8 us are
// 66 % of the copy rate, a third of them from L2; what is left is a warp's chain (159 registers, 12 warps a SM).
constexpr int UW_WARPS = 4;
template <int G, int CPL>
constexpr int unpool_warp_ctas() { return G * CPL >= 40 ? 3 : G * CPL > 16 ? 4 : G * CPL == 16 ? 6 : 8; }

// What a lane reads for a grid row at a grain of STEP x STEP: all of it on its way at once.
template <int G, int CPL, int STEP>
struct UnpoolRow {
    static constexpr int TPG = RG * G / 32, PATCHES = (TPG + STEP - 1) / STEP;
    static constexpr bool FINE = STEP == 1;              // (a token is its own patch: see above)
    Vec<bf16> row[FINE ? 1 : TPG][CPL], q[PATCHES][CPL], c[FINE ? 1 : PATCHES][CPL];
    __device__ __forceinline__ void load(const bf16* __restrict__ qp, const bf16* __restrict__ cp, const bf16* rp, int C, int sub) {
        if (!FINE)
#pragma unroll
            for (int j = 0; j < TPG; ++j) load_row<bf16, CPL>(row[FINE ? 0 : j], rp + (size_t)j * C, sub, G);
#pragma unroll
        for (int j = 0; j < PATCHES; ++j) {
            load_row<bf16, CPL>(q[j], qp + (size_t)j * C, sub, G);
            if (!FINE) load_row<bf16, CPL>(c[FINE ? 0 : j], cp + (size_t)j * C, sub, G);
        }
    }
};

// One region's tokens at a grain of STEP x STEP; acc (group 0): their sum.
template <int G, int CPL, int STEP>
__device__ __forceinline__ void unpool_rows(float (&acc)[CPL][8], const bf16* __restrict__ q, const bf16* __restrict__ comp, const bf16* ref,
                                            bf16* out, const RegionGeom& g, size_t tok0, int first, int sub, int grp, const NextBlock& nx) {
    using U = UnpoolRow<G, CPL, STEP>;
    constexpr int VN = 8, GROUPS = 32 / G, TPG = U::TPG;
    auto load = [&](U& u, int w) {
        const size_t from = (size_t)(first + (w / STEP) * (RG / STEP) + grp * TPG / STEP) * g.C;
        u.load(q + from, comp + from, ref + (tok0 + (size_t)w * g.W + grp * TPG) * g.C, g.C, sub);
    };
    U cur, next;
    load(cur, 0);
#pragma unroll 1
    for (int w = 0; w < RG; ++w) {
        if (w + 1 < RG) load(next, w + 1);
        const size_t tok = tok0 + (size_t)w * g.W + grp * TPG;
        float s1[TPG], s2[TPG];                          // of a token: the sums of row_sums, in its order
#pragma unroll
        for (int j = 0; j < TPG; ++j) s1[j] = s2[j] = 0.f;
#pragma unroll
        for (int ch = 0; ch < CPL; ++ch) {
            float2 sum[VN / 2], d[VN / 2];
#pragma unroll
            for (int j = 0; j < TPG; ++j) {
                Vec<bf16> o;
                if (U::FINE) {
                    o = cur.q[j / STEP][ch];
                } else {
                    if (j % STEP == 0)
#pragma unroll
                        for (int i = 0; i < VN / 2; ++i) d[i] = sub2(pair_of(cur.q[j / STEP][ch], i), pair_of(cur.c[U::FINE ? 0 : j / STEP][ch], i));
#pragma unroll
                    for (int i = 0; i < VN / 2; ++i) set_pair(o, i, add2(d[i], pair_of(cur.row[U::FINE ? 0 : j][ch], i)));
                }
                o.store(out + (tok + j) * g.C + (sub + G * ch) * VN);
#pragma unroll
                for (int i = 0; i < VN / 2; ++i) {
                    const float2 v = pair_of(o, i);                    // the rounded values
                    s1[j] = s1[j] + v.x + v.y;
                    s2[j] = fmaf(v.y, v.y, fmaf(v.x, v.x, s2[j]));
                    sum[i] = j == 0 ? v : add2(sum[i], v);
                }
            }
            if (nx.gw) {
#pragma unroll
                for (int i = 0; i < VN; ++i) {
                    float v = i & 1 ? sum[i / 2].y : sum[i / 2].x;
                    if (GROUPS == 4) v += __shfl_xor_sync(0xffffffffu, v, G);      // the left or right pair of the row
                    acc[ch][i] += v;
                    if (GROUPS >= 2) acc[ch][i] += __shfl_xor_sync(0xffffffffu, v, 16);
                }
            }
        }
        if (nx.stats_x) {
#pragma unroll
            for (int j = 0; j < TPG; ++j) {
                const float2 st = mean_rstd(make_float2(group_sum<G>(s1[j]), group_sum<G>(s2[j])), g.C, nx.eps);
                if (sub == 0) nx.stats_x[tok + j] = st;
            }
        }
        cur = next;
    }
}

template <int G, int CPL>
__global__ void __launch_bounds__(UW_WARPS * 32, (unpool_warp_ctas<G, CPL>()))
unpool_warp_kernel(const bf16* __restrict__ q, const bf16* __restrict__ comp, const bf16* ref, bf16* out, RegionGeom g,
                   const int32_t* __restrict__ idx, const int32_t* __restrict__ region_first,
                   const int32_t* __restrict__ offsets, Splits sp, NextBlock nx) {
    pdl_begin();
    constexpr int GROUPS = 32 / G;
    const int lane = threadIdx.x & 31, sub = lane % G, grp = lane / G, warp = threadIdx.x >> 5;
    const int R = g.Hr * g.Wr, regions = g.B * R, blocks = (regions + UW_WARPS - 1) / UW_WARPS;

    if ((int)blockIdx.x >= blocks) {                     // extra tokens, one per group
        const int e = (((int)blockIdx.x - blocks) * UW_WARPS + warp) * GROUPS + grp;
        if (e >= g.B * g.num_extra) return;
        const int b = e / g.num_extra, t = e % g.num_extra;
        unpool_extra<bf16, G, CPL>(q, comp, ref, out, g, b, t, (size_t)(offsets[b] + t), sub, nx);
        return;
    }
    const int rid = (int)blockIdx.x * UW_WARPS + warp;
    if (rid >= regions) return;
    const int b = rid / R, rr = rid % R;
    const int ry = rr / g.Wr, rx = rr % g.Wr;
    const int step = RG / sp.v[min(max(idx[rid], 0), sp.n - 1)];
    const int first = region_first[rid];
    const size_t tok0 = (size_t)b * g.N + g.num_extra + (size_t)ry * RG * g.W + rx * RG;
    float acc[CPL][8];
    zero_f<bf16, CPL>(acc);
    if (step == 1) unpool_rows<G, CPL, 1>(acc, q, comp, ref, out, g, tok0, first, sub, grp, nx);
    else if (step == 2) unpool_rows<G, CPL, 2>(acc, q, comp, ref, out, g, tok0, first, sub, grp, nx);
    else unpool_rows<G, CPL, 4>(acc, q, comp, ref, out, g, tok0, first, sub, grp, nx);
    if (nx.gw)
        gate_of_sum<bf16, G, CPL>(acc, g.C, sub, lane == 0, nx.gw, nx.gb, nx.S, nx.logits, nx.idx, rid, nx.counts ? nx.counts + b : nullptr, sp,
                                  nx.image_bias ? nx.image_bias + (size_t)b * nx.S : nullptr);
}

// Stand-alone gate (first block of a model, or a block called on its own); optionally also
// writes the LayerNorm statistics of every token row it reads.
template <typename T, int G, int CPL>
__global__ void __launch_bounds__((Lay<T, G, CPL>::THREADS))
gate_region_kernel(const T* __restrict__ x, RegionGeom g, const float* __restrict__ gw,
                   const float* __restrict__ gb, int S, float* __restrict__ logits_out,
                   int32_t* __restrict__ idx_out, float2* __restrict__ stats_x, float eps,
                   const float* __restrict__ image_bias, int32_t* __restrict__ counts, Splits sp) {
    pdl_begin();
    using L = Lay<T, G, CPL>;
    constexpr int VN = L::VN, GROUPS = L::GROUPS, TPG = L::TPG;
    extern __shared__ float part[];          // [SLOTS][C]
    const int lane = threadIdx.x & 31, sub = lane % G;
    const int gi = (int)(threadIdx.x >> 5) * GROUPS + lane / G;
    const int w = gi * TPG / RG, col0 = gi * TPG % RG;
    const int R = g.Hr * g.Wr;
    const int rid = blockIdx.x;
    if (rid >= g.B * R) {
        // extra (cls) tokens only matter for the statistics
        const int e = (rid - g.B * R) * (RG * RG / TPG) + gi;
        if (!stats_x || e >= g.B * g.num_extra) return;
        const size_t tok = (size_t)(e / g.num_extra) * g.N + e % g.num_extra;
        Vec<T> row[CPL];
        load_row<T, CPL>(row, x + tok * g.C, sub, G);
        float f[CPL][VN];
        to_f<T, CPL>(f, row);
        const float2 st = mean_rstd(row_sums<T, G, CPL>(f), g.C, eps);
        if (sub == 0) stats_x[tok] = st;
        return;
    }
    const int b = rid / R, rr = rid % R;
    const int ry = rr / g.Wr, rx = rr % g.Wr;
    const size_t tok0 = (size_t)b * g.N + g.num_extra + (size_t)(ry * RG + w) * g.W + rx * RG + col0;
    Vec<T> rows[TPG][CPL];
#pragma unroll
    for (int j = 0; j < TPG; ++j) load_row<T, CPL>(rows[j], x + (tok0 + j) * g.C, sub, G);
    float acc[CPL][VN];
    zero_f<T, CPL>(acc);
#pragma unroll
    for (int j = 0; j < TPG; ++j) {
        float f[CPL][VN];
        to_f<T, CPL>(f, rows[j]);
        if (stats_x) {
            const float2 st = mean_rstd(row_sums<T, G, CPL>(f), g.C, eps);
            if (sub == 0) stats_x[tok0 + j] = st;
        }
#pragma unroll
        for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
            for (int i = 0; i < VN; ++i) acc[ch][i] += f[ch][i];
    }
    publish_partials<T, G, CPL>(part, acc, gi, sub, g.C);
    if (gi != 0) return;
    gate_from_partials<T, G, CPL>(part, g.C, sub, gw, gb, S, logits_out, idx_out, rid, counts ? counts + b : nullptr, sp,
                                  image_bias ? image_bias + (size_t)b * S : nullptr);
}

// -------------------------------------------------------------- gated decompress (training)
// out[b,tok] = ref[b,tok] + (x[p] - comp[p]) * gate[region] for the patch p that covers the token, gate[region] being the value of the
// region's grain; extra tokens without a gate.  Differences and products are rounded to T, as the separate operations do.  One launch where
// those took eight, and the gradient one for eleven (DeiT-S layer, 48 images, forward and backward, whose time is the host's: 2.43 -> 2.18 ms).
template <typename T, int G, int CPL>
__device__ __forceinline__ void gated_rows(float (&d)[CPL][Vec<T>::N], const T* __restrict__ x, const T* __restrict__ comp, size_t p, int C, int sub) {
    Vec<T> xv[CPL], cv[CPL];
    load_row<T, CPL>(xv, x + p * C, sub, G);
    load_row<T, CPL>(cv, comp + p * C, sub, G);
    float c[CPL][Vec<T>::N];
    to_f<T, CPL>(d, xv);
    to_f<T, CPL>(c, cv);
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch) {
#pragma unroll
        for (int i = 0; i < Vec<T>::N; ++i) d[ch][i] -= c[ch][i];
        xv[ch].from_float(d[ch]);
        xv[ch].to_float(d[ch]);
    }
}
template <typename T, int CPL>
__device__ __forceinline__ void times(float (&d)[CPL][Vec<T>::N], float g) {
#pragma unroll
    for (int ch = 0; ch < CPL; ++ch) {
        Vec<T> v;
#pragma unroll
        for (int i = 0; i < Vec<T>::N; ++i) d[ch][i] = __fmul_rn(d[ch][i], g);      // (not part of an fma)
        v.from_float(d[ch]);
        v.to_float(d[ch]);
    }
}

template <typename T, int G, int CPL>
__global__ void __launch_bounds__((Lay<T, G, CPL>::THREADS))
gated_unpool_kernel(const GatedArgs a) {
    pdl_begin();
    using L = Lay<T, G, CPL>;
    constexpr int GROUPS = L::GROUPS, TPG = L::TPG;
    const T *x = (const T*)a.x, *comp = (const T*)a.comp, *ref = (const T*)a.ref;
    T* out = (T*)a.out;
    const RegionGeom& g = a.g;
    const int lane = threadIdx.x & 31, sub = lane % G;
    const int gi = (int)(threadIdx.x >> 5) * GROUPS + lane / G;
    const int w = gi * TPG / RG, col0 = gi * TPG % RG;
    const int R = g.Hr * g.Wr, rid = blockIdx.x;
    const bool extra = rid >= g.B * R;
    const int e = (rid - g.B * R) * (RG * RG / TPG) + gi;
    if (extra && e >= g.B * g.num_extra) return;
    const int b = extra ? e / g.num_extra : rid / R;
    int s = RG, first;
    float gate = 1.f;
    size_t tok0;
    if (extra) {
        first = a.offsets[b] + e % g.num_extra;
        tok0 = (size_t)b * g.N + e % g.num_extra;
    } else {
        const int k = min(max(a.idx[rid], 0), a.sp.n - 1), rr = rid % R;
        s = a.sp.v[k];
        first = a.region_first[rid];
        gate = to_f32(((const T*)a.gate)[(size_t)rid * a.sp.n + k]);
        tok0 = (size_t)b * g.N + g.num_extra + (size_t)(rr / g.Wr * RG + w) * g.W + rr % g.Wr * RG + col0;
    }
    if (first < 0 || first + (extra ? 1 : s * s) > g.l_max) {
        if (sub == 0 && a.status) atomicOr(a.status, STATUS_BAD_INDEX);
        return;
    }
    const int step = RG / s;
    float d[CPL][Vec<T>::N];
#pragma unroll
    for (int j = 0; j < TPG; ++j) {
        if (extra && j > 0) break;
        const int col = col0 + j;
        Vec<T> row[CPL];
        load_row<T, CPL>(row, ref + (tok0 + j) * g.C, sub, G);
        if (j == 0 || col % step == 0) {
            gated_rows<T, G, CPL>(d, x, comp, (size_t)(extra ? first : first + w / step * s + col / step), g.C, sub);
            if (!extra) times<T, CPL>(d, gate);
        }
        float o[CPL][Vec<T>::N];
        to_f<T, CPL>(o, row);
#pragma unroll
        for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
            for (int i = 0; i < Vec<T>::N; ++i) o[ch][i] = d[ch][i] + o[ch][i];
        round_store<T, CPL>(o, out + (tok0 + j) * g.C, sub, G);
    }
}

// Its gradients: r[p] = the sum of grad_out over the tokens of patch p (rounded to T); grad_x[p] = r[p] * gate, grad_comp = -grad_x, and
// grad_gate[region][its grain] = the sum over its patches of r[p] . (x - comp)[p], in fp32; 0 for the other grains.
template <typename T, int G, int CPL>
__global__ void __launch_bounds__((Lay<T, G, CPL>::THREADS))
gated_unpool_grad_kernel(const GatedArgs a) {
    pdl_begin();
    using L = Lay<T, G, CPL>;
    constexpr int VN = L::VN, GROUPS = L::GROUPS, TPG = L::TPG, ALL = L::THREADS / G;
    extern __shared__ float part[];          // [SLOTS][C] partial sums
    __shared__ float dots[ALL];
    const T *x = (const T*)a.x, *comp = (const T*)a.comp, *grad = (const T*)a.grad_out;
    T *gx = (T*)a.grad_x, *gc = (T*)a.grad_comp;
    const RegionGeom& g = a.g;
    const int lane = threadIdx.x & 31, sub = lane % G;
    const int gi = (int)(threadIdx.x >> 5) * GROUPS + lane / G;
    const int w = gi * TPG / RG, col0 = gi * TPG % RG;
    const int R = g.Hr * g.Wr, rid = blockIdx.x;
    float dot = 0.f;
    // one patch's row: the gradients, and its part of the gate's
    auto finish = [&](float (&sum)[CPL][VN], size_t p, float gate) {
        float d[CPL][VN];
        gated_rows<T, G, CPL>(d, x, comp, p, g.C, sub);
        times<T, CPL>(sum, 1.f);
#pragma unroll
        for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
            for (int i = 0; i < VN; ++i) dot = fmaf(sum[ch][i], d[ch][i], dot);
        times<T, CPL>(sum, gate);
        round_store<T, CPL>(sum, gx + p * g.C, sub, G);
#pragma unroll
        for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
            for (int i = 0; i < VN; ++i) sum[ch][i] = -sum[ch][i];
        round_store<T, CPL>(sum, gc + p * g.C, sub, G);
    };
    if (rid >= g.B * R) {
        const int e = (rid - g.B * R) * (RG * RG / TPG) + gi;
        if (e >= g.B * g.num_extra) return;
        const int b = e / g.num_extra, t = e % g.num_extra, p = a.offsets[b] + t;
        if (p < 0 || p >= g.l_max) {
            if (sub == 0 && a.status) atomicOr(a.status, STATUS_BAD_INDEX);
            return;
        }
        Vec<T> row[CPL];
        load_row<T, CPL>(row, grad + ((size_t)b * g.N + t) * g.C, sub, G);
        float f[CPL][VN];
        to_f<T, CPL>(f, row);
        finish(f, (size_t)p, 1.f);
        return;
    }
    const int k = min(max(a.idx[rid], 0), a.sp.n - 1), rr = rid % R, b = rid / R;
    const int s = a.sp.v[k], step = RG / s, first = a.region_first[rid];
    if (first < 0 || first + s * s > g.l_max) {
        if (threadIdx.x == 0 && a.status) atomicOr(a.status, STATUS_BAD_INDEX);
        return;
    }
    const float gate = to_f32(((const T*)a.gate)[(size_t)rid * a.sp.n + k]);
    const size_t tok0 = (size_t)b * g.N + g.num_extra + (size_t)(rr / g.Wr * RG + w) * g.W + rr % g.Wr * RG + col0;
    Vec<T> rows[TPG][CPL];
#pragma unroll
    for (int j = 0; j < TPG; ++j) load_row<T, CPL>(rows[j], grad + (tok0 + j) * g.C, sub, G);
    float acc[CPL][VN];
    zero_f<T, CPL>(acc);
#pragma unroll
    for (int j = 0; j < TPG; ++j) {
        float f[CPL][VN];
        to_f<T, CPL>(f, rows[j]);
        if (step == 1) {
            finish(f, (size_t)(first + w * RG + col0 + j), gate);
            continue;
        }
#pragma unroll
        for (int ch = 0; ch < CPL; ++ch)
#pragma unroll
            for (int i = 0; i < VN; ++i) acc[ch][i] += f[ch][i];
        if (TPG == 4 && step == 2 && j == 1) {
            smem_store<T, CPL>(part + (size_t)(w * 2) * g.C, acc, sub, G);
            zero_f<T, CPL>(acc);
        }
    }
    if (step != 1) {
        if (TPG == 4 && step == 2) {
            smem_store<T, CPL>(part + (size_t)(w * 2 + 1) * g.C, acc, sub, G);
            __syncthreads();
        } else {
            publish_partials<T, G, CPL>(part, acc, gi, sub, g.C);
        }
        if (gi < s * s) {
            const int dy = step == 2 ? gi >> 1 : 0, dx = step == 2 ? gi & 1 : 0;
            zero_f<T, CPL>(acc);
            if (step == 2) {
                add_row<T, G, CPL, 1>(acc, part, 2 * dy, dx, sub, g.C);
                add_row<T, G, CPL, 1>(acc, part, 2 * dy + 1, dx, sub, g.C);
            } else {
#pragma unroll 1
                for (int r2 = 0; r2 < RG; ++r2) add_row<T, G, CPL, 2>(acc, part, r2, 0, sub, g.C);
            }
            finish(acc, (size_t)(first + dy * s + dx), gate);
        }
    }
    dot = group_sum<G>(dot);
    if (sub == 0) dots[gi] = dot;
    __syncthreads();
    if (a.grad_gate && threadIdx.x < a.sp.n) {
        float sum = 0.f;
        for (int i = 0; i < ALL; ++i) sum += dots[i];
        ((T*)a.grad_gate)[(size_t)rid * a.sp.n + threadIdx.x] = from_f32<T>((int)threadIdx.x == k ? sum : 0.f);
    }
}

// ------------------------------------------------------------------------------- host

// (G, CPL) with G * CPL == number of 16-byte chunks in a row; false if the row does not factor
static bool pick_layout(int nchunks, int* G, int* CPL) {
    static const int cpls[] = {3, 2, 1, 6, 4, 5};      // 5: C = 320 (PVT stage 3) is 8 lanes x 5 chunks in bf16
    for (int c : cpls)
        for (int g = 32; g >= 8; g >>= 1)
            if (g * c == nchunks && (g == 32 || c <= 3 || c == 5)) { *G = g; *CPL = c; return true; }
    return false;
}

template <typename L>
static size_t region_smem(int C) { return (size_t)L::SLOTS * C * sizeof(float); }
// (static shared memory counts towards the 48 KB that need no leave)
template <typename Kernel>
static void allow_smem(Kernel kern, size_t bytes) {
    if (bytes > 47 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <typename T, int G, int CPL>
static void launch_pool_t(const RegionPoolArgs& a, cudaStream_t st) {
    const int R = a.g.Hr * a.g.Wr;
    using L = Lay<T, G, CPL>;
    const int grid = a.g.B * R + ceil_div(a.g.B * a.g.num_extra, RG * RG / L::TPG);
    const dim3 block(L::THREADS);
    const size_t smem = region_smem<L>(a.g.C);
    if constexpr (sizeof(T) == 4) {
        if (a.qn_terms) {
            const int split_grid = a.split.ctas(L::THREADS);
            allow_smem(pool_region_terms_kernel<G, CPL>, smem);
            launch_kernel(pool_region_terms_kernel<G, CPL>, true, 1, dim3(split_grid + grid), block, smem, st, (const float*)a.x, a.g,
                a.idx, a.region_first, a.offsets, a.counts, a.offsets_out, a.region_first_out, a.counts_next, a.sp, (float*)a.comp,
                a.lnw, a.lnb, a.eps, (float*)a.xn, (float*)a.qn, a.xn_terms ? 3 : 2, split_grid, a.split);
            return;
        }
    }
    if constexpr (sizeof(T) == 2 && G <= 16 && G * CPL <= 48) {
        // Eight regions a SM: the line of the unpool, which see; both forms write the same.  But for the rows of a convolution where channels are
        // many (three blocks a SM, each as long as a round of all) not while a second round is less than two fifths full.  Four blocks in a
        // chain, C = 320, sr = 2, us a block at three grain mixes, block | warp: 96 images (0.9 rounds) 101 106 133 | 96 103 132, 112 (1.01) 111 117
        // 151 | 111 117 151, 128 (1.2) 117 123 159 | 120 126 161, 144 (1.3) 125 131 169 | 125 132 169, 160 (1.4) 131 139 180 | 131 139 180, 192
        // (1.7) 142 161 212 | 138 159 213; a block with its gate given, 128 images, 109 116 154 | 114 121 157.
        const int blocks = ceil_div(a.g.B * R, PW_WARPS) + ceil_div(a.g.B * a.g.num_extra, PW_WARPS * L::GROUPS);
        const int round = pool_warp_ctas<G, CPL, POOL_COLS>() * sm_count();
        const bool short_round = a.sr > 1 && G * CPL >= 40 && blocks > round && 5 * blocks < 7 * round;
        if (a.stats_q && a.g.l_max == 0 && a.g.B * R >= 8 * sm_count() && !short_round) {
            auto kern = a.sr > 1 ? pool_warp_kernel<G, CPL, POOL_COLS> : pool_warp_kernel<G, CPL, POOL_STATS>;
            launch_chain(kern, dim3(blocks), dim3(PW_WARPS * 32), 0, st, (const T*)a.x, a.g, a.idx, a.region_first, a.offsets, a.counts,
                a.offsets_out, a.region_first_out, a.counts_next, a.sp, (T*)a.comp, a.stats_x, a.stats_q, a.stats_acc,
                a.stats_x_ready ? 0 : 1, a.lnw, a.lnb, a.eps, (T*)a.cols, a.sr);
            return;
        }
    }
    auto launch = [&](auto kern, auto... args) {
        allow_smem(kern, smem);
        launch_chain(kern, dim3(grid), block, smem, st, args...);
    };
    if (a.stats_q && a.sr > 1)
        launch(pool_region_kernel<T, G, CPL, POOL_COLS>,
            (const T*)a.x, a.g, a.idx, a.region_first, a.offsets, a.counts, a.offsets_out, a.region_first_out,
            a.counts_next, a.sp, (T*)a.comp, a.stats_x, a.stats_q, a.stats_acc, a.stats_x_ready ? 0 : 1, a.lnw,
            a.lnb, a.eps, (T*)a.cols, nullptr, 0, a.sr, nullptr);
    else if (a.stats_q)
        launch(pool_region_kernel<T, G, CPL, POOL_STATS>,
            (const T*)a.x, a.g, a.idx, a.region_first, a.offsets, a.counts, a.offsets_out, a.region_first_out,
            a.counts_next, a.sp, (T*)a.comp, a.stats_x, a.stats_q, a.stats_acc, a.stats_x_ready ? 0 : 1, nullptr,
            nullptr, a.eps, nullptr, nullptr, 0, 1, nullptr);
    else if (a.xn && a.qn)
        launch(pool_region_kernel<T, G, CPL, POOL_LN>,
            (const T*)a.x, a.g, a.idx, a.region_first, a.offsets, a.counts, a.offsets_out, a.region_first_out,
            a.counts_next, a.sp, (T*)a.comp, nullptr, nullptr, nullptr, 0, a.lnw, a.lnb, a.eps, (T*)a.xn, (T*)a.qn, 0, 1, nullptr);
    else
        launch(pool_region_kernel<T, G, CPL, POOL_PLAIN>,
            (const T*)a.x, a.g, a.idx, a.region_first, a.offsets, a.counts, a.offsets_out, a.region_first_out,
            a.counts_next, a.sp, (T*)a.comp, nullptr, nullptr, nullptr, 0, nullptr, nullptr, a.eps, nullptr, nullptr,
            a.sum_only ? 1 : 0, 1, device_status_ptr());
}

template <typename T, int G, int CPL>
static void launch_unpool_t(const RegionUnpoolArgs& a, cudaStream_t st) {
    const int R = a.g.Hr * a.g.Wr;
    using L = Lay<T, G, CPL>;
    const int grid = a.g.B * R + ceil_div(a.g.B * a.g.num_extra, RG * RG / L::TPG);
    // A warp per region from eight regions a SM on: with fewer its chain, four grid rows in turn, is longer than that of a block per region.
    // DeiT-S forward, block | warp, us: 32 images (3.5 a SM) 800 | 838, 64 (6.9) 1130 | 1133, 96 (10.4) 1481 | 1408; DeiT-Ti, 64 images
    // 796 | 789, 96 939 | 890, 128 1109 | 1036.  Rows of a whole warp (C = 512, 768) are four tokens in a row each: 7 | 21 us, not used.
    if constexpr (sizeof(T) == 2 && G <= 16 && G * CPL <= 48) {
        if (a.g.B * R >= 8 * sm_count()) {
            const int blocks = ceil_div(a.g.B * R, UW_WARPS) + ceil_div(a.g.B * a.g.num_extra, UW_WARPS * L::GROUPS);
            launch_chain(unpool_warp_kernel<G, CPL>, dim3(blocks), dim3(UW_WARPS * 32), 0, st, (const T*)a.q, (const T*)a.comp, (const T*)a.ref,
                (T*)a.out, a.g, a.idx, a.region_first, a.offsets, a.sp, a.next);
            return;
        }
    }
    const size_t smem = a.next.gw ? region_smem<L>(a.g.C) : 0;
    allow_smem(unpool_region_kernel<T, G, CPL>, smem);
    launch_chain(unpool_region_kernel<T, G, CPL>, dim3(grid), dim3(L::THREADS), smem, st,
        (const T*)a.q, (const T*)a.comp, (const T*)a.ref, (T*)a.out, a.g, a.idx, a.region_first, a.offsets, a.sp, a.next);
}

template <typename T, int G, int CPL>
static void launch_gate_t(const RegionGateArgs& a, cudaStream_t st) {
    const int R = a.g.Hr * a.g.Wr;
    using L = Lay<T, G, CPL>;
    const int grid = a.g.B * R + (a.stats_x ? ceil_div(a.g.B * a.g.num_extra, RG * RG / L::TPG) : 0);
    const size_t smem = region_smem<L>(a.g.C);
    allow_smem(gate_region_kernel<T, G, CPL>, smem);
    launch_chain(gate_region_kernel<T, G, CPL>, dim3(grid), dim3(L::THREADS), smem, st,
        (const T*)a.x, a.g, a.gw, a.gb, a.S, a.logits_out, a.idx_out, a.stats_x, a.eps, a.image_bias, a.counts, a.sp);
}

template <typename T, int G, int CPL>
static void launch_gated_t(const GatedArgs& a, cudaStream_t st) {
    using L = Lay<T, G, CPL>;
    const dim3 grid(a.g.B * a.g.Hr * a.g.Wr + ceil_div(a.g.B * a.g.num_extra, RG * RG / L::TPG)), block(L::THREADS);
    if (!a.grad_out) {
        launch_chain(gated_unpool_kernel<T, G, CPL>, grid, block, 0, st, a);
        return;
    }
    const size_t smem = region_smem<L>(a.g.C);
    allow_smem(gated_unpool_grad_kernel<T, G, CPL>, smem);
    launch_chain(gated_unpool_grad_kernel<T, G, CPL>, grid, block, smem, st, a);
}

#define VTP_DISPATCH_LAYOUT(FN, T, ARGS, ST)                                    \
    do {                                                                        \
        int G = 0, CPL = 0;                                                     \
        if (!pick_layout((ARGS).g.C / Vec<T>::N, &G, &CPL))                     \
            return fail(VTP_ERR_SHAPE, "C=%d has no lane layout", (ARGS).g.C);  \
        if (G == 32 && CPL == 3) FN<T, 32, 3>(ARGS, ST);                        \
        else if (G == 16 && CPL == 3) FN<T, 16, 3>(ARGS, ST);                   \
        else if (G == 8 && CPL == 3) FN<T, 8, 3>(ARGS, ST);                     \
        else if (G == 32 && CPL == 2) FN<T, 32, 2>(ARGS, ST);                   \
        else if (G == 16 && CPL == 2) FN<T, 16, 2>(ARGS, ST);                   \
        else if (G == 8 && CPL == 2) FN<T, 8, 2>(ARGS, ST);                     \
        else if (G == 32 && CPL == 1) FN<T, 32, 1>(ARGS, ST);                   \
        else if (G == 16 && CPL == 1) FN<T, 16, 1>(ARGS, ST);                   \
        else if (G == 8 && CPL == 1) FN<T, 8, 1>(ARGS, ST);                     \
        else if (G == 32 && CPL == 6) FN<T, 32, 6>(ARGS, ST);                   \
        else if (G == 32 && CPL == 4) FN<T, 32, 4>(ARGS, ST);                   \
        else if (G == 32 && CPL == 5) FN<T, 32, 5>(ARGS, ST);                   \
        else if (G == 16 && CPL == 5) FN<T, 16, 5>(ARGS, ST);                   \
        else if (G == 8 && CPL == 5) FN<T, 8, 5>(ARGS, ST);                     \
        else return fail(VTP_ERR_SHAPE, "C=%d has no lane layout", (ARGS).g.C); \
    } while (0)

template <typename T> int region_pool_t(const RegionPoolArgs& a, cudaStream_t st) {
    VTP_DISPATCH_LAYOUT(launch_pool_t, T, a, st);
    return check_launch("pool (region)");
}
template <typename T> int region_unpool_t(const RegionUnpoolArgs& a, cudaStream_t st) {
    VTP_DISPATCH_LAYOUT(launch_unpool_t, T, a, st);
    return check_launch("unpool (region)");
}
template <typename T> int region_gate_t(const RegionGateArgs& a, cudaStream_t st) {
    VTP_DISPATCH_LAYOUT(launch_gate_t, T, a, st);
    return check_launch("router gate (region)");
}
template <typename T> int region_gated_t(const GatedArgs& a, cudaStream_t st) {
    VTP_DISPATCH_LAYOUT(launch_gated_t, T, a, st);
    return check_launch("gated unpool (region)");
}
#undef VTP_DISPATCH_LAYOUT

}  // namespace vtp
