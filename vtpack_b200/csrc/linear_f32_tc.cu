// fp32 Linear on tcgen05 tensor cores, at fp32 accuracy.
//
//   y[m, n] = act(sum_k a[m,k] w[n,k] + bias[n]) + res[m, n],   everything fp32
//
// Every operand element is split into three bf16 terms, 2^16 x = h + m + l (8 significant bits each, so the three hold
// the 24 bits of an fp32 number), and a k-block's product is the sum of six bf16 products accumulated in fp32:
//   l*h + h*l + m*m + m*h + h*m + h*h      (smallest first; the sum of the three left out is below 2^-23 of |a||w|,
// m*l and l*m below 2^-24 each).  The factor 2^16 takes the last bit of the smallest fp32 number, 2^-149, to that of
// the smallest bf16 number, 2^-133, so that the split is exact for every finite operand (without it, operands below
// 2^-111 lost bits: 2e-5 of the result at 2^-118); a finished sum is multiplied by 2^-32.  (DeiT-S, 12 images: 1 %.)
// The tensor core keeps an accumulator for one k-block (64) only; epilogue warps add the k-blocks in fp32
// registers, rounding to nearest, so a long reduction does not collect the accumulator's own rounding.  Measured
// against float64 the result is as close as the CUDA-core kernel's sequential fmaf chain (tests/test_gpu_ops.py).
//
// For fp32 operands as they are: single Linears, the patch embedding, the head, dense blocks.  The Linears of a DGE block read operands
// that are terms already (linear_f32_terms.cu); figures of a forward below are from when they ran here.
//
// Bound: the SM's shared-memory / L1 port (128 bytes per clock).  A k-block of a 128 x 64 tile passes 96 KB of loads
// through the L1, 72 KB of operand writes and 144 KB of operand reads (24 MMAs), 2450 cycles, which is its measured
// time; fewer MMAs or no operand writes shorten it in proportion, more converter warps do not.  32-byte loads move the
// same bytes in half as many requests (8192 x 8192 x 2048: 2185 -> 1860 us).  DeiT-S, 12 images: the CUDA-core kernel
// took 70 us per launch (11 TFLOP/s), 4.3 of the 5.8 ms of a forward.
//
// A long reduction with few tiles (fc2 of a small batch: 54 tiles, 24 k-blocks) is split over the CTAs of a cluster:
// each takes a share of the k-blocks, they exchange their partial sums through distributed shared memory, and each
// finishes a slice of the tile's columns.  The sums are formed the same way whether it is split or not, so that a
// row's bits depend on K alone and not on how many rows and tiles a launch has: the k-blocks are cut into one, two or
// four groups by their number, a group is added up from zero, and the groups are added as (0 + 1) + (2 + 3).  A CTA
// with several groups keeps the sums of the earlier ones in tensor memory (three loads and stores a tile: DeiT-S, 12
// images, 2453 -> 2507 us against sums that were grouped by the number of tiles).
//
// Persistent, one CTA per SM, 128 x BN tiles (BN = 64 where 128-wide tiles would leave SMs idle):
//   warps 0-10 / 0-14  fetch the next k-block with 16-byte loads one k-block ahead (in registers), split it and write the
//                six operand tiles as 128-byte-swizzled rows (no TMA: the split has to pass through registers)
//   one warp     issues the MMAs into one of two TMEM accumulators, one per k-block
//   eight warps  add finished accumulators to their registers (one row x BN / 2 columns per thread); after the last
//                k-block bias / GELU / residual and 128-byte stores through a per-warp shared-memory transpose
//
// An infinite or NaN operand (and a finite one of 2^112 or more, whose first term is inf) turns every sum it enters into
// NaN through its second term, inf - inf, and a sum of 2^96 or more comes out infinite.  Sums that come out non-finite
// are therefore worked out again as a plain fmaf chain over the fp32 operands (unscale_or_redo): results are infinite,
// NaN or finite where that chain's are.  The check is one fmaf per output.
//
// Replaces nn.Linear q/kv/proj/fc1/fc2/head, nn.GELU and the residual adds of
// vtpack/models/dge/deit_dge.py:38-44,72-74,96,127-128 in fp32, where the operands are fp32 rows: single Linears, patch embedding,
// head and dense blocks.  The Linears of DGE blocks are linear_f32_terms.cu.
#include "f32_terms.cuh"
#include "linear.h"
#include "linear_f32.cuh"
#include "runtime.h"
#include "sm100.cuh"

namespace vtp {

using namespace sm100;

constexpr int F_EPI = 256;              // epilogue threads
// Converter warps: as many as the registers of an SM allow beside the tile's accumulators.  (Eight measured the
// same: the port is the bound, see above.)
constexpr int conv_warps(int bn) { return bn == 128 ? 11 : 15; }
constexpr int F_STAGES = 2;

template <int BN>
struct F32Smem {
    static constexpr int A_TERM = FM * FK * 2, B_TERM = BN * FK * 2;
    static constexpr int STAGE = 3 * (A_TERM + B_TERM);
    static constexpr int OUT = (F_EPI / 32) * 32 * 128;        // per epilogue warp: 32 rows x 32 fp32 columns
    static constexpr int USED = F_STAGES * STAGE + OUT + 128;
    static constexpr int TOTAL = USED + 1024;                   // the operand tiles want 1024-byte alignment
    static_assert(TOTAL <= 232448, "shared memory budget");
};

struct F32Args {
    const float* a; long long lda; const float* w; const float* bias; const float* res; long long ldr;
    float* y; long long ldy;
    int m_max; const int32_t* m_dev; int N, K; int gelu, wide;       // wide: 32-byte loads
    int groups_log2;                                                  // groups of k-blocks, see f32_groups_log2
    RowMap rm;
};

// Eight consecutive fp32 values: one 32-byte load.
__device__ __forceinline__ void ldg_f8(const float* p, float4& lo, float4& hi) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(lo.x), "=f"(lo.y), "=f"(lo.z), "=f"(lo.w), "=f"(hi.x), "=f"(hi.y), "=f"(hi.z), "=f"(hi.w)
                 : "l"(p));
}

// Eight fp32 values -> the three bf16 terms, packed eight to 16 bytes.
__device__ __forceinline__ void split8(const float4& x0, const float4& x1, uint4 (&t)[3]) {
    const float v[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
    uint32_t w[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t h[2], m[2], l[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) split_scaled(v[2 * i + j] * F_SCALE, h[j], m[j], l[j]);
        w[0][i] = __byte_perm(h[0], h[1], 0x7632);       // the upper halves of both: element 2 i in the low half
        w[1][i] = __byte_perm(m[0], m[1], 0x7632);
        w[2][i] = __byte_perm(l[0], l[1], 0x7632);
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) t[p] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

// acc: NC columns n0.. of row m0 + lane, sums of scaled products, which are scaled back.  Rows with a sum that is not
// finite are worked out again, a row at a time, a lane per column (K and lda are multiples of four floats, see linear_f32_tc_supported).
template <int NC>
__device__ __forceinline__ void unscale_or_redo(float (&acc)[NC], const F32Args& g, int M, int m0, int n0, int lane) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        t = fmaf(acc[i], 0.f, t);              // inf * 0 and NaN * 0 are NaN
        acc[i] *= F_UNSCALE;
    }
    unsigned bad = __ballot_sync(0xffffffffu, t != t && m0 + lane < M);
    while (bad) {
        const int r = __ffs(bad) - 1;
        bad &= bad - 1;
        const float4* a = reinterpret_cast<const float4*>(g.a + (size_t)(m0 + r) * g.lda);
#pragma unroll
        for (int c0 = 0; c0 < NC; c0 += 32) {
            const int n = n0 + c0 + lane;
            float s = 0.f;
            if (c0 + lane < NC && n < g.N) {
                const float4* w = reinterpret_cast<const float4*>(g.w + (size_t)n * g.K);
#pragma unroll 1
                for (int k = 0; k < g.K / 4; ++k) {
                    const float4 x = __ldg(a + k), y = __ldg(w + k);
                    s = fmaf(x.x, y.x, s); s = fmaf(x.y, y.y, s); s = fmaf(x.z, y.z, s); s = fmaf(x.w, y.w, s);
                }
            }
#pragma unroll
            for (int i = 0; i < 32 && c0 + i < NC; ++i) {
                const float v = __shfl_sync(0xffffffffu, s, i);
                if (lane == r) acc[c0 + i] = v;
            }
        }
    }
}

// SPLIT: CTAs of a cluster that share a tile's reduction (1: none); it divides the number of groups.
template <int BN, int SPLIT>
__global__ void __launch_bounds__(conv_warps(BN) * 32 + 32 + F_EPI, 1)
linear_f32_tc_kernel(const F32Args g, int* status) {
    using S = F32Smem<BN>;
    constexpr int NCW = conv_warps(BN);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + F_STAGES * S::STAGE + S::OUT);
    uint64_t* full = bars;                        // [2] a stage's operand tiles are written
    uint64_t* empty = bars + 2;                   // [2] its MMAs have read them
    uint64_t* acc_full = bars + 4;                // [2]
    uint64_t* acc_empty = bars + 6;               // [2]
    uint64_t* part_full = bars + 8;               // the other CTAs' partial sums of this CTA's columns have arrived
    uint64_t* part_free = bars + 9;               // the other CTAs have added the ones this CTA sent them
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* void_s = reinterpret_cast<int*>(tmem_slot + 2);   // [2] launch_is_void in front of the wait and behind it
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&full[i], NCW);
            mbar_init(&empty[i], 1);
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], F_EPI / 32);
        }
        mbar_init(part_full, SPLIT > 1 ? (SPLIT - 1) * (F_EPI / 32) : 1);
        mbar_init(part_free, SPLIT > 1 ? (SPLIT - 1) * (F_EPI / 32) : 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == NCW) {
        tmem_alloc(tmem_slot, F_TMEM * BN);
        tmem_relinquish();
    }
    if (threadIdx.x == (NCW + 1) * 32) void_s[0] = launch_is_void(status) ? 1 : 0;
    tc_fence_before_sync();
    __syncthreads();
    if (SPLIT > 1) cluster_sync_all();            // the partners' barriers exist
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const bool known_void = lead_word<SPLIT>(void_s) != 0;
    pdl_begin();

    int M = g.m_max;
    if (g.m_dev) M = min(*reinterpret_cast<const volatile int32_t*>(g.m_dev), g.m_max);
    const int n_tiles = (g.N + BN - 1) / BN;
    const int total = known_void ? 0 : ((M + FM - 1) / FM) * n_tiles;
    const int rank = SPLIT > 1 ? (int)cluster_ctarank() : 0;
    const int all_kb = (g.K + FK - 1) / FK;
    const int kb0 = all_kb * rank / SPLIT, num_kb = all_kb * (rank + 1) / SPLIT - kb0;    // this CTA's k-blocks
    const int first_tile = (int)blockIdx.x / SPLIT, tile_step = (int)gridDim.x / SPLIT;

    if (warp < NCW) {
        // ------------------------------------------------------------ fetch, split, stage
        // a unit = 8 consecutive k of one row (two 16-byte loads, 16 bytes of each term); a warp takes four rows of a
        // at a time or four of w: eight lanes cover a row's 64, so a quarter-warp writes one whole swizzled row
        constexpr int GROUPS = (FM + BN) / 4, U = (GROUPS + NCW - 1) / NCW;
        const int ch = lane & 7;
        float4 raw[U][2];
        const float* src[U];                            // row of the tile whose k-blocks are being fetched; null: zeros
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        auto aim = [&](int tile) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int row = (warp + u * NCW) * 4 + (lane >> 3);
                const int gm = (tile / n_tiles) * FM + row, gn = (tile % n_tiles) * BN + row - FM;
                const bool is_a = row < FM;
                src[u] = is_a ? g.a + (size_t)gm * g.lda : g.w + (size_t)gn * g.K;
                if (row >= FM + BN || (is_a ? gm >= M : gn >= g.N)) src[u] = nullptr;
            }
        };
        auto fetch = [&](int u, int kb) {
            const int k = (kb0 + kb) * FK + ch * 8;
            const bool ok = src[u] != nullptr;
            if (g.wide) {
                raw[u][0] = raw[u][1] = zero;
                if (ok && k + 8 <= g.K) ldg_f8(src[u] + k, raw[u][0], raw[u][1]);
                return;
            }
            raw[u][0] = (ok && k + 4 <= g.K) ? __ldg(reinterpret_cast<const float4*>(src[u] + k)) : zero;
            raw[u][1] = (ok && k + 8 <= g.K) ? __ldg(reinterpret_cast<const float4*>(src[u] + k) + 1) : zero;
        };
        const uint32_t sbase = smem_u32(base);
        int it = 0;
        bool ok = true;
        if (first_tile < total) {
            aim(first_tile);
#pragma unroll
            for (int u = 0; u < U; ++u) fetch(u, 0);
        }
        for (int tile = first_tile; tile < total && ok; tile += tile_step) {
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                const int s = it & 1;
                ok = mbar_wait(&empty[s], ((it >> 1) & 1) ^ 1, abort_flag, status, STATUS_GEMM_PRODUCER);
                if (!ok) {
                    // a lane that gives up still meets the others in the __syncwarp of every k-block that is left (a vote behind
                    // the wait costs these warps registers: DeiT-S, 12 images, 2370 -> 2408 us)
                    for (int n = (total - 1 - tile) / tile_step * num_kb + num_kb - kb; n > 0; --n) __syncwarp();
                    break;
                }
                const bool same = kb + 1 < num_kb, more = same || tile + tile_step < total;
                if (!same && more) aim(tile + tile_step);
                const int kb_n = same ? kb + 1 : 0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int row = (warp + u * NCW) * 4 + (lane >> 3);
                    if (GROUPS % NCW != 0 && row >= FM + BN) continue;
                    uint4 t[3];
                    split8(raw[u][0], raw[u][1], t);
                    if (more) fetch(u, kb_n);                           // in flight for a whole k-block
                    const bool is_a = row < FM;
                    const int r = is_a ? row : row - FM;
                    const uint32_t at = sbase + s * S::STAGE + (is_a ? 0 : 3 * S::A_TERM) + (uint32_t)r * 128u +
                                        ((uint32_t)(ch ^ (r & 7)) << 4);
                    const uint32_t step = is_a ? S::A_TERM : S::B_TERM;
#pragma unroll
                    for (int p = 0; p < 3; ++p) sts_u4(at + p * step, t[p]);
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
            }
        }
    } else if (warp == NCW) {
        if (elect_one()) {
            // -------------------------------------------------------------- MMA issuer
            const uint32_t idesc = idesc_bf16_f32(FM, BN, 0, 0);
            const uint32_t sbase = smem_u32(base);
            // (term of a, term of w): smallest products first
            constexpr int TA[6] = {2, 0, 1, 1, 0, 0}, TB[6] = {0, 2, 1, 0, 1, 0};
            int it = 0;
            bool ok = true;
            for (int tile = first_tile; tile < total && ok; tile += tile_step) {
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it & 1;
                    const uint32_t ph = (it >> 1) & 1;
                    ok = mbar_wait(&acc_empty[s], ph ^ 1, abort_flag, status, STATUS_GEMM_MMA) &&
                         mbar_wait(&full[s], ph, abort_flag, status, STATUS_GEMM_MMA);
                    if (!ok) break;
                    tc_fence_after_sync();
                    const uint32_t sa = sbase + s * S::STAGE, sb = sa + 3 * S::A_TERM;
#pragma unroll
                    for (int c = 0; c < 6; ++c) {
                        const uint64_t ad = smem_desc_sw128(sa + TA[c] * S::A_TERM);
                        const uint64_t bd = smem_desc_sw128(sb + TB[c] * S::B_TERM);
#pragma unroll
                        for (int k = 0; k < FK / 16; ++k)
                            umma_ss(tmem_base + s * BN, ad + 2 * k, bd + 2 * k, idesc, (c | k) != 0 ? 1u : 0u);
                    }
                    umma_commit(&empty[s]);
                    umma_commit(&acc_full[s]);
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------- epilogue
        constexpr int CW = BN / 2;                       // columns per thread: half a tile row
        const int ew = warp - NCW - 1;
        const int quarter = warp & 3;                    // TMEM lane quarter this warp may read
        const int half = ew >> 2;                        // the first four: left half of the columns, the others: right half
        const uint32_t tacc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * CW;
        const uint32_t stage = smem_u32(base + F_STAGES * S::STAGE) + ew * (32 * 128);
        const bool vec = g.N % 4 == 0 && g.ldy % 4 == 0 && (!g.res || g.ldr % 4 == 0);
        const int own_groups = (1 << g.groups_log2) / SPLIT;         // this CTA's: 1, 2 or 4
        const uint32_t tsum = tacc + 2 * BN;             // sums of its earlier groups: 0 (+ 1), and 2
        // in a launch that turns out to be void the sums still change hands, but this CTA has no rows to store
        if (threadIdx.x == (NCW + 1) * 32) void_s[1] = launch_is_void(status) ? 1 : 0;
        named_barrier(1, F_EPI);
        if (void_s[1] != 0) M = 0;
        int it = 0, n_done = 0;                           // k-blocks, tiles
        bool ok = true;
        for (int tile = first_tile; tile < total && ok; tile += tile_step, ++n_done) {
            const int m0 = (tile / n_tiles) * FM + quarter * 32, n0 = (tile % n_tiles) * BN + half * CW;
            float acc[CW];
#pragma unroll
            for (int i = 0; i < CW; ++i) acc[i] = 0.f;
            int grp = 0;
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                const int s = it & 1;
                ok = mbar_wait_warp(&acc_full[s], (it >> 1) & 1, abort_flag, status, STATUS_GEMM_EPILOGUE);
                if (!ok) break;
                tc_fence_after_sync();
#pragma unroll
                for (int c0 = 0; c0 < CW; c0 += 32) {
                    uint32_t r[32];
                    __syncwarp();
                    tmem_ld_32x32(tacc + s * BN + c0, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) acc[c0 + i] += __uint_as_float(r[i]);
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[s]);
                if constexpr (SPLIT < 4) {
                    // the CTA has one group, or this k-block does not end one
                    if (own_groups == 1 || kb + 1 != (all_kb * (rank * own_groups + grp + 1) >> g.groups_log2) - kb0) continue;
                    if (grp & 1) stash_add<CW>(tsum + (SPLIT == 1 ? (grp >> 1) * BN : 0), acc);
                    if (SPLIT == 1 && grp == 3) stash_add<CW>(tsum, acc);            // (0 + 1) + (2 + 3)
                    if (++grp == own_groups) continue;
                    stash_store<CW>(tsum + (SPLIT == 1 && grp == 3 ? BN : 0), acc);
#pragma unroll
                    for (int i = 0; i < CW; ++i) acc[i] = 0.f;
                }
            }
            if (!ok) break;
            if constexpr (SPLIT > 1) {
                // every CTA of the cluster finishes SC of this warp's columns: the others' partial sums of them come
                // through distributed shared memory (one slot per source CTA in the transpose buffers), 512
                // consecutive bytes per store
                constexpr int SC = CW / SPLIT;
                static_assert(CW * 32 * 4 <= 32 * 128 && SC % 4 == 0, "the exchange fits the warp's transpose buffer");
                if (n_done > 0) ok = mbar_wait_cluster_warp(part_free, (n_done - 1) & 1, abort_flag, status, STATUS_GEMM_EPILOGUE);
                if (!ok) break;
#pragma unroll
                for (int d = 0; d < SPLIT; ++d) {
                    if (d == rank) continue;
                    const uint32_t dst = mapa_u32(stage, d) + (rank < d ? rank : rank - 1) * (SC * 128) + lane * 16;
#pragma unroll
                    for (int j = 0; j < SC / 4; ++j) {
                        const int c = d * SC + 4 * j;
                        stc_f4(dst + j * 512, make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]));
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive_release_cluster(mapa_u32(smem_u32(part_full), d));
                }
                ok = mbar_wait_cluster_warp(part_full, n_done & 1, abort_flag, status, STATUS_GEMM_EPILOGUE);
                if (!ok) break;
                float own[SC];
#pragma unroll
                for (int d = 0; d < SPLIT; ++d)                   // (a runtime index would put acc into local memory)
                    if (d == rank) {
#pragma unroll
                        for (int j = 0; j < SC; ++j) own[j] = acc[d * SC + j];
                    }
                // four partial sums: this CTA's pair first, then the other pair's sum (slots are in source order without
                // this CTA: 1 2 3, 0 2 3, 0 1 3, 0 1 2)
                const uint32_t mine = stage + lane * 16 + (SPLIT == 4 && rank >= 2 ? 2 : 0) * (SC * 128);
                const uint32_t other = stage + lane * 16 + (rank >= 2 ? 0 : 1) * (SC * 128);
#pragma unroll
                for (int j = 0; j < SC / 4; ++j) {
                    const float4 p = lds_f4(mine + j * 512);
                    own[4 * j] += p.x; own[4 * j + 1] += p.y; own[4 * j + 2] += p.z; own[4 * j + 3] += p.w;
                    if constexpr (SPLIT == 4) {
                        const float4 a = lds_f4(other + j * 512), c = lds_f4(other + SC * 128 + j * 512);
                        own[4 * j] += a.x + c.x; own[4 * j + 1] += a.y + c.y;
                        own[4 * j + 2] += a.z + c.z; own[4 * j + 3] += a.w + c.w;
                    }
                }
                __syncwarp();
                if (lane == 0) {
#pragma unroll
                    for (int d = 0; d < SPLIT; ++d)
                        if (d != rank) mbar_arrive_release_cluster(mapa_u32(smem_u32(part_free), d));
                }
                unscale_or_redo<SC>(own, g, M, m0, n0 + rank * SC, lane);
                const int m = m0 + lane;
                if (m >= M) continue;
                float* y = g.y + map_out_row(g.rm, m) * g.ldy;
                const float* r = g.res ? g.res + map_res_row(g.rm, m) * g.ldr : nullptr;
#pragma unroll
                for (int j = 0; j < SC; j += 4) {
                    const int n = n0 + rank * SC + j;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        own[j + i] += (g.bias && n + i < g.N) ? __ldg(g.bias + n + i) : 0.f;
                        if (g.gelu) own[j + i] = gelu_erf(own[j + i]);
                    }
                    if (vec && n < g.N) {
                        float4 v = make_float4(own[j], own[j + 1], own[j + 2], own[j + 3]);
                        if (r) {
                            const float4 r4 = *reinterpret_cast<const float4*>(r + n);
                            v.x += r4.x; v.y += r4.y; v.z += r4.z; v.w += r4.w;
                        }
                        *reinterpret_cast<float4*>(y + n) = v;
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (n + i < g.N) y[n + i] = own[j + i] + (r ? r[n + i] : 0.f);
                    }
                }
                continue;
            }
            unscale_or_redo<CW>(acc, g, M, m0, n0, lane);
            // 32 columns at a time through the warp's transpose buffer (rows of eight 16-byte chunks, XOR-swizzled):
            // a lane then holds four columns of a row and eight lanes a whole 128-byte line
#pragma unroll
            for (int c0 = 0; c0 < CW; c0 += 32) {
                __syncwarp();                             // the previous block has been read
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    sts_u4(stage + lane * 128 + ((j ^ (lane & 7)) << 4),
                           make_uint4(__float_as_uint(acc[c0 + 4 * j]), __float_as_uint(acc[c0 + 4 * j + 1]),
                                      __float_as_uint(acc[c0 + 4 * j + 2]), __float_as_uint(acc[c0 + 4 * j + 3])));
                __syncwarp();
                const int n = n0 + c0 + (lane & 7) * 4;
                float bb[4] = {0.f, 0.f, 0.f, 0.f};
                if (g.bias) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) bb[i] = n + i < g.N ? __ldg(g.bias + n + i) : 0.f;
                }
#pragma unroll 2
                for (int q = 0; q < 8; ++q) {
                    const int rr = q * 4 + (lane >> 3), m = m0 + rr;
                    const float4 v4 = lds_f4(stage + rr * 128 + (((lane & 7) ^ (rr & 7)) << 4));
                    if (m >= M || n >= g.N) continue;
                    float v[4] = {v4.x + bb[0], v4.y + bb[1], v4.z + bb[2], v4.w + bb[3]};
                    if (g.gelu) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) v[i] = gelu_erf(v[i]);
                    }
                    float* y = g.y + map_out_row(g.rm, m) * g.ldy + n;
                    const float* r = g.res ? g.res + map_res_row(g.rm, m) * g.ldr + n : nullptr;
                    if (vec) {
                        if (r) {
                            const float4 r4 = *reinterpret_cast<const float4*>(r);
                            v[0] += r4.x; v[1] += r4.y; v[2] += r4.z; v[3] += r4.w;
                        }
                        *reinterpret_cast<float4*>(y) = make_float4(v[0], v[1], v[2], v[3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (n + i < g.N) y[i] = v[i] + (r ? r[i] : 0.f);
                    }
                }
            }
        }
    }
    if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) { }     // let MMAs in flight finish before releasing memory
    }
    tc_fence_before_sync();
    __syncthreads();
    if (SPLIT > 1) cluster_sync_all();           // no partner signals this CTA's barriers any more
    if (warp == NCW) tmem_dealloc(tmem_base, F_TMEM * BN);
}

template <int BN, int SPLIT>
static int launch_f32(const F32Args& g, cudaStream_t st) {
    auto kern = linear_f32_tc_kernel<BN, SPLIT>;
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, F32Smem<BN>::TOTAL);
        if (e != cudaSuccess) {
            set_error("linear (fp32, tcgen05): cannot reserve %d bytes of shared memory: %s", F32Smem<BN>::TOTAL,
                      cudaGetErrorString(e));
            return (int)e;
        }
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    const long long tiles = (long long)ceil_div(g.N, BN) * ceil_div(g.m_max, FM);
    const int grid = (int)(tiles * SPLIT <= sm_count() ? tiles * SPLIT : sm_count() / SPLIT * SPLIT);
    // every launch starts early: a CTA takes an SM by itself and sets itself up while the kernel in front ends (DeiT-S, 12
    // images: 2449 -> 2374 us with the elected MMA thread; one DeiT-Ti layer, 2 images: 83.2 -> 80.7)
    const cudaError_t le = launch_kernel(kern, true, SPLIT, dim3(grid), dim3(conv_warps(BN) * 32 + 32 + F_EPI),
                                         (size_t)F32Smem<BN>::TOTAL, st, g, device_status_ptr());
    if (le != cudaSuccess) {
        cudaGetLastError();
        set_error("linear (fp32, tcgen05): %s", cudaGetErrorString(le));
        return (int)le;
    }
    return check_launch("linear (fp32, tcgen05)");
}

// 16-byte loads along k: both row pitches a multiple of four floats
bool linear_f32_tc_supported(const LinearArgs& p) {
    return p.dtype == VTP_F32 && p.K % 4 == 0 && p.lda % 4 == 0 && p.ln_mode == 0 && !p.emit_stats;
}

int linear_f32_tcgen05(const LinearArgs& p, cudaStream_t st) {
    if (p.m_max == 0) return VTP_OK;
    F32Args g;
    g.a = (const float*)p.a; g.lda = p.lda; g.w = (const float*)p.w; g.bias = p.bias; g.res = (const float*)p.res;
    g.ldr = p.ldr; g.y = (float*)p.y; g.ldy = p.ldy; g.m_max = p.m_max; g.m_dev = p.m_dev; g.N = p.N; g.K = p.K;
    g.gelu = (p.flags & VTP_FLAG_GELU) ? 1 : 0;
    auto aligned32 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 31u) == 0; };
    g.wide = p.K % 8 == 0 && p.lda % 8 == 0 && aligned32(p.a) && aligned32(p.w);
    g.rm = RowMap{p.out_grp, p.out_skip, p.res_mod, p.res_off};
    g.groups_log2 = f32_groups_log2(ceil_div(p.K, FK));
    // With a device-side row count the worst case is about three times the packed rows of a DGE block.
    const long long sms = sm_count(), likely = p.m_dev ? 3 : 1;
    // 128-wide tiles only where they keep the SMs busy for two rounds
    const long long wide = (long long)ceil_div(p.N, 128) * ceil_div(p.m_max, FM);
    if (wide >= 2 * likely * sms) return launch_f32<128, 1>(g, st);
    // a reduction is split where the tiles leave SMs idle
    const long long tiles = (long long)ceil_div(p.N, 64) * ceil_div(p.m_max, FM);
    if (g.groups_log2 == 2 && tiles * 4 <= likely * sms) return launch_f32<64, 4>(g, st);
    if (g.groups_log2 >= 1 && tiles * 2 <= likely * sms) return launch_f32<64, 2>(g, st);
    return launch_f32<64, 1>(g, st);
}

}  // namespace vtp
