// fp32 Linear on tcgen05 tensor cores with operands that arrive as terms (f32_terms.cuh), for the blocks of fp32 models.
//
//   y[m, n] = act(sum_k a[m,k] w[n,k] + bias[n]) + res[m, n]
//
// The products and sums are those of linear_f32_tc.cu, in the same order, so a row's bits are the same: six bf16 products of
// terms per k-block of 64, smallest first, a fresh TMEM accumulator for each k-block, k-blocks added in fp32 registers in one,
// two or four groups that K alone decides, sums that come out infinite or NaN worked out again from the decoded operands.
// There every CTA splits the rows it multiplies: a row of the weights once per 128 rows of the batch, a row of the batch once per
// 64 columns, and the splitting bounds it.  Here the kernels that produce the operands leave terms, once, and TMA brings them.
//
// Persistent, one CTA per SM, 128 x BN tiles:
//   warp 0        (one lane) TMA: the three terms of a k-block of a and of w, two stages; a product starts when its own two have
//                 landed
//   warp 1        (one lane) issues the MMAs into one of two TMEM accumulators, one per k-block
//   16 warps      one per TMEM lane quarter and quarter of the columns: add finished accumulators to their registers; after the last
//                 k-block bias / GELU / residual, 64 bytes of a row per store through a per-warp transpose buffer
// A long reduction with few tiles is split over the CTAs of a cluster as in linear_f32_tc.cu.
#include <string.h>

#include "f32_terms.cuh"
#include "linear.h"
#include "linear_f32.cuh"
#include "runtime.h"

namespace vtp {

constexpr int FT_EPI_WARPS = 16, FT_FIRST_EPI = 2, FT_THREADS = (FT_FIRST_EPI + FT_EPI_WARPS) * 32;
constexpr int FT_STAGES = 2;
constexpr int FT_OUT = 32 * 64;          // bytes of a warp's transpose buffer: 32 rows x 16 fp32 columns

template <int BN>
struct FtSmem {
    static constexpr int A_TERM = FM * FK * 2, B_TERM = BN * FK * 2;
    static constexpr int STAGE = 3 * (A_TERM + B_TERM);
    static constexpr int USED = FT_STAGES * STAGE + FT_EPI_WARPS * FT_OUT + 256;
    static constexpr int TOTAL = USED + 1024;                   // the operand tiles want 1024-byte alignment
    static_assert(TOTAL <= 232448, "shared memory budget");
};

struct FtProblem {
    const bf16* a; const bf16* w; const float* bias; const float* res; long long ldr;
    float* y; long long ldy;
    const int32_t* m_dev; int m_max, N;
    FastDiv n_tiles;                     // column tiles of a row of tiles
};
// A launch works through one problem or two independent ones (same K and kind of output): the tiles of the second fill the last, partial
// round of the first (q and kv of DeiT-S, 12 images, 31.6 us in two launches, 22.0 in one).
struct FtArgs {
    FtProblem p[2];
    int K, groups_log2;
    FastDiv step;                        // CTAs (clusters) of the grid
};
// a [m_max][3][K], w [N][3][K] as maps {K, 3, rows} with boxes of 64 elements of one term of a tile's rows; w also in boxes of half
// and of a quarter of a tile's columns.
struct FtMaps { CUtensorMap a, w[3]; };
struct FtMapsOf { FtMaps p[2]; };

// The work items of a CTA (SPLIT of a cluster), in order: tiles first, first + step, ...; where they are cut, the tiles of the
// last, partial round are two or four column strips, one per CTA, so that it takes a fraction of a tile's time.
// (A row's bits do not depend on it: a column's sums are the same in any tile.)
template <int BN, int NPROB>
struct FtItems {
    FastDiv n_tiles[NPROB];
    uint32_t tot0, full, strips, step, first;
    int cut;                                     // log2 of the strips of a tile
    // M: rows of the problems; a void launch that is known has no items
    __device__ __forceinline__ FtItems(const int (&M)[NPROB], bool known_void, const FtArgs& g, uint32_t first_, bool strips_pay) : step(g.step.d), first(first_) {
        uint32_t total = 0;
        tot0 = 0;
#pragma unroll
        for (int i = 0; i < NPROB; ++i) {
            n_tiles[i] = g.p[i].n_tiles;
            if (i == 1) tot0 = total;
            total += (uint32_t)((M[i] + FM - 1) / FM) * n_tiles[i].d;
        }
        if (known_void) total = 0;
        full = !strips_pay ? total : total < step ? 0 : fast_div(total, g.step) * step;
        const uint32_t rest = total - full;
        cut = BN == 128 && rest * 4 <= step ? 2 : rest * 2 <= step ? 1 : 0;
        strips = rest << cut;
    }
    // (a strip beyond the columns of a narrow tile is an item like any other: its sums are not stored)
    struct Item { int p, mt, n0, cut; };         // problem, row of tiles, first column, log2 of BN / columns
    __device__ __forceinline__ bool at(uint32_t j, Item& it) const {
        uint32_t tile = first + j * step, sub = 0;
        it.cut = 0;
        if (tile >= full) {
            const uint32_t u = tile - full;
            if (u >= strips) return false;
            tile = full + (u >> cut);
            sub = u & ((1u << cut) - 1);
            it.cut = cut;
        }
        it.p = NPROB == 2 && tile >= tot0 ? 1 : 0;
        if (NPROB == 2 && it.p) tile -= tot0;
        const FastDiv nt = NPROB == 2 && it.p ? n_tiles[NPROB - 1] : n_tiles[0];
        const uint32_t mt = fast_div(tile, nt);
        it.mt = (int)mt;
        it.n0 = (int)(tile - mt * nt.d) * BN + (int)sub * (BN >> it.cut);
        return true;
    }
};

// Where the terms of a k-block lie: two sets of three slots for a and three for w, which k-blocks take in turn.  Terms are read for
// the last time in the order l, m, h but needed in the order (l, h), (h, l), (m, m): the next k-block of a set takes each slot as
// it falls free, so that its loads are spread over the products of the one before and each is under way for the time of
// eight products or more.
struct FtSlots {
    int a[3] = {0, 1, 2}, b[3] = {0, 1, 2};      // of h, m, l
    // sets[0] becomes the other set's, sets[1] this one's for its next k-block: a's l stays, its h goes where m was, m where h was; w's h
    // goes where l was, its l where m was, m where h was
    static __device__ __forceinline__ void next(FtSlots (&sets)[2]) {
        const FtSlots s = sets[0];
        sets[0] = sets[1];
        sets[1].a[0] = s.a[1]; sets[1].a[1] = s.a[0]; sets[1].a[2] = s.a[2];
        sets[1].b[0] = s.b[2]; sets[1].b[1] = s.b[0]; sets[1].b[2] = s.b[1];
    }
};

// acc: NC columns of row m0 + lane, sums of scaled products, which are scaled back.  Returns the rows of the warp that have a sum that is
// not finite: those are not stored, redo_rows works them out again.
template <int NC>
__device__ __forceinline__ unsigned unscale(float (&acc)[NC], int M, int m0, int lane) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        t = fmaf(acc[i], 0.f, t);              // inf * 0 and NaN * 0 are NaN
        acc[i] *= F_UNSCALE;
    }
    return __ballot_sync(0xffffffffu, t != t && m0 + lane < M);
}

// What the outputs are: + res, as fp32; as terms; GELU, as terms.
constexpr int FT_ROWS = 0, FT_TERMS = 1, FT_HIDDEN = 2;
// Four output columns of row m from column n on, N and n multiples of four.
template <int OUT>
__device__ __forceinline__ void finish4(const FtProblem& g, int m, int n, const float4& s, const float4& bias, const float4& res) {
    float v[4] = {s.x + bias.x, s.y + bias.y, s.z + bias.z, s.w + bias.w};
    if (OUT != FT_ROWS) {
        if (OUT == FT_HIDDEN) {
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = gelu_erf(v[i]);
        }
        store_terms4(reinterpret_cast<bf16*>(g.y) + (size_t)m * 3 * g.N + n, (size_t)g.N, v);
    } else {
        if (g.res) { v[0] += res.x; v[1] += res.y; v[2] += res.z; v[3] += res.w; }
        *reinterpret_cast<float4*>(g.y + (size_t)m * g.ldy + n) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

// Columns n0 .. n0 + cols - 1 of rows m0 + lane, those of `bad`, as fmaf chains over the decoded operands (see linear_f32_tc.cu).  Sixteen
// columns at a time, all rows of the warp at once: an operand that is not finite is a column of the weights or a row of the batch in
// front, and then most rows are bad.  A lane decodes its own row and column lane % 16, the columns go round by shuffles.  (A DeiT-S
// block, 12 images, us: all finite 98, a NaN among the weights of fc2 228; a row at a time, a lane per column, by scalar loads 4500;
// fp32 rows in linear_f32_tc.cu 1700.  Inlined: as a function of its own it cost DeiT-S, 12 images, 11 of 1217 us where all is finite.)
template <int OUT>
__device__ __forceinline__ void redo_rows(const FtProblem& g, int K, int M, int m0, int n0, int cols, unsigned bad, int lane) {
    constexpr int CH = 16;
    const int m = min(m0 + lane, M - 1);
    const bf16* a = g.a + (size_t)m * 3 * K;
#pragma unroll 1
    for (int c0 = 0; c0 < cols; c0 += CH) {
        const bf16* w = g.w + (size_t)min(n0 + c0 + (lane & (CH - 1)), g.N - 1) * 3 * K;
        float s[CH];
#pragma unroll
        for (int c = 0; c < CH; ++c) s[c] = 0.f;
#pragma unroll 1
        for (int k = 0; k < K; k += 8) {
            float x[8], y[8];
            join8(a + k, (size_t)K, x);
            join8(w + k, (size_t)K, y);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int c = 0; c < CH; ++c) s[c] = fmaf(x[i], __shfl_sync(0xffffffffu, y[i], c), s[c]);
        }
        if (!(bad >> lane & 1)) continue;
#pragma unroll
        for (int c = 0; c < CH; c += 4) {
            const int n = n0 + c0 + c;
            if (c0 + c >= cols || n >= g.N) continue;
            const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
            finish4<OUT>(g, m, n, make_float4(s[c], s[c + 1], s[c + 2], s[c + 3]),
                         g.bias ? __ldg(reinterpret_cast<const float4*>(g.bias + n)) : zero4,
                         OUT == FT_ROWS && g.res ? *reinterpret_cast<const float4*>(g.res + (size_t)m * g.ldr + n) : zero4);
        }
    }
}

// SPLIT: CTAs of a cluster that share a tile's reduction (1: none); it divides the number of groups.
template <int BN, int SPLIT, int OUT, int NPROB>
__global__ void __launch_bounds__(FT_THREADS, 1)
linear_f32_terms_kernel(const __grid_constant__ FtMapsOf maps, const __grid_constant__ FtArgs g, int* status) {
    using S = FtSmem<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + FT_STAGES * S::STAGE + FT_EPI_WARPS * FT_OUT);
    uint64_t* full = bars;                        // [2][3] per set of slots: the terms of the first product have landed, those of the
                                                  //     second, the other two (FtSlots)
    uint64_t* empty = bars + 6;                   // [2][3] the slots that these go to have been read
    uint64_t* acc_full = bars + 12;               // [2]
    uint64_t* acc_empty = bars + 14;              // [2]
    uint64_t* part_full = bars + 16;              // the other CTAs' partial sums of this CTA's columns have arrived
    uint64_t* part_free = bars + 17;              // the other CTAs have added the ones this CTA sent them
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* void_s = reinterpret_cast<int*>(tmem_slot + 2);   // [2] launch_is_void in front of the wait and behind it
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 6; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], FT_EPI_WARPS);
        }
        mbar_init(part_full, 1);
        mbar_init(part_free, SPLIT > 1 ? (SPLIT - 1) * FT_EPI_WARPS : 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, F_TMEM * BN);
        tmem_relinquish();
    }
    if (warp == FT_FIRST_EPI && elect_one()) {
        for (int p = 0; p < NPROB; ++p) {
            prefetch_tmap(&maps.p[p].a);
            for (int i = 0; i < 3; ++i) prefetch_tmap(&maps.p[p].w[i]);
        }
    }
    // (parameters are cold in every launch, each line of them is a miss: not on the way to the first load)
    if (warp == FT_FIRST_EPI + 2)
        for (int i = lane; i < (int)(sizeof(FtArgs) / 4); i += 32) asm volatile("" ::"r"(reinterpret_cast<const uint32_t*>(&g)[i]));
    if (threadIdx.x == (FT_FIRST_EPI + 1) * 32) void_s[0] = launch_is_void(status) ? 1 : 0;
    tc_fence_before_sync();
    __syncthreads();
    if (SPLIT > 1) cluster_sync_all();            // the partners' barriers exist
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const bool known_void = lead_word<SPLIT>(void_s) != 0;
    pdl_begin();

    int rows[NPROB];
#pragma unroll
    for (int i = 0; i < NPROB; ++i) {
        rows[i] = g.p[i].m_max;
        if (g.p[i].m_dev) rows[i] = min(max(*reinterpret_cast<const volatile int32_t*>(g.p[i].m_dev), 0), rows[i]);
    }
    const int rank = SPLIT > 1 ? (int)cluster_ctarank() : 0;
    const int all_kb = (g.K + FK - 1) / FK;
    const int kb0 = all_kb * rank / SPLIT, num_kb = all_kb * (rank + 1) / SPLIT - kb0;    // this CTA's k-blocks
    const FtItems<BN, NPROB> items(rows, known_void, g, blockIdx.x / SPLIT, SPLIT == 1);
    // (term of a, term of w) of the products, smallest first; the first three bring every term once
    constexpr int TA[6] = {2, 0, 1, 1, 0, 0}, TB[6] = {0, 2, 1, 0, 1, 0};
    FtSlots sets[2];
    typename FtItems<BN, NPROB>::Item wi;
    int it = 0;                                   // k-blocks so far
    bool ok = true;

    if (warp == 0) {
        if (elect_one()) {
            // ------------------------------------------------------------ TMA producer
            const uint32_t sbase = smem_u32(base);
            for (uint32_t j = 0; ok && items.at(j, wi); ++j) {
                const FtMaps& mp = maps.p[NPROB == 2 ? wi.p : 0];
                const CUtensorMap* wmap = &mp.w[wi.cut];
                const uint32_t b_term = S::B_TERM >> wi.cut;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it & 1;
                    const FtSlots& in = sets[0];
                    const uint32_t sa = sbase + s * S::STAGE, sb = sa + 3 * S::A_TERM;
                    const int k = (kb0 + kb) * FK;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        ok = mbar_wait(&empty[3 * s + c], ((it >> 1) & 1) ^ 1, abort_flag, status, STATUS_GEMM_PRODUCER);
                        if (!ok) break;
                        const uint32_t bar = smem_u32(&full[3 * s + c]);
                        mbar_arrive_expect_tx_a(bar, S::A_TERM + b_term);
                        tma_load_3d_a(sa + in.a[TA[c]] * S::A_TERM, &mp.a, bar, k, TA[c], wi.mt * FM);
                        tma_load_3d_a(sb + in.b[TB[c]] * S::B_TERM, wmap, bar, k, TB[c], wi.n0);
                    }
                    if (!ok) break;
                    FtSlots::next(sets);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            // -------------------------------------------------------------- MMA issuer
            const uint32_t sbase = smem_u32(base);
            for (uint32_t j = 0; ok && items.at(j, wi); ++j) {
                const uint32_t idesc = idesc_bf16_f32(FM, BN >> wi.cut, 0, 0);
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it & 1;
                    const uint32_t ph = (it >> 1) & 1;
                    ok = mbar_wait(&acc_empty[s], ph ^ 1, abort_flag, status, STATUS_GEMM_MMA);
                    if (!ok) break;
                    const FtSlots& in = sets[0];
                    const uint32_t sa = sbase + s * S::STAGE, sb = sa + 3 * S::A_TERM;
#pragma unroll
                    for (int c = 0; c < 6; ++c) {
                        if (c < 3) {
                            ok = mbar_wait(&full[3 * s + c], ph, abort_flag, status, STATUS_GEMM_MMA);
                            if (!ok) break;
                            tc_fence_after_sync();
                        }
                        const uint64_t ad = smem_desc_sw128(sa + in.a[TA[c]] * S::A_TERM);
                        const uint64_t bd = smem_desc_sw128(sb + in.b[TB[c]] * S::B_TERM);
#pragma unroll
                        for (int k = 0; k < FK / 16; ++k)
                            umma_ss(tmem_base + s * BN, ad + 2 * k, bd + 2 * k, idesc, (c | k) != 0 ? 1u : 0u);
                        // l of both has been read; m of both; h
                        if (c == 1 || c >= 4) umma_commit(&empty[3 * s + (c == 1 ? 0 : c - 3)]);
                    }
                    if (!ok) break;
                    umma_commit(&acc_full[s]);
                    FtSlots::next(sets);
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------- epilogue
        constexpr int CW = BN / 4;                       // columns of a warp
        const int ew = warp - FT_FIRST_EPI;
        const int quarter = warp & 3;                    // TMEM lane quarter this warp may read
        const int col = (ew >> 2) * CW;                  // its first column of an item
        const uint32_t tacc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + col;
        const uint32_t stage = smem_u32(base + FT_STAGES * S::STAGE) + ew * FT_OUT;
        const int own_groups = (1 << g.groups_log2) / SPLIT;         // this CTA's: 1, 2 or 4
        const uint32_t tsum = tacc + 2 * BN;             // sums of its earlier groups: 0 (+ 1), and 2
        const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
        // in a launch that turns out to be void the sums still change hands, but this CTA has no rows to store
        if (threadIdx.x == FT_FIRST_EPI * 32) void_s[1] = launch_is_void(status) ? 1 : 0;
        named_barrier(1, FT_EPI_WARPS * 32);
        const bool stores = void_s[1] == 0;
        int n_sent = 0;                                   // exchanges
        for (uint32_t j = 0; ok && items.at(j, wi); ++j) {
            const FtProblem& q = g.p[NPROB == 2 ? wi.p : 0];
            const int M = !stores ? 0 : NPROB == 2 && wi.p ? rows[NPROB - 1] : rows[0];
            const int m0 = wi.mt * FM + quarter * 32, n0 = wi.n0 + col;
            const bool has = col < (BN >> wi.cut);        // a strip leaves some warps without columns
            // What an output needs besides its sum travels while the operands are loaded and multiplied.  SPLIT: SC columns of row
            // `lane`, else of every sixteen columns four of rows lane / 4 + 8 q.
            constexpr int SC = CW / SPLIT;
            constexpr int NV = SPLIT > 1 ? SC / 4 : CW / 4;
            float4 res[OUT != FT_ROWS ? 1 : NV], bias[SPLIT > 1 ? NV : CW / 16];
            auto col_of = [&](int v) { return SPLIT > 1 ? n0 + rank * SC + 4 * v : n0 + (v >> 2) * 16 + (lane & 3) * 4; };
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const int m = SPLIT > 1 ? m0 + lane : m0 + (v & 3) * 8 + (lane >> 2), n = col_of(v);
                if (OUT == FT_ROWS) res[v] = q.res && has && m < M && n < q.N ? *reinterpret_cast<const float4*>(q.res + (size_t)m * q.ldr + n) : zero4;
                if (SPLIT > 1 || (v & 3) == 0)
                    bias[SPLIT > 1 ? v : v >> 2] = q.bias && has && n < q.N ? __ldg(reinterpret_cast<const float4*>(q.bias + n)) : zero4;
            }
            float acc[CW];
#pragma unroll
            for (int i = 0; i < CW; ++i) acc[i] = 0.f;
            int grp = 0;
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                const int s = it & 1;
                ok = mbar_wait_warp(&acc_full[s], (it >> 1) & 1, abort_flag, status, STATUS_GEMM_EPILOGUE);
                if (!ok) break;
                tc_fence_after_sync();
                if (has) stash_add<CW, 16>(tacc + s * BN, acc);
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[s]);
                if constexpr (SPLIT < 4) {
                    // the CTA has one group, or this k-block does not end one
                    if (own_groups == 1 || kb + 1 != (all_kb * (rank * own_groups + grp + 1) >> g.groups_log2) - kb0) continue;
                    if (grp & 1) stash_add<CW, 16>(tsum + (SPLIT == 1 ? (grp >> 1) * BN : 0), acc);
                    if (SPLIT == 1 && grp == 3) stash_add<CW, 16>(tsum, acc);            // (0 + 1) + (2 + 3)
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
                constexpr int ROUNDS = (SPLIT - 1) * SC * 128 > FT_OUT ? 2 : 1, XC = SC / ROUNDS;     // what the slots hold
                static_assert((SPLIT - 1) * XC * 128 <= FT_OUT && XC % 4 == 0, "the exchange fits the warp's transpose buffer");
                float own[SC];
                typename FtItems<BN, NPROB>::Item next;
#pragma unroll
                for (int d = 0; d < SPLIT; ++d)                   // (a runtime index would put acc into local memory)
                    if (d == rank) {
#pragma unroll
                        for (int i = 0; i < SC; ++i) own[i] = acc[d * SC + i];
                    }
#pragma unroll
                for (int x = 0; x < ROUNDS; ++x, ++n_sent) {
                    if (n_sent > 0) ok = mbar_wait_cluster_warp(part_free, (n_sent - 1) & 1, abort_flag, status, STATUS_GEMM_EPILOGUE);
                    if (!ok) break;
#pragma unroll
                    for (int d = 0; d < SPLIT; ++d) {
                        if (d == rank) continue;
                        const uint32_t dst = mapa_u32(stage, d) + (rank < d ? rank : rank - 1) * (XC * 128) + lane * 16;
                        const uint32_t bar = mapa_u32(smem_u32(part_full), d);
#pragma unroll
                        for (int i = 0; i < XC / 4; ++i) {
                            const int c = d * SC + x * XC + 4 * i;
                            stc_async_f4(dst + i * 512, make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]), bar);
                        }
                    }
                    // (bytes may arrive before they are expected: the phase also waits for this arrival)
                    if (threadIdx.x == FT_FIRST_EPI * 32) mbar_arrive_expect_tx(part_full, (SPLIT - 1) * FT_EPI_WARPS * XC * 128);
                    ok = mbar_wait_cluster_warp(part_full, n_sent & 1, abort_flag, status, STATUS_GEMM_EPILOGUE);
                    if (!ok) break;
                    // four partial sums: this CTA's pair first, then the other pair's sum (slots are in source order without
                    // this CTA: 1 2 3, 0 2 3, 0 1 3, 0 1 2)
                    const uint32_t mine = stage + lane * 16 + (SPLIT == 4 && rank >= 2 ? 2 : 0) * (XC * 128);
                    const uint32_t other = stage + lane * 16 + (rank >= 2 ? 0 : 1) * (XC * 128);
#pragma unroll
                    for (int i = 0; i < XC / 4; ++i) {
                        float* o = own + x * XC + 4 * i;
                        const float4 p = lds_f4(mine + i * 512);
                        o[0] += p.x; o[1] += p.y; o[2] += p.z; o[3] += p.w;
                        if constexpr (SPLIT == 4) {
                            const float4 c = lds_f4(other + i * 512), d = lds_f4(other + XC * 128 + i * 512);
                            o[0] += c.x + d.x; o[1] += c.y + d.y; o[2] += c.z + d.z; o[3] += c.w + d.w;
                        }
                    }
                    // (nothing follows the last exchange of the last item)
                    __syncwarp();
                    if (lane == 0 && (x + 1 < ROUNDS || items.at(j + 1, next))) {
#pragma unroll
                        for (int d = 0; d < SPLIT; ++d)
                            if (d != rank) mbar_arrive_release_cluster(mapa_u32(smem_u32(part_free), d));
                    }
                }
                if (!ok) break;
                const unsigned bad = unscale<SC>(own, M, m0, lane);
                if (m0 + lane < M && !(bad >> lane & 1)) {
#pragma unroll
                    for (int v = 0; v < NV; ++v)
                        if (col_of(v) < q.N)
                            finish4<OUT>(q, m0 + lane, col_of(v), make_float4(own[4 * v], own[4 * v + 1], own[4 * v + 2], own[4 * v + 3]),
                                            bias[v], res[OUT != FT_ROWS ? 0 : v]);
                }
                if (bad) redo_rows<OUT>(q, g.K, M, m0, n0 + rank * SC, SC, bad, lane);
            } else if (has) {
                const unsigned bad = unscale<CW>(acc, M, m0, lane);
                // 16 columns at a time through the warp's transpose buffer (rows of four 16-byte chunks, XOR-swizzled): a lane
                // then holds four columns of a row and four lanes 64 consecutive bytes
#pragma unroll
                for (int b = 0; b < CW / 16; ++b) {
                    __syncwarp();                             // the previous block has been read
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        sts_u4(stage + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4),
                               make_uint4(__float_as_uint(acc[16 * b + 4 * i]), __float_as_uint(acc[16 * b + 4 * i + 1]),
                                          __float_as_uint(acc[16 * b + 4 * i + 2]), __float_as_uint(acc[16 * b + 4 * i + 3])));
                    __syncwarp();
                    const int n = n0 + 16 * b + (lane & 3) * 4;
                    auto finish = [&](int r8) {
                        const int rr = r8 * 8 + (lane >> 2);
                        const float4 v = lds_f4(stage + rr * 64 + (((lane & 3) ^ ((rr >> 1) & 3)) << 4));
                        if (m0 + rr < M && n < q.N && !(bad >> rr & 1)) finish4<OUT>(q, m0 + rr, n, v, bias[b], res[OUT != FT_ROWS ? 0 : 4 * b + r8]);
                    };
                    if constexpr (OUT == FT_HIDDEN) {
                        // (not unrolled: most launches run this once per warp, and then what it costs is its fetch)
#pragma unroll 1
                        for (int r8 = 0; r8 < 4; ++r8) finish(r8);
                    } else {
#pragma unroll
                        for (int r8 = 0; r8 < 4; ++r8) finish(r8);
                    }
                }
                // (behind the stores, where there are no outputs to keep beside it)
                if (bad) redo_rows<OUT>(q, g.K, M, m0, n0, CW, bad, lane);
            }
        }
    }
    if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) { }     // let copies and MMAs in flight finish before releasing memory
    }
    tc_fence_before_sync();
    __syncthreads();
    if (SPLIT > 1) cluster_sync_all();           // no partner signals this CTA's barriers any more
    if (warp == 1) tmem_dealloc(tmem_base, F_TMEM * BN);
}

template <int BN, int SPLIT, int OUT, int NPROB>
static int launch_terms(FtArgs& g, const FtMapsOf& maps, cudaStream_t st) {
    auto kern = linear_f32_terms_kernel<BN, SPLIT, OUT, NPROB>;
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FtSmem<BN>::TOTAL);
        if (e != cudaSuccess) {
            set_error("linear (fp32 terms): cannot reserve %d bytes of shared memory: %s", FtSmem<BN>::TOTAL, cudaGetErrorString(e));
            return (int)e;
        }
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    long long tiles = 0;
    for (int i = 0; i < NPROB; ++i) {
        g.p[i].n_tiles = make_fast_div((uint32_t)ceil_div(g.p[i].N, BN));
        tiles += (long long)ceil_div(g.p[i].N, BN) * ceil_div(g.p[i].m_max, FM);
    }
    if (SPLIT == 1) tiles *= BN / 32;                        // few tiles are cut into strips (FtItems): a CTA for each
    const int grid = (int)(tiles * SPLIT <= sm_count() ? tiles * SPLIT : sm_count() / SPLIT * SPLIT);
    g.step = make_fast_div((uint32_t)(grid / SPLIT));
    const cudaError_t le = launch_kernel(kern, true, SPLIT, dim3(grid), dim3(FT_THREADS), (size_t)FtSmem<BN>::TOTAL, st, maps, g,
                                         device_status_ptr());
    if (le != cudaSuccess) {
        cudaGetLastError();
        set_error("linear (fp32 terms): %s", cudaGetErrorString(le));
        return (int)le;
    }
    return check_launch("linear (fp32 terms)");
}

// What a launch of this tile width and split takes, in cycles: rounds of tiles, the k-blocks of each, a tile's end (GELU and the
// exchange of a split among it; clusters of four do not fill the chip).  Fitted to the launches below (us; * what it picks):
//                                        64 / 1    64 / 2    64 / 4   128 / 1   128 / 2   128 / 4
//   3084 x 768, K = 384                    21.0      24.5               19.0*     25.4
//   1100 x 384, K = 384                     9.5       8.3*              10.6      11.4
//   1100 x 1536, K = 384, GELU             18.4      22.0               16.3*     26.3
//   1100 x 384, K = 1536, residual         26.6      18.1      21.5     27.6      23.0      15.7*
//   771 x 1536, K = 768                    26.8      25.4      43.8     21.0*     25.2      37.9
//   270 x 768, K = 768, residual           15.0      11.4*     14.8     16.3      15.7      11.4
//   270 x 768, K = 3072, residual          48.2      29.1      32.3     49.4      36.4      22.3*
//   180 x 192, K = 768, residual           14.0      10.7       7.4*    15.4      15.0      10.5
//   4400 x 768, K = 192, GELU              18.0                         17.4*
// (tiles: of a launch without splits, 128 rows x bn columns, the second problem's included)
static double terms_cost(int bn, int split, bool hidden, long long tiles, int num_kb, int sms) {
    const bool wide = bn == 128;
    const double kb_cost = wide ? 2050 : 1640;
    const double end = (split == 1 ? (wide ? 3000 : 1500) : split == 2 ? (wide ? 5000 : 2500) : (wide ? 7500 : 3000)) +
                       (hidden ? (wide ? 6000 : 3500) : 0);
    const long long lanes = split == 4 ? sms * 9 / 40 : sms / split;
    const long long full = tiles / lanes, rest = tiles - full * lanes;
    double rounds = (double)full;
    if (rest) rounds += split > 1 ? 1.0 : (wide && rest * 4 <= lanes) ? 0.65 : rest * 2 <= lanes ? 0.8 : 1.0;
    return rounds * (ceil_div(num_kb, split) * kb_cost + end);
}

static int fill_terms(FtProblem& q, FtMaps& maps, const LinearArgs& p, int bn) {
    q.a = (const bf16*)p.a; q.w = (const bf16*)p.w; q.bias = p.bias; q.res = (const float*)p.res; q.ldr = p.ldr;
    q.y = (float*)p.y; q.ldy = p.ldy; q.m_max = p.m_max; q.m_dev = p.m_dev; q.N = p.N;
    const unsigned long long strides[2] = {(unsigned long long)p.K * 2, (unsigned long long)p.K * 6};
    const unsigned long long da[3] = {(unsigned long long)p.K, 3, (unsigned long long)p.m_max};
    const unsigned long long dw[3] = {(unsigned long long)p.K, 3, (unsigned long long)p.N};
    const unsigned ba[3] = {FK, 1, FM};
    if (int rc = make_tmap_bf16(&maps.a, p.a, 3, da, strides, ba)) return rc;
    for (int i = 0; i < 3; ++i) {
        const unsigned bw[3] = {FK, 1, (unsigned)(bn >> (bn == 128 ? i : i > 0))};      // (64-wide tiles are cut in two only)
        if (int rc = make_tmap_bf16(&maps.w[i], p.w, 3, dw, strides, bw)) return rc;
    }
    return VTP_OK;
}

// p1: null, or a second problem (split 1 only).
static int linear_f32_terms_as(const LinearArgs& p, const LinearArgs* p1, int bn, int split, cudaStream_t st) {
    FtArgs g;
    FtMapsOf maps;
    g.K = p.K;
    g.groups_log2 = f32_groups_log2(ceil_div(p.K, FK));
    if (int rc = fill_terms(g.p[0], maps.p[0], p, bn)) return rc;
    if (p1) {
        if (int rc = fill_terms(g.p[1], maps.p[1], *p1, bn)) return rc;
        if (bn == 128) return p.out_terms ? launch_terms<128, 1, FT_TERMS, 2>(g, maps, st) : launch_terms<128, 1, FT_ROWS, 2>(g, maps, st);
        return p.out_terms ? launch_terms<64, 1, FT_TERMS, 2>(g, maps, st) : launch_terms<64, 1, FT_ROWS, 2>(g, maps, st);
    }
    g.p[1] = g.p[0];
    maps.p[1] = maps.p[0];
#define VTP_TERMS_CASE(BN, SPLIT) \
    if (bn == BN && split == SPLIT) return !p.out_terms ? launch_terms<BN, SPLIT, FT_ROWS, 1>(g, maps, st) \
                                             : (p.flags & VTP_FLAG_GELU) ? launch_terms<BN, SPLIT, FT_HIDDEN, 1>(g, maps, st) \
                                                                         : launch_terms<BN, SPLIT, FT_TERMS, 1>(g, maps, st)
    VTP_TERMS_CASE(128, 1);
    VTP_TERMS_CASE(128, 2);
    VTP_TERMS_CASE(128, 4);
    VTP_TERMS_CASE(64, 1);
    VTP_TERMS_CASE(64, 2);
    VTP_TERMS_CASE(64, 4);
#undef VTP_TERMS_CASE
    return fail(VTP_ERR_UNSUPPORTED, "linear (fp32 terms): no kernel for tiles of %d columns, %d CTAs", bn, split);
}

static int check_terms(const LinearArgs& p) {
    if (int rc = linear_validate(p)) return rc;
    VTP_REQUIRE(p.dtype == VTP_F32 && p.N % 8 == 0 && p.K % 8 == 0 && p.ldy % 4 == 0 && (!p.res || p.ldr % 4 == 0), VTP_ERR_SHAPE,
                "linear (fp32 terms): N=%d K=%d", p.N, p.K);
    VTP_REQUIRE(p.ln_mode == 0 && !p.emit_stats && p.out_grp == 0 && p.res_mod == 0 && (p.out_terms || !(p.flags & VTP_FLAG_GELU)) &&
                    !(p.out_terms && p.res), VTP_ERR_UNSUPPORTED,
                "linear (fp32 terms): plain rows; GELU only with terms out, a residual only with fp32 out");
    return VTP_OK;
}

// Of rows that are counted on the device a third: about 5.5 queries of 16 tokens with untrained routers.  Unlike the bf16 launch of one tile
// per CTA (small_tiles) this kernel goes on with the next tile where there are more.
static long long likely_tiles(const LinearArgs& p, int bn) {
    return (long long)ceil_div(p.m_dev ? ceil_div(p.m_max, 3) : p.m_max, FM) * ceil_div(p.N, bn);
}
static double best_terms(const LinearArgs& p, int* bn, int* split) {
    const int num_kb = ceil_div(p.K, FK), sms = sm_count();
    double best = 0;
    for (int b = 64; b <= 128; b *= 2)
        for (int s = 1; s <= (1 << f32_groups_log2(num_kb)); s *= 2) {
            const double c = terms_cost(b, s, (p.flags & VTP_FLAG_GELU) != 0, likely_tiles(p, b), num_kb, sms);
            if (best == 0 || c < best) { best = c; *bn = b; *split = s; }
        }
    return best;
}

int linear_f32_terms(const LinearArgs& p, cudaStream_t st) {
    if (int rc = check_terms(p)) return rc;
    if (p.m_max == 0) return VTP_OK;
    int bn = 64, split = 1;
    best_terms(p, &bn, &split);
    return linear_f32_terms_as(p, nullptr, bn, split, st);
}

// Two problems that do not depend on each other, with the same K and kind of output: in one launch where that looks the shorter (a launch
// costs some 4000 cycles beside its tiles; one of both splits no reduction).  Blocks, us, at a third / two thirds / all of the
// regions on the finest grain, with this rule and apart: DeiT-S, 1 image 64.5 65.4 67.0 and 73.8 75.5 76.4; 12 images 98.4 127 178 and
// 107 141 192; 64 images 280 413 531 and 277 413 533; DeiT-B, 1 image 103 116 133 and 107 119 144; 24 images 373 509 598 and 369 511 598;
// PVT stage 1, 8 images 106 135 154 and 109 139 157; stage 3, 64 images 222 309 392 and 225 317 396.
int linear_f32_terms_pair(const LinearArgs& a, const LinearArgs& b, cudaStream_t st) {
    if (int rc = check_terms(a)) return rc;
    if (int rc = check_terms(b)) return rc;
    const int num_kb = ceil_div(a.K, FK), sms = sm_count();
    int bn = 64, split = 1;
    const double apart = best_terms(a, &bn, &split) + best_terms(b, &bn, &split) + 4000;
    double together = 0;
    for (int w = 64; w <= 128; w *= 2) {
        const double c = terms_cost(w, 1, false, likely_tiles(a, w) + likely_tiles(b, w), num_kb, sms);
        if (together == 0 || c < together) { together = c; bn = w; }
    }
    const bool fit = a.K == b.K && a.out_terms == b.out_terms && !((a.flags | b.flags) & VTP_FLAG_GELU) && a.m_max > 0 && b.m_max > 0;
    if (fit && together < apart) return linear_f32_terms_as(a, &b, bn, 1, st);
    if (int rc = linear_f32_terms(a, st)) return rc;
    return linear_f32_terms(b, st);
}

}  // namespace vtp
