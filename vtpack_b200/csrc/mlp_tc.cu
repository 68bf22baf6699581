// The MLP of a block in one launch (tcgen05, bf16 operands, fp32 accumulate):
//
//   y[m, :] = res[m, :] + GELU(a[m, :] W1^T + b1) W2^T + b2
//
// FOLD: a and res are the same rows and their LayerNorm is folded into W1 (C = 192, 320, 384); else a holds the normalised rows (C = 64, 128).
// The hidden activations, four or eight times as wide as a row, stay on the SM.  A pair of CTAs (cta_group::2, one per SM) takes 256 rows and
// walks their hidden units 128 at a time: fc1 into 128 columns of tensor memory, the GELU from there into shared memory as the A operand of
// fc2, which adds 128 of its K to the accumulators of all C output columns.
//   loaders     (warps 0, 1, 3, one thread each) TMA: the CTA's 128 rows of a, with W1 through a ring; W2 through a ring; res if it is not a
//   MMA         (warp 2, one thread of rank 0) fc1 of the chunks in front, then fc2 of the chunk whose GELU is there.  In rank 1 the warp
//               tells rank 0 of its rows of a
//   epilogue    (16 warps) GELU; then the output, over the rows of res in shared memory, and out by TMA
// A row's sums are formed in the same order as by two Linears (linear_tc.cu): its bits do not depend on which of the two forms runs.
// Every mbarrier wait is bounded (sm100.cuh).
//
// What bounds it: for C = 384 the tensor core, 3080 cycles a chunk (measured 3070 to 3600), and per 256 rows 5 us beside the chunks (first
// operands, the GELU of the first chunk and the output, which nothing overlaps); narrower rows the epilogue, some 2500 cycles a chunk, 1024 of
// them the special-function unit's (tanh).  Two launches / this one, us: figures at mlp_tcgen05_pays.  DeiT-S, 256 images: 3304 -> 3094 us,
// PVT-small, 96 images: 2731 -> 2622.
// What it took (C = 384, one pair running, cycles a chunk):  5500  a box of W (4 MMAs) a stage, eight epilogue warps a chunk;  3900  two boxes
// a stage, and the next stage looked at in front of a stage's MMAs;  3300  two MMAs of 192 columns for fc2 instead of three of 128 (an MMA
// costs its thread about 45 cycles to issue; one of 128 columns takes 64).  Two threads for fc1 and fc2: 3500 to 4800, as their MMAs take
// turns on the tensor core and both end late.  Two groups of epilogue warps gain where nothing else bounds a chunk (C = 64; 254 -> 242
// instead of 246 a block of 96 images), and lose the shared memory of a second H where rings and rows need it.
//
// Replaces Mlp.forward and the residual around it (vtpack/models/dge/deit_dge.py:38-44,128; pvt_dge.py the same).
#include "linear_tc.cuh"

namespace vtp {

using namespace sm100;

struct WaitCtx { volatile int* abort_flag; int* status; };

// A ring of stages, each up to BOXES boxes of W, 64 of K and half of an MMA's columns; for one thread of a CTA that loads, or one of rank 0
// that multiplies.
template <int STAGES, int BOXES, int BOX, bool RESIDENT>
struct WRing {
    uint32_t full, empty, data;         // first barriers, first stage
    uint32_t s = 0, ph = 0, n = 0;      // stage, its phase, stages so far
    bool peeked = false;
    __device__ __forceinline__ WRing(uint32_t full_a, uint32_t empty_a, uint32_t data_a) : full(full_a), empty(empty_a), data(data_a) {}
    __device__ __forceinline__ void next() { ++n; if (++s == STAGES) { s = 0; ph ^= 1; } }
    // `boxes` of them, (dx, dy) apart; of an MMA's rows from y on the second half is the partner's.  Both CTAs' bytes are counted on rank 0's
    // barrier.
    __device__ __forceinline__ bool load(const WaitCtx& c, int rank, const CUtensorMap* m, int x, int y, int boxes, int dx, int dy) {
        if (!mbar_wait_a(empty + 8 * s, ph ^ 1, c.abort_flag, c.status, STATUS_GEMM_PRODUCER)) return false;
        const uint32_t fb = full + 8 * s, lead = mapa_u32(fb, 0), dst = data + s * (BOXES * BOX);
        if (rank == 0) mbar_arrive_expect_tx_a(fb, 2 * BOX * boxes);
        for (int b = 0; b < boxes; ++b) tma_load_2d_a<2>(dst + b * BOX, m, lead, x + b * dx, y + b * dy + rank * (BOX / (TBK * 2)));
        next();
        return true;
    }
    // The last commits arrive in this CTA, for rank 1 from the partner: the loader waits for those of its last fills, so that nothing is
    // signalled into a CTA that has retired.
    __device__ __forceinline__ bool drain(const WaitCtx& c) {
        for (uint32_t d = n > (uint32_t)STAGES ? n - STAGES : 0; d < n; ++d)
            if (!mbar_wait_a(empty + 8 * (d % STAGES), (d / STAGES) & 1, c.abort_flag, c.status, STATUS_GEMM_PRODUCER)) return false;
        return true;
    }
    // The next stage is looked at in front of a stage's MMAs: a wait that is issued behind them returns when the tensor core has taken them.
    __device__ __forceinline__ bool ready(const WaitCtx& c) {
        // (the fence is also for the waits in front: accumulators that have been read, operands; where the weights stay it is all that is left, and a
        // branch of its own: in one with the rest it cost 1.5 % of a block of 96 images, 368 -> 374 us, all rows valid, now 368)
        if (RESIDENT && n >= (uint32_t)STAGES) {
            tc_fence_after_sync();
            return true;
        }
        if (!peeked && !mbar_wait_a(full + 8 * s, ph, c.abort_flag, c.status, STATUS_GEMM_MMA)) return false;
        tc_fence_after_sync();
        const bool wrap = s + 1 == STAGES;
        peeked = mbar_try_wait_a(wrap ? full : full + 8 * (s + 1), wrap ? ph ^ 1 : ph);
        return true;
    }
    // One box against 64 columns of A
    __device__ __forceinline__ void mma(uint32_t d_tmem, uint32_t adesc, int box, uint32_t idesc, bool first) {
        const uint32_t bdesc = (uint32_t)smem_desc_sw128(data + s * (BOXES * BOX) + box * BOX);
        if (first) umma_ss_pair_lo<false>(d_tmem, adesc, bdesc, idesc);
        else umma_ss_pair_lo<true>(d_tmem, adesc, bdesc, idesc);
#pragma unroll
        for (int k = 1; k < TBK / 16; ++k) umma_ss_pair_lo<true>(d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc);
    }
    __device__ __forceinline__ void done() {
        if (!RESIDENT) umma_commit_a<2>(empty + 8 * s);
        next();
    }
};

template <int C>
struct MlpConf {
    static constexpr bool FOLD = C > 128;
    static constexpr int KB = C / TBK;                        // k-blocks of fc1 = 64-column slabs of a row
    static constexpr int CHUNK = 128;                         // hidden units at a time
    static constexpr int PIECES = C > 256 ? 2 : 1, PIECE = C / PIECES;       // columns of an MMA of fc2
    static constexpr bool SPLITS = PIECES == 2 && PIECE % SLAB == 0;         // the last round's rows may be two pairs' (Items)
    static constexpr int GROUPS = C == 64 ? 2 : 1;            // of epilogue warps that take every GROUPS-th chunk, each with its H
    static constexpr int TBUFS = C <= 192 ? 2 : 1;            // accumulators of fc1
    static constexpr bool RESIDENT = C == 64;                 // all of W1 and W2 (512 hidden units) stays in shared memory
    static constexpr int SLAB_A = TBM * TBK * 2;              // one slab of a CTA's rows
    static constexpr int XBUFS = C <= 192 ? 2 : 1;
    static constexpr int H_BYTES = TBM * CHUNK * 2;
    // Rings of boxes of 64 of K and an MMA's columns, half of them in each CTA: two of K a stage (W1), a k-block's (W2)
    static constexpr int BOXES1 = KB > 1 ? 2 : 1, STAGES1 = RESIDENT ? 4 : 3, STAGES2 = RESIDENT ? 8 : C == 128 ? 6 : 4 / PIECES;
    static constexpr int BOX1 = CHUNK / 2 * TBK * 2, BOX2 = PIECE / 2 * TBK * 2;
    static constexpr int EW = 16, FIRST_EPI = 4, THREADS = (FIRST_EPI + EW) * 32;
    static constexpr int SM_R = XBUFS * KB * SLAB_A, SM_H = SM_R + (FOLD ? 0 : KB * SLAB_A), SM_RING1 = SM_H + GROUPS * H_BYTES;
    static constexpr int SM_RING2 = SM_RING1 + STAGES1 * BOXES1 * BOX1, SM_CTRL = SM_RING2 + STAGES2 * PIECES * BOX2;
    static constexpr int CTRL = 512, SM_BIAS = SM_CTRL + CTRL;
    static constexpr int USED = SM_BIAS + C * 4, TOTAL = USED + 1024;
    static constexpr int T_COL = 512 - TBUFS * CHUNK;        // tensor memory: the output in [0, C), fc1 from here on
    static_assert(C % TBK == 0 && PIECE % 16 == 0 && BOX2 % 1024 == 0 && C <= T_COL && TOTAL <= SMEM_MAX, "budgets");
};

struct MlpArgs {
    const float *b1, *s1, *b2;         // fc1's bias and, folded, column sums; fc2's bias
    bf16* y; long long ldy;
    const int32_t* m_dev; int m_max;
    int hidden;
    LnFold ln;
};
struct MlpLaunch { CUtensorMap ta, tr, tw1, tw2, ty; MlpArgs a; };

// What a pair works through: 256 rows at a time, all columns of the output.  Rows of the last, partial round go to two pairs each, one half
// of the columns, where there are as many: both form all of fc1, and half of fc2 each, three quarters of the time (the second round of
// 24,665 rows, C = 384: a block 232 -> 226 us).
template <int C>
struct Items {
    using S = MlpConf<C>;
    int pairs, whole, count;
    bool split;
    __device__ __forceinline__ Items(int M, bool none) {
        const int units = none ? 0 : (M + 2 * TBM - 1) / (2 * TBM);
        pairs = (int)gridDim.x >> 1;
        whole = units / pairs * pairs;
        split = S::SPLITS && 2 * (units - whole) <= pairs;
        if (!split) whole = units;
        count = whole + 2 * (units - whole);
    }
    __device__ __forceinline__ int row0(int it) const { return (S::SPLITS && it >= whole ? whole + ((it - whole) >> 1) : it) * 2 * TBM; }
    __device__ __forceinline__ int piece0(int it) const { return S::SPLITS && it >= whole ? (it - whole) & 1 : 0; }
    __device__ __forceinline__ int pieces(int it) const { return S::SPLITS && it >= whole ? 1 : S::PIECES; }
};

template <int C>
__global__ void __launch_bounds__(MlpConf<C>::THREADS, 1)
mlp_tc_kernel(const __grid_constant__ MlpLaunch L, int* status) {
    using S = MlpConf<C>;
    constexpr int KB = S::KB, STAGES = S::STAGES1 + S::STAGES2, EW = S::EW, XBUFS = S::XBUFS, GROUPS = S::GROUPS, TBUFS = S::TBUFS;
    constexpr bool FOLD = S::FOLD;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* smem_x = base;
    uint8_t* smem_r = FOLD ? base : base + S::SM_R;
    uint8_t* smem_h = base + S::SM_H;
    uint64_t* w_full = reinterpret_cast<uint64_t*>(base + S::SM_CTRL);      // [STAGES] of W1, then of W2; rank 0's
    uint64_t* w_empty = w_full + STAGES;
    uint64_t* x_full = w_empty + STAGES;         // [XBUFS][KB] this CTA's slab of a has landed
    uint64_t* x_peer = x_full + XBUFS * KB;      // rank 0's: the partner's has
    uint64_t* x_empty = x_peer + XBUFS * KB;     // fc1 has read it (FOLD: its columns of the output have left)
    uint64_t* r_full = x_empty + XBUFS * KB;     // [KB] not FOLD: res
    uint64_t* r_empty = r_full + KB;
    uint64_t* t_full = r_empty + KB;             // [TBUFS]
    uint64_t* t_empty = t_full + TBUFS;          // [TBUFS] rank 0's
    uint64_t* h_full = t_empty + TBUFS;          // [GROUPS][2] rank 0's: of each 64 hidden units
    uint64_t* h_empty = h_full + 2 * GROUPS;
    uint64_t* acc_full = h_empty + 2 * GROUPS;
    uint64_t* acc_empty = acc_full + 1;          // rank 0's
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
    static_assert((2 * STAGES + 3 * XBUFS * KB + 2 * KB + 2 * TBUFS + 4 * GROUPS + 2) * 8 + 16 <= S::CTRL, "barrier area");
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* void_s = reinterpret_cast<int*>(tmem_slot + 2);               // [2] launch_is_void in front of the wait and behind it

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank();
    const MlpArgs& P = L.a;
    const int chunks = P.hidden / S::CHUNK;

    bool void_launch = false;
    if (threadIdx.x == S::FIRST_EPI * 32) void_launch = launch_is_void(status);
    if (warp == 0 && elect_one()) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], 1); }
        for (int i = 0; i < XBUFS * KB; ++i) { mbar_init(&x_full[i], 1); mbar_init(&x_peer[i], 1); mbar_init(&x_empty[i], FOLD ? 8 : 1); }
        for (int i = 0; i < KB; ++i) { mbar_init(&r_full[i], 1); mbar_init(&r_empty[i], 8); }
        for (int i = 0; i < TBUFS; ++i) { mbar_init(&t_full[i], 1); mbar_init(&t_empty[i], 2 * EW / GROUPS); }     // a group's warps of both CTAs
        for (int i = 0; i < 2 * GROUPS; ++i) { mbar_init(&h_full[i], EW / GROUPS); mbar_init(&h_empty[i], 1); }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 2 * EW);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&L.ta);
        prefetch_tmap(&L.tw1);
    }
    if (warp == 1 && elect_one()) {
        prefetch_tmap(&L.tw2);
        prefetch_tmap(&L.ty);
        if (!FOLD) prefetch_tmap(&L.tr);
    }
    if (warp == 3) { tmem_alloc_pair(tmem_slot, 512); tmem_relinquish_pair(); }
    if (threadIdx.x == S::FIRST_EPI * 32) void_s[0] = void_launch ? 1 : 0;
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();                  // the partner's barriers exist before anything arrives on them
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const bool known_void = lead_word<2>(void_s) != 0;

    // Everything above is independent of the kernel in front of this one on the stream; from here on its results are read.
    pdl_begin();
    int M = P.m_max;
    if (P.m_dev) M = min(max(*reinterpret_cast<const volatile int32_t*>(P.m_dev), 0), M);
    const Items<C> items(M, known_void);
    const int pair = (int)blockIdx.x >> 1, pairs = items.pairs;
    using Ring1 = WRing<S::STAGES1, S::BOXES1, S::BOX1, S::RESIDENT>;
    using Ring2 = WRing<S::STAGES2, S::PIECES, S::BOX2, S::RESIDENT>;
    const uint32_t ring1 = smem_u32(base + S::SM_RING1), ring2 = smem_u32(base + S::SM_RING2);
    const WaitCtx ctx{abort_flag, status};

    if (warp == 0) {
        if (elect_one()) {
            // ------------------------------------------------------------ loader of a and W1
            Ring1 w(smem_u32(w_full), smem_u32(w_empty), ring1);
            bool ok = true;
            int i = 0;
            for (int it = pair; ok && it < items.count; it += pairs, ++i) {
                const int x0 = i % XBUFS * KB, m0 = items.row0(it) + rank * TBM;
                for (int kb = 0; ok && kb < KB; ++kb) {
                    ok = mbar_wait(&x_empty[x0 + kb], ((i / XBUFS) & 1) ^ 1, abort_flag, status, STATUS_GEMM_PRODUCER);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&x_full[x0 + kb], S::SLAB_A);
                    tma_load_2d(smem_x + (x0 + kb) * S::SLAB_A, &L.ta, &x_full[x0 + kb], kb * TBK, m0);
                    if (kb % 2 == 0 && (!S::RESIDENT || i == 0)) ok = w.load(ctx, rank, &L.tw1, kb * TBK, 0, kb + 1 < KB ? 2 : 1, TBK, 0);
                }
                for (int j = 1; j < chunks && ok && (!S::RESIDENT || i == 0); ++j)
                    for (int kb = 0; kb < KB && ok; kb += 2) ok = w.load(ctx, rank, &L.tw1, kb * TBK, j * S::CHUNK, kb + 1 < KB ? 2 : 1, TBK, 0);
            }
            if (!S::RESIDENT) ok = ok && w.drain(ctx);
            if (!FOLD)                           // (x_empty is a commit's)
                for (int d = i > XBUFS ? i - XBUFS : 0; d < i && ok; ++d)
                    for (int kb = 0; ok && kb < KB; ++kb)
                        ok = mbar_wait(&x_empty[d % XBUFS * KB + kb], (d / XBUFS) & 1, abort_flag, status, STATUS_GEMM_PRODUCER);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            // ------------------------------------------------------------ loader of W2
            Ring2 w(smem_u32(w_full + S::STAGES1), smem_u32(w_empty + S::STAGES1), ring2);
            bool ok = true;
            for (int it = pair; ok && it < items.count && (!S::RESIDENT || it == pair); it += pairs)
                for (int k = 0; k < P.hidden && ok; k += TBK) ok = w.load(ctx, rank, &L.tw2, k, items.piece0(it) * S::PIECE, items.pieces(it), 0, S::PIECE);
            if (!S::RESIDENT && ok) w.drain(ctx);
        }
        __syncwarp();
    } else if (warp == 2) {
        if (rank == 0 && elect_one()) {
            // ------------------------------------------------------------ MMAs of the pair
            // fc1 is TBUFS chunks ahead of fc2: the epilogue takes a chunk out of tensor memory during the fc2 in front.  (Into the next
            // rows where a second buffer holds them.)
            Ring1 w1(smem_u32(w_full), smem_u32(w_empty), ring1);
            Ring2 w2(smem_u32(w_full + S::STAGES1), smem_u32(w_empty + S::STAGES1), ring2);
            constexpr uint32_t idesc1 = idesc_bf16_f32(2 * TBM, S::CHUNK, 0, 0), idesc2 = idesc_bf16_f32(2 * TBM, S::PIECE, 0, 0);
            const uint32_t xdesc = (uint32_t)smem_desc_sw128(smem_u32(smem_x)), hdesc0 = (uint32_t)smem_desc_sw128(smem_u32(smem_h));
            uint32_t g1 = 0, g2 = 0;             // chunks of fc1 and fc2 so far
            int i1 = 0, j1 = 0;                  // the next chunk of fc1, of this pair's i1-th rows
            bool ok = true;
            auto fc1 = [&] {
                const int x0 = i1 % XBUFS * KB;
                const uint32_t tb = g1 % TBUFS, d = tmem_base + S::T_COL + tb * S::CHUNK, a = xdesc + x0 * (S::SLAB_A >> 4);
                ok = mbar_wait(&t_empty[tb], ((g1 / TBUFS) & 1) ^ 1, abort_flag, status, STATUS_GEMM_MMA);
#pragma unroll
                for (int kb = 0; kb < KB; kb += 2) {
                    if (j1 == 0)
                        for (int q = x0 + kb; q < x0 + KB && q < x0 + kb + 2 && ok; ++q)
                            ok = mbar_wait(&x_full[q], (i1 / XBUFS) & 1, abort_flag, status, STATUS_GEMM_MMA) &&
                                 mbar_wait(&x_peer[q], (i1 / XBUFS) & 1, abort_flag, status, STATUS_GEMM_MMA);
                    if (!ok || !(ok = w1.ready(ctx))) return;
                    w1.mma(d, a + kb * (S::SLAB_A >> 4), 0, idesc1, kb == 0);
                    if (kb + 1 < KB) w1.mma(d, a + (kb + 1) * (S::SLAB_A >> 4), 1, idesc1, false);
                    w1.done();
                }
                umma_commit_a<2>(smem_u32(&t_full[tb]));
                ++g1;
                if (++j1 == chunks) {
                    if (!FOLD) for (int kb = 0; kb < KB; ++kb) umma_commit_a<2>(smem_u32(&x_empty[x0 + kb]));
                    j1 = 0;
                    ++i1;
                }
            };
            int i = 0;
            for (int it = pair; ok && it < items.count; it += pairs, ++i) {
                const int pieces = items.pieces(it);
                const bool more = XBUFS == 2 && it + pairs < items.count;
                for (int j = 0; j < chunks && ok; ++j) {
                    while (ok && (i1 == i ? j1 <= j + TBUFS : more && i1 == i + 1 && j1 + chunks <= j + TBUFS)) fc1();
                    if (ok && j == 0) ok = mbar_wait(acc_empty, (i & 1) ^ 1, abort_flag, status, STATUS_GEMM_MMA);
                    const uint32_t hb = g2 % GROUPS, hdesc = hdesc0 + hb * (S::H_BYTES >> 4);
#pragma unroll
                    for (int kb = 0; kb < 2; ++kb) {
                        ok = ok && mbar_wait(&h_full[2 * hb + kb], (g2 / GROUPS) & 1, abort_flag, status, STATUS_GEMM_MMA);
                        if (!ok || !(ok = w2.ready(ctx))) break;
                        const uint32_t a = hdesc + kb * (S::SLAB_A >> 4);
                        w2.mma(tmem_base, a, 0, idesc2, j == 0 && kb == 0);
                        if (S::PIECES == 2 && pieces == 2) w2.mma(tmem_base + S::PIECE, a, 1, idesc2, j == 0 && kb == 0);
                        w2.done();
                        umma_commit_a<2>(smem_u32(&h_empty[2 * hb + kb]));
                    }
                    ++g2;
                }
                if (ok) umma_commit_a<2>(smem_u32(acc_full));
            }
        } else if (rank == 1) {
            if (elect_one()) {
                // ------------------------------------------------------------ rank 0 learns that this CTA's rows of a are there
                bool ok = true;
                int i = 0;
                for (int it = pair; ok && it < items.count; it += pairs, ++i)
                    for (int q = i % XBUFS * KB; ok && q < i % XBUFS * KB + KB; ++q) {
                        ok = mbar_wait(&x_full[q], (i / XBUFS) & 1, abort_flag, status, STATUS_GEMM_PRODUCER);
                        if (ok) mbar_arrive_cluster(mapa_u32(smem_u32(&x_peer[q]), 0));
                    }
            }
        }
        __syncwarp();
    } else if (warp == 3) {
        if (!FOLD) {
            if (elect_one()) {
                // ------------------------------------------------------------ loader of res
                bool ok = true;
                int i = 0;
                for (int it = pair; ok && it < items.count; it += pairs, ++i)
                    for (int kb = 0; ok && kb < KB; ++kb) {
                        ok = mbar_wait(&r_empty[kb], (i & 1) ^ 1, abort_flag, status, STATUS_GEMM_PRODUCER);
                        if (!ok) break;
                        mbar_arrive_expect_tx(&r_full[kb], S::SLAB_A);
                        tma_load_2d(smem_r + kb * S::SLAB_A, &L.tr, &r_full[kb], kb * TBK, items.row0(it) + rank * TBM);
                    }
            }
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------- epilogue
        const int e = warp - S::FIRST_EPI;
        const int quarter = warp & 3, set = e >> 2;          // set: four warps, one of each lane quarter
        const int group = GROUPS == 2 ? set >> 1 : 0;
        // of a chunk a warp takes 32 hidden units, 64 where two groups take turns: of the first 64 (kb = 0) or the others
        constexpr int NC = GROUPS == 2 ? 8 : 4;              // ... as 8-column chunks
        const int kb = GROUPS == 2 ? set & 1 : set >> 1, c0 = GROUPS == 2 ? 0 : (set & 1) * NC;
        const bool leader = elect_one();
        const uint32_t lanes = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        const uint32_t t_empty_a = mapa_u32(smem_u32(t_empty), 0), h_full_a = mapa_u32(smem_u32(h_full), 0), acc_empty_a = mapa_u32(smem_u32(acc_empty), 0);
        auto arrive_lead = [&](uint32_t bar) {               // rank 0's
            __syncwarp();
            if (leader) mbar_arrive_cluster(bar);
        };
        // In a launch that turns out to be void everything changes hands, but this CTA has no rows to store.
        if (threadIdx.x == S::FIRST_EPI * 32) void_s[1] = launch_is_void(status) ? 1 : 0;
        float* bias_s = reinterpret_cast<float*>(base + S::SM_BIAS);      // fc2's
        const uint32_t bias_a = smem_u32(bias_s);
        for (int c = threadIdx.x - S::FIRST_EPI * 32; c < C; c += EW * 32) bias_s[c] = P.b2 ? __ldg(P.b2 + c) : 0.f;
        // fc1's vectors go through the first-level cache, which nothing else here uses: its misses are taken while the first rows travel
        for (int n = (threadIdx.x - S::FIRST_EPI * 32) * 32; n < P.hidden; n += EW * 32 * 32) {
            if (P.b1) asm volatile("prefetch.global.L1 [%0];" ::"l"(P.b1 + n));
            if (FOLD) asm volatile("prefetch.global.L1 [%0];" ::"l"(P.s1 + n));
        }
        named_barrier(1, EW * 32);
        const int rows_valid = void_s[1] == 0 ? M : 0;
        bool ok = true;
        uint32_t g0 = 0;                                     // chunks in front of this pair's current rows
        int i = 0;
        // cells of four 8 x 8 matrices at a time: rows 16 h + 0..7 and + 8..15 of two 16-byte chunks of the warp's 32 x 64
        const uint32_t row_off = (uint32_t)(quarter * 32 + (lane & 15)) * 128u, cx = (uint32_t)(lane & 7);
        float fa[4] = {1.f, 1.f, 1.f, 1.f}, fb[4];           // FOLD: the LayerNorm of rows lane / 4 + 8 k of the warp's
        auto fold_rows = [&](int it) {
            const int m = items.row0(it) + rank * TBM + quarter * 32 + lane;
            float ln_a = 1.f, ln_b = 0.f;
            if (m < M) row_fold(P.ln, m, ln_a, ln_b);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                fa[k] = __shfl_sync(0xffffffffu, ln_a, (lane >> 2) + 8 * k);
                fb[k] = __shfl_sync(0xffffffffu, ln_b, (lane >> 2) + 8 * k);
            }
        };
        if (FOLD && pair < items.count) fold_rows(pair);
        for (int it = pair; ok && it < items.count; it += pairs, ++i, g0 += chunks) {
            const int wrow0 = items.row0(it) + rank * TBM + quarter * 32;       // the warp's first row
            for (int j = GROUPS == 2 ? (int)((group + g0) & 1) : 0; j < chunks; j += GROUPS) {
                const uint32_t g = g0 + j, tb = g % TBUFS, buf = g % GROUPS, ph = (g / GROUPS) & 1;
                const int n0 = j * S::CHUNK + kb * 64 + c0 * 8 + 2 * (lane & 3);
                float2 b1[NC], s1[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    b1[c] = __ldg(reinterpret_cast<const float2*>(P.b1 ? P.b1 + n0 + 8 * c : g_no_bias));
                    if (FOLD) s1[c] = __ldg(reinterpret_cast<const float2*>(P.s1 + n0 + 8 * c));
                }
                ok = mbar_wait_warp(&t_full[tb], (g / TBUFS) & 1, abort_flag, status, STATUS_GEMM_EPILOGUE);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t tacc = lanes + S::T_COL + tb * S::CHUNK + kb * 64 + c0 * 8;
                constexpr int HALVES = GROUPS == 2 ? 1 : 2;        // of the 32 rows in registers at a time
                uint32_t r[HALVES][4 * NC], o[HALVES][2 * NC];
                auto take = [&](int h) {
                    __syncwarp();
                    if constexpr (GROUPS == 1) tmem_ld_16x256b_x4(tacc + (static_cast<uint32_t>(16 * h) << 16), r[h]);
                    else tmem_ld_16x256b_x8(tacc + (static_cast<uint32_t>(16 * h) << 16), r[0]);
                };
                const uint32_t at = smem_u32(smem_h) + buf * S::H_BYTES + kb * S::SLAB_A + row_off;
                if (GROUPS == 1) take(0);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int hh = h % HALVES;
                    if (GROUPS == 2) take(h);
                    if (GROUPS == 2 || h == 0) {
                        if (GROUPS == 1) take(1);
                        tmem_ld_wait();
                        if (GROUPS == 1 || h == 1) {               // fc1 may go on there
                            tc_fence_before_sync();
                            arrive_lead(t_empty_a + 8 * tb);
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 2 * NC; ++q) {             // matrix q: eight columns q / 2, rows lane / 4 + 16 h + 8 (q % 2)
                        const int c = q >> 1, k = 2 * h + (q & 1);
                        float2 v = make_float2(__uint_as_float(r[hh][2 * q]), __uint_as_float(r[hh][2 * q + 1]));
                        if (FOLD) v = fma2(make_float2(fa[k], fa[k]), v, fma2(make_float2(fb[k], fb[k]), s1[c], b1[c]));
                        else v = make_float2(v.x + b1[c].x, v.y + b1[c].y);
                        const uint32_t gl = gelu_pair_f16(v.x, v.y);
                        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&gl));
                        const __nv_bfloat162 t = __floats2bfloat162_rn(f.x, f.y);
                        o[hh][q] = *reinterpret_cast<const uint32_t*>(&t);
                    }
                    if (GROUPS == 1 && h == 0) continue;
                    if (GROUPS == 1 || h == 0) {
                        // fc2 of the chunk in front has read
                        ok = mbar_wait_warp(&h_empty[2 * buf + kb], ph ^ 1, abort_flag, status, STATUS_GEMM_EPILOGUE);
                        if (!ok) break;
                    }
#pragma unroll
                    for (int k = GROUPS == 1 ? 0 : h; k <= h; ++k)
#pragma unroll
                        for (int c = 0; c < NC; c += 2) {
                            const uint32_t* oo = o[k % HALVES];
                            const uint32_t m4[4] = {oo[2 * c], oo[2 * c + 1], oo[2 * c + 2], oo[2 * c + 3]};
                            stmatrix_x4(at + 16 * k * 128u + (((uint32_t)(c0 + c + (lane >> 4)) ^ cx) << 4), m4);
                        }
                }
                if (!ok) break;
                fence_proxy_async_smem();
                arrive_lead(h_full_a + 8 * (2 * buf + kb));
            }
            if (!ok) break;
            // ---- the output: accumulator + bias + res, over the rows of res, 16 rows and 64 columns at a time, and out from there
            if (FOLD && it + pairs < items.count) fold_rows(it + pairs);
            ok = mbar_wait_warp(acc_full, i & 1, abort_flag, status, STATUS_GEMM_EPILOGUE);
            if (!ok) break;
            tc_fence_after_sync();
            const int slab0 = items.piece0(it) * (S::PIECE / SLAB), halves = 2 * (items.pieces(it) == S::PIECES ? KB : S::PIECE / SLAB);
            const int r0 = FOLD ? i % XBUFS * KB : 0;
            uint64_t* landed = FOLD ? x_full : r_full;
            const uint32_t lph = FOLD ? (i / XBUFS) & 1 : i & 1;
#pragma unroll 1
            for (int t = set; t < halves; t += EW / 4) {
                const int slab = slab0 + (t >> 1), n0 = slab * SLAB, h = t & 1;
                uint32_t r[32];
                __syncwarp();
                tmem_ld_16x256b_x8(lanes + (static_cast<uint32_t>(16 * h) << 16) + (n0 - slab0 * SLAB), r);
                ok = mbar_wait_warp(&landed[r0 + slab], lph, abort_flag, status, STATUS_GEMM_EPILOGUE);
                if (!ok) break;
                tmem_ld_wait();
                const uint32_t tile = smem_u32(smem_r) + (r0 + slab) * S::SLAB_A + (quarter * 32 + 16 * h) * 128;
#pragma unroll
                for (int c = 0; c < 8; c += 2) {
                    const uint32_t at = tile + (lane & 15) * 128u + (((uint32_t)(c + (lane >> 4)) ^ cx) << 4);
                    uint32_t rv[4], o[4];
                    ldmatrix_x4(at, rv);
                    float2 b2[2];
#pragma unroll
                    for (int q = 0; q < 2; ++q) b2[q] = lds_f2(bias_a + (n0 + 8 * (c + q) + 2 * (lane & 3)) * 4);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {              // matrix q: chunk c + q / 2, rows + 8 * (q % 2)
                        const int cc = c + (q >> 1);
                        const float2 x2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&rv[q]));
                        const float v0 = (__uint_as_float(r[4 * cc + 2 * (q & 1)]) + b2[q >> 1].x) + x2.x;
                        const float v1 = (__uint_as_float(r[4 * cc + 2 * (q & 1) + 1]) + b2[q >> 1].y) + x2.y;
                        const __nv_bfloat162 t2 = __floats2bfloat162_rn(v0, v1);
                        o[q] = *reinterpret_cast<const uint32_t*>(&t2);
                    }
                    stmatrix_x4(at, o);
                }
                const int m0 = wrow0 + 16 * h;
                if (m0 + 16 <= rows_valid) {
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (leader) {
                        tma_store_2d_a(&L.ty, tile, n0, m0);
                        bulk_commit_group();
                    }
                } else {
                    // rows beyond the last valid one among them: eight lanes copy a row's 128 bytes
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int rr = q * 4 + (lane >> 3);
                        const uint4 v = lds_u4(tile + rr * 128 + (((lane & 7) ^ (rr & 7)) << 4));
                        if (m0 + rr < rows_valid) *reinterpret_cast<uint4*>(P.y + (long long)(m0 + rr) * P.ldy + n0 + 8 * (lane & 7)) = v;
                    }
                    fence_proxy_async_smem();              // (the next rows come by TMA)
                    __syncwarp();
                }
            }
            if (!ok) break;
            tc_fence_before_sync();
            arrive_lead(acc_empty_a);
            if (leader) {
                bulk_wait_group_read0();
                // (slabs that are the other pair's too)
                for (int t = set; t < 2 * KB; t += EW / 4) mbar_arrive(FOLD ? &x_empty[r0 + (t >> 1)] : &r_empty[t >> 1]);
            }
            __syncwarp();
        }
        if (leader) bulk_wait_group0();               // every TMA store has landed before the CTA retires
        __syncwarp();
        // ... and the commits of the last chunks of fc2 have arrived
        if (g0 > 0)
            for (uint32_t g = g0 - GROUPS; g < g0 && ok; ++g)
                for (int kb = 0; kb < 2 && ok; ++kb)
                    ok = mbar_wait_warp(&h_empty[2 * (g % GROUPS) + kb], (g / GROUPS) & 1, abort_flag, status, STATUS_GEMM_EPILOGUE);
    }
    if (*abort_flag) {
        // Unwinding after a wait gave up: give copies still in flight time to land before shared memory and TMEM are released.
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) { }
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();     // the partner no longer reads this CTA's operands or signals its barriers
    if (warp == 3) tmem_dealloc_pair(tmem_base, 512);
}

// ------------------------------------------------------------------------------ host

// fc1 (GELU; from C = 192 on with its LayerNorm folded) and fc2 back onto rows of fc1's width, as one launch.  The widths are those of this
// framework's models: 256 would fit and no model has it; 512 and 768 do not, as the output's columns (512 at most, and fc1's beside them: C <= 384)
// stand in tensor memory.
bool mlp_tcgen05_supported(const LinearArgs& f, const LinearArgs& p) {
    const bool fold = f.K == 192 || f.K == 320 || f.K == 384, rows = f.K == 64 || f.K == 128;
    return f.dtype == VTP_BF16 && p.dtype == VTP_BF16 && f.flags == VTP_FLAG_GELU && p.flags == 0 && p.N == f.K && p.K == f.N &&
           f.N % 256 == 0 && (f.K != 64 || f.N == 512) && ((fold && f.ln_mode == 2 && f.ln_dim == f.K && f.bias && p.res == f.a && p.ldr == f.lda) || (rows && f.ln_mode == 0 && p.res)) &&
           !f.res && !f.emit_stats && p.ln_mode == 0 && !p.emit_stats && p.a == f.y && p.lda == f.ldy && p.m_max == f.m_max && p.m_dev == f.m_dev &&
           f.out_grp == 0 && p.out_grp == 0 && p.res_mod <= 0 && p.y != p.res && p.y != f.a;
}

// From how many rows on (those the host has to allow for; a third to a half of them are valid where a router picks) one launch is shorter
// than two: it takes its time by rounds of 256 rows a pair, 18,944 at a time, however few are valid.  The lines are for a quarter of the regions on the
// finest grain and more (random weights give a quarter, and a budget of half of the operations two fifths); that mixes without any lose up to 5 % of a block
// up to about twice a line, and those with a tenth up to 3 %, is accepted, as only the device knows the mix.  Blocks, us, two launches / one, at a
// tenth / quarter / two fifths / all of the regions on the finest grain (without any: C = 128, 32,768 rows 58/61, C = 192, 20,560 54/56,
// C = 320, 24,576 87/91, 49,152 131/133, C = 384, 32,125 105/110, 49,344 137/139, 65,792 180/176):
//   C = 64    16,384 rows 55/55 56/56 56/56 58/56, 32,768 62/61 65/63 65/62 73/71, 393,216 203/195 241/228 280/264 422/388
//   C = 128   24,576 61/63 63/64 66/65 80/81, 32,768 67/68 70/67 74/70 92/88, 98,304 108/110 124/118 142/133 209/191
//   C = 192   16,448 52/54 55/56 58/57 71/64, 20,560 59/60 62/61 69/66 92/87, 51,400 100/96 106/98 119/115 176/161
//   C = 320   20,480 91/94 97/97 104/100 125/127, 24,576 97/99 102/100 114/106 140/136, 49,152 147/140 158/144 176/171 241/217
//   C = 384   25,700 103/107 117/115 125/118 187/180, 32,125 115/118 130/126 148/137 229/207, 65,792 204/192 233/229 274/252 410/385
bool mlp_tcgen05_pays(const LinearArgs& f) {
    const int least = f.K <= 128 ? 32768 : f.K == 192 ? 20000 : f.K == 320 ? 24000 : 32000;
    return f.m_max >= least;
}

template <int C>
static int launch_mlp(const LinearArgs& f, const LinearArgs& p, cudaStream_t st) {
    using S = MlpConf<C>;
    MlpLaunch L;
    if (int rc = operand_maps(&L.ta, &L.tw1, f, S::CHUNK / 2)) return rc;
    if (int rc = operand_maps(nullptr, &L.tw2, p, S::PIECE / 2)) return rc;
    const unsigned whole[2] = {TBK, TBM}, box[2] = {SLAB, 16};
    const unsigned long long dims[2] = {(unsigned long long)C, (unsigned long long)p.m_max};
    const unsigned long long res_stride[1] = {(unsigned long long)p.ldr * 2ull}, out_stride[1] = {(unsigned long long)p.ldy * 2ull};
    L.tr = L.ta;
    if (!S::FOLD) if (int rc = make_tmap_bf16(&L.tr, p.res, 2, dims, res_stride, whole)) return rc;
    if (int rc = make_tmap_bf16(&L.ty, p.y, 2, dims, out_stride, box)) return rc;
    L.a.b1 = f.bias; L.a.s1 = f.ln_s; L.a.b2 = p.bias;
    L.a.y = (bf16*)p.y; L.a.ldy = p.ldy; L.a.m_dev = p.m_dev; L.a.m_max = p.m_max; L.a.hidden = f.N;
    L.a.ln = LnFold{f.ln_stats, f.ln_s, f.ln_mode, f.ln_dim, f.ln_eps, nullptr, f.ln_slots, ceil_div(f.ln_dim, SLAB)};
    auto kern = mlp_tc_kernel<C>;
    static bool reserved[64] = {};   // per instantiation and device
    if (int rc = reserve_smem(kern, S::TOTAL, reserved)) return rc;
    // (few rows are two pairs' each: Items)
    const int units = ceil_div(p.m_max, 2 * TBM) * (S::SPLITS ? 2 : 1), pairs = sm_count() / 2;
    return launched(launch_kernel(kern, true, 2, dim3(2 * (units < pairs ? units : pairs)), dim3(S::THREADS), (size_t)S::TOTAL, st, L,
                                  device_status_ptr()));
}

int mlp_tcgen05(const LinearArgs& f, const LinearArgs& p, cudaStream_t st) {
    if (f.m_max == 0) return VTP_OK;
    for (const LinearArgs* q : {&f, &p}) {
        if (int rc = linear_validate(*q)) return rc;
        if (int rc = check_tc_args(*q)) return rc;
    }
    VTP_REQUIRE(mlp_tcgen05_supported(f, p), VTP_ERR_UNSUPPORTED, "mlp (tcgen05): these two Linears cannot share a launch");
    if (f.K == 64) return launch_mlp<64>(f, p, st);
    if (f.K == 128) return launch_mlp<128>(f, p, st);
    if (f.K == 192) return launch_mlp<192>(f, p, st);
    if (f.K == 320) return launch_mlp<320>(f, p, st);
    return launch_mlp<384>(f, p, st);
}

}  // namespace vtp
