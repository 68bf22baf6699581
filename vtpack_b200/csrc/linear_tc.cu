// Linear layer on 5th-generation tensor cores (tcgen05), bf16 operands, fp32 accumulate in
// tensor memory, operands staged by TMA with a 128-byte swizzle.
//
//   y[m, n] = act(sum_k a[m,k] w[n,k] + bias[n]) + res[m, n]
//
// linear_tc_kernel is persistent and warp-specialised: one CTA per SM, alone or in pairs (cta_group::2), walks 128 x BN or
// 256 x BN output tiles (n fastest, so the CTAs running at the same time share an A row tile in L2).
//   producer warps  (one lane each) TMA: fill a ring of {A 128x64, W BNx64} k-blocks in turn; the ring runs across tile
//                   boundaries, so the next tile's operands stream in during the current tile's epilogue
//   MMA warp        (one lane) issues tcgen05.mma (K = 16 at a time) into one of two TMEM accumulators and commits each stage
//                   back to the producers
//   epilogue warps  one per TMEM lane quarter (the 32 rows it may read) and 64-column slab of the tile: tcgen05.ld, bias /
//                   LayerNorm fold / GELU / residual, then through a 4 KB staging buffer of the warp's own (full 128-byte lines)
//                   to its own TMA store.  No warp waits for another one's part of the tile.  Warps with rows beyond the last
//                   valid one and row-remapped outputs copy the buffer out themselves; fp32 outputs go straight from registers.
// The two accumulators let the MMA of tile i+1 overlap the epilogue of tile i.
// The tiles left for the last, partial round of the grid are cut into two to four column strips
// (their own W boxes, a narrower MMA), one per CTA, so that round costs a fraction of a tile.
// The number of valid rows is read from device memory: tiles beyond it do not exist, rows
// beyond it are never stored.
// linear_tc_small_kernel and linear_tc_pair_kernel (below) are the forms for problems of few tiles.
//
// What bounds it, and what was measured (B200, launches replayed back to back in a graph, us; the kernel before: one CTA per
// tile, staging slabs shared by all epilogue warps, a store thread):
//                                                         before   now   cuBLAS (no epilogue)
//   65792 x 768, K = 384 (DeiT-S kv, 256 images)           43.3   41.2   39.1    HBM and L2 writes: without stores 29.8
//   23040 x 1536, K = 384, GELU (fc1)                      34.0   29.8   28.6    epilogue and writes
//   23040 x 384, K = 1536, residual (fc2)                  39.0   30.8   25.5    2.4 rounds of tiles, their tail
//   8481 x 1536, K = 768 (DeiT-B kv, 33 images)            24.6   21.7   18.1    2.8 rounds, start (4 us) and tail
//   2970 x 768, K = 3072, residual (DeiT-B fc2)            21.0   17.5   13.9    one round
//   172000 x 512, K = 64, GELU (PVT stage 1 fc1)           63.4   42.5   36.2    epilogue instructions, HBM (floor 31)
//   393216 x 64, K = 64                                    28.3   19.5   18.0    HBM (floor 16)
//   50176 x 3072, K = 768                                 199    183    201      tensor core under the power limit
//   90 x 768, K = 192, GELU (DeiT-Ti fc1, one image)        5.5    3.3    2.6    latency (small kernel)
//   90 x 192, K = 768, residual (DeiT-Ti fc2)               6.6    3.9    3.2    latency (pair kernel; 4.7 before it): 48 MMA steps in a row
// A k-block's loads cost their producer thread 265 to 450 cycles (try_wait 42, an arrival that the next try_wait waits behind
// 130, the loads themselves), the MMAs of 192 or 256 columns 384 or 512: three producers take k-blocks in turn.
//
// Every mbarrier wait is bounded (see sm100.cuh); a wait that gives up ORs a code into the
// device status word and the CTA unwinds.
//
// Replaces nn.Linear q/kv/proj/fc1/fc2/head, nn.GELU and the residual adds of
// vtpack/models/dge/deit_dge.py:38-44,72-74,96,127-128 (cuBLAS + ATen kernels there).
#include <string.h>

#include <memory>
#include <new>

#include "linear_tc.cuh"

namespace vtp {

using namespace sm100;

// EPI: what the epilogue does besides the bias, fixed at compile time so that a kernel only
// issues the instructions of the variant it is (a runtime flag would be if-converted and the
// GELU / LayerNorm arithmetic issued, predicated off, by every GEMM).
constexpr int EPI_GELU = 1, EPI_LN = 2, EPI_EMIT = 4, EPI_RES = 8;

template <int BN, int CG>
struct TcConf {
    static constexpr int EW = BN / SLAB * 4;             // epilogue warps: one per TMEM lane quarter and 64-column slab
    static constexpr int PRODUCERS = 3;                  // warps that take the k-blocks in turn
    static constexpr int FIRST_EPI = PRODUCERS + 1;      // ... behind the MMA warp
    static constexpr int THREADS = (FIRST_EPI + EW) * 32;
    static constexpr int A_BYTES = TBM * TBK * 2;
    static constexpr int B_BYTES = (BN / CG) * TBK * 2;  // this CTA's share of the W rows
    static constexpr int STAGING = EW * SLAB_BYTES;
    static constexpr int CTRL = 1024;                    // barriers, then the launch's scalars at CTRL_SCALARS
    static constexpr int CTRL_SCALARS = 512;
    // as deep a ring as fits; dynamic shared memory is only promised 16-byte alignment and the ring wants 1024, so
    // the kernel checks that what is left behind the aligned base fits (in practice the base is aligned already)
    static constexpr int FIT = (SMEM_MAX - STAGING - CTRL) / (A_BYTES + B_BYTES);
    static constexpr int STAGES = FIT > 8 ? 8 : FIT;
    static constexpr int RING = STAGES * (A_BYTES + B_BYTES);
    static constexpr int USED = RING + STAGING + CTRL;
    static constexpr int TOTAL = (USED + 1024 <= SMEM_MAX) ? USED + 1024 : SMEM_MAX;
    static constexpr int TMEM_COLS = 2 * BN <= 256 ? 256 : 512;
    static_assert(STAGES >= 3, "operand ring");
    static_assert((2 * STAGES + 4 + EW) * 8 + 16 <= CTRL_SCALARS, "barrier area");
};

// One GEMM problem of a launch: its tensor maps, and the scalars the kernel reads.  Each CTA copies the scalars of a launch
// to shared memory before it waits for the kernel in front: parameters are cold in every launch, and read where they are
// needed each line of them is a miss of some 500 cycles on the way to the first load, and another on the way to the first store.
struct TcScalars {
    const float* bias; const bf16* res; long long ldr;
    void* y; long long ldy;
    const int32_t* m_dev; int m_max; int N;
    FastDiv n_tiles;
    RowMap rm; LnFold ln;
    int use_tma_store;
};
struct TcMaps { CUtensorMap ta, tw, tws, ty, tr; };   // A, W (a whole tile's rows / 64 columns' rows), output, residual
// A launch works through one problem or two independent ones (same K, tile shape and epilogue kind): the
// tiles of the second fill the last, partial round of the first, and one launch's ramp and tail is saved.
struct TcSharedScalars { TcScalars p[2]; FastDiv groups; };
struct TcLaunch { TcMaps m[2]; TcSharedScalars s; };
static_assert(sizeof(TcSharedScalars) % 4 == 0 && sizeof(TcSharedScalars) <= 512, "copied to shared memory in words");

// The work items of one CTA group, in order.  Everything an item is worked out from is kept in registers: the first one
// stands between the kernel in front and this one's first load.
template <int BN, int CG, int NPROB>
struct Schedule {
    int M[NPROB], N[NPROB];
    FastDiv nt[NPROB];
    uint32_t G, tot0, full_items, strips, group;
    int parts;
    struct Item { int p, m0, ct0, width; };     // problem, first row of this CTA, output columns ct0 .. ct0 + width

    __device__ __forceinline__ Schedule(const TcSharedScalars& L, bool void_launch) {
        uint32_t total = 0;
        tot0 = 0;
#pragma unroll
        for (int i = 0; i < NPROB; ++i) {
            const int32_t* m_dev = L.p[i].m_dev;
            M[i] = L.p[i].m_max;
            N[i] = L.p[i].N;
            nt[i] = L.p[i].n_tiles;
            if (m_dev) M[i] = min(max(*reinterpret_cast<const volatile int32_t*>(m_dev), 0), M[i]);
            if (i == 1) tot0 = total;
            total += (uint32_t)((M[i] + TBM * CG - 1) / (TBM * CG)) * nt[i].d;
        }
        if (void_launch) total = 0;
        G = L.groups.d;
        group = blockIdx.x / CG;
        // Tail splitting.  A CTA group takes tiles group, group + G, ...; the R tiles left for the last, partial round are
        // cut into `parts` column strips of BN / parts columns, one per group, so that the round costs a fraction of a
        // tile instead of a whole one with most SMs idle.  A problem with fewer tiles than groups is all last round.
        // (Every sum of the epilogue covers at most one 64-column slab, so a row's bits do not depend on the strips.)
        full_items = total < G ? 0 : fast_div(total, L.groups) * G;
        const uint32_t R = total - full_items;
        parts = 1;
        if (BN == 256) parts = (R * 4 <= G) ? 4 : (R * 2 <= G ? 2 : 1);
        else if (BN == 192) parts = (R * 3 <= G) ? 3 : 1;
        else if (BN == 128) parts = (R * 2 <= G) ? 2 : 1;
        strips = R * (uint32_t)parts;
    }
    __device__ __forceinline__ bool at(uint32_t j, Item& it) const {
        uint32_t tile = group + j * G, sub = 0;
        int strip = BN;
        if (tile >= full_items) {
            const uint32_t u = tile - full_items;
            if (u >= strips) return false;
            const uint32_t q = parts == 3 ? u / 3u : u >> (parts == 4 ? 2 : parts - 1);
            tile = full_items + q;
            sub = u - q * (uint32_t)parts;
            strip = parts == 1 ? BN : (parts == 2 ? BN / 2 : SLAB);
        }
        it.p = (NPROB == 2 && tile >= tot0) ? 1 : 0;       // one-problem launches index their problem statically
        const bool second = NPROB == 2 && it.p;
        const uint32_t lt = tile - (second ? tot0 : 0);
        const FastDiv n_tiles = second ? nt[NPROB - 1] : nt[0];
        const uint32_t mt = fast_div(lt, n_tiles);
        const int nt0 = (int)(lt - mt * n_tiles.d) * BN;
        it.m0 = (int)mt * (TBM * CG) + (CG == 2 ? (int)cluster_ctarank() * TBM : 0);
        // the last column tile is as wide as the columns left, in 64s
        const int tile_w = min(BN, ((second ? N[NPROB - 1] : N[0]) - nt0 + SLAB - 1) & ~(SLAB - 1));
        it.ct0 = nt0 + (int)sub * strip;
        it.width = min(strip, tile_w - (int)sub * strip);
        return true;                                       // (a strip beyond a narrow tile's columns has no width)
    }
};

template <int BN, int CG, int EPI, bool F32, int NPROB>
__global__ void __launch_bounds__(TcConf<BN, CG>::THREADS, 1)
linear_tc_kernel(const __grid_constant__ TcLaunch L, int K, int* status) {
    using S = TcConf<BN, CG>;
    using Sched = Schedule<BN, CG, NPROB>;
    using Item = typename Sched::Item;
    constexpr int STAGES = S::STAGES, EW = S::EW, PRODUCERS = S::PRODUCERS;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* smem_a = base;
    uint8_t* smem_b = base + STAGES * S::A_BYTES;
    if (static_cast<int>(base - smem_raw) + S::USED > S::TOTAL) {
        if (threadIdx.x == 0 && status) atomicOr(status, STATUS_GEMM_PRODUCER);
        return;
    }
    uint8_t* smem_out = base + S::RING;
    uint8_t* ctrl = smem_out + S::STAGING;
    uint64_t* full = reinterpret_cast<uint64_t*>(ctrl);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;       // [2]
    uint64_t* acc_empty = acc_full + 2;        // [2]
    uint64_t* res_full = acc_empty + 2;        // [EW] the warp's residual slab has landed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(res_full + EW);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* void_s = reinterpret_cast<int*>(tmem_slot + 2);               // [2] launch_is_void in front of the wait and behind it
    const TcSharedScalars& sc = *reinterpret_cast<const TcSharedScalars*>(ctrl + S::CTRL_SCALARS);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rank = CG == 2 ? (int)cluster_ctarank() : 0;             // this CTA within its group

    bool void_launch = false;
    if (threadIdx.x == S::FIRST_EPI * 32) void_launch = launch_is_void(status);
    for (int i = threadIdx.x; i < (int)sizeof(TcSharedScalars) / 4; i += S::THREADS)
        reinterpret_cast<uint32_t*>(ctrl + S::CTRL_SCALARS)[i] = reinterpret_cast<const uint32_t*>(&L.s)[i];
    if (warp == 0 && elect_one()) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], CG * EW);       // rank 0's: the epilogue warps of the whole group
        }
        for (int b = 0; b < EW; ++b) mbar_init(&res_full[b], 1);
        *abort_flag = 0;
        fence_barrier_init();
        for (int i = 0; i < NPROB; ++i) {
            prefetch_tmap(&L.m[i].ta);
            prefetch_tmap(&L.m[i].tw);
            prefetch_tmap(&L.m[i].tws);
        }
    }
    if (warp == PRODUCERS) {
        if (CG == 2) { tmem_alloc_pair(tmem_slot, S::TMEM_COLS); tmem_relinquish_pair(); }
        else { tmem_alloc(tmem_slot, S::TMEM_COLS); tmem_relinquish(); }
    }
    if (warp == 1 && elect_one()) {
        for (int i = 0; i < NPROB; ++i) {
            prefetch_tmap(&L.m[i].ty);
            if (EPI & EPI_RES) prefetch_tmap(&L.m[i].tr);
        }
    }
    if (threadIdx.x == S::FIRST_EPI * 32) void_s[0] = void_launch ? 1 : 0;
    tc_fence_before_sync();
    __syncthreads();
    if (CG == 2) cluster_sync_all();     // the partner's barriers exist before anything arrives on them
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const bool known_void = lead_word<CG>(void_s) != 0;

    // Everything above is independent of the kernel in front of this one on the stream; from
    // here on its results (row count, operands, residual, statistics) are read.
    pdl_begin();
    const Sched sched(sc, known_void);

    // The two loops below run in one thread each, and a k-block has a few hundred cycles: shared memory goes by 32-bit
    // addresses that advance with the ring.
    const uint32_t full_a = smem_u32(full), empty_a = smem_u32(empty);
    if (warp < PRODUCERS) {
        if (elect_one()) {
            // ------------------------------------------------------------ TMA producers
            // A k-block costs its producer some 400 cycles (the wait, the barrier, two loads), which is about what the tensor core
            // takes for it: three warps take them in turn.
            const uint32_t ring_a = smem_u32(smem_a), ring_b = smem_u32(smem_b);
            int s = 0, turn = warp;
            uint32_t ph = 1, filled = 0;
            bool ok = true;
            Item wi;
            for (uint32_t j = 0; ok && sched.at(j, wi); ++j) {
                if (wi.width <= 0) continue;
                const TcMaps& P = L.m[wi.p];
                const bool whole = wi.width == BN;
                const int wshare = wi.width / CG;
                const uint32_t bytes = CG * (S::A_BYTES + (uint32_t)wshare * TBK * 2);     // of the whole group
                const int wrow = wi.ct0 + rank * wshare;
                for (int x = 0; x < K; x += TBK) {
                    if (turn == 0) {
                        const uint32_t fb = full_a + 8 * s, da = ring_a + s * S::A_BYTES, db = ring_b + s * S::B_BYTES;
                        ok = mbar_wait_a(empty_a + 8 * s, ph, abort_flag, status, STATUS_GEMM_PRODUCER);
                        if (!ok) break;
                        // (both CTAs' bytes of a pair are counted on rank 0's barrier, which its MMA thread waits on)
                        if (CG == 1 || rank == 0) mbar_arrive_expect_tx_a(fb, bytes);
                        const uint32_t lead = CG == 1 ? fb : mapa_u32(fb, 0);
                        tma_load_2d_a<CG>(da, &P.ta, lead, x, wi.m0);
                        if (whole) tma_load_2d_a<CG>(db, &P.tw, lead, x, wrow);
                        else for (int c = 0; c < wshare; c += SLAB / CG) tma_load_2d_a<CG>(db + c * (TBK * 2), &P.tws, lead, x, wrow + c);
                        turn = PRODUCERS;
                    }
                    --turn;
                    ++filled;
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
            if (CG == 2 && ok) {
                // The MMA thread's last commits arrive on this CTA's `empty` barriers, from the partner for rank 1: wait for
                // them, so that nothing is signalled into a CTA that has retired.  Each producer for its own last fills: it
                // has seen the stage's commit before, so the parity is that of the commit it means.
                for (uint32_t f = filled > (uint32_t)STAGES ? filled - STAGES : 0; f < filled && ok; ++f)
                    if (f % PRODUCERS == (uint32_t)warp)
                        ok = mbar_wait_a(empty_a + 8 * (f % STAGES), (f / STAGES) & 1, abort_flag, status, STATUS_GEMM_PRODUCER);
            }
        }
        __syncwarp();
    } else if (warp == PRODUCERS) {
        if (rank == 0 && elect_one()) {
            // -------------------------------------------------------------- MMA issuer (of the group)
            int s = 0, lt = 0;
            uint32_t ph = 0;
            bool ok = true;
            const uint64_t adesc0 = smem_desc_sw128(smem_u32(smem_a));
            const uint64_t bdesc0 = smem_desc_sw128(smem_u32(smem_b));
            Item wi;
            for (uint32_t j = 0; ok && sched.at(j, wi); ++j) {
                if (wi.width <= 0) continue;
                const uint32_t idesc = idesc_bf16_f32(TBM * CG, wi.width, 0, 0);
                const int buf = lt & 1;
                ok = mbar_wait(&acc_empty[buf], ((lt >> 1) & 1) ^ 1, abort_flag, status, STATUS_GEMM_MMA);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + buf * BN;
                for (int x = 0; x < K; x += TBK) {
                    ok = mbar_wait_a(full_a + 8 * s, ph, abort_flag, status, STATUS_GEMM_MMA);
                    if (!ok) break;
                    tc_fence_after_sync();
                    const uint64_t adesc = adesc0 + (uint64_t)(s * (S::A_BYTES >> 4));
                    const uint64_t bdesc = bdesc0 + (uint64_t)(s * (S::B_BYTES >> 4));
#pragma unroll
                    for (int k = 0; k < TBK / 16; ++k) {
                        // 16 bf16 of K = 32 bytes = 2 descriptor address units inside the swizzle row
                        if (CG == 2) umma_ss_pair(d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc, (x | k) != 0 ? 1u : 0u);
                        else umma_ss(d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc, (x | k) != 0 ? 1u : 0u);
                    }
                    umma_commit_a<CG>(empty_a + 8 * s);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                if (ok) umma_commit_a<CG>(smem_u32(&acc_full[buf]));
                ++lt;
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------- epilogue
        // A warp works on its own: TMEM lanes 32 * (warp % 4) .. + 31 (the rows it may read) of one 64-column slab of each
        // item, through a staging buffer of its own that its own TMA store empties; no warp waits for another.
        const int e = warp - S::FIRST_EPI;
        const int quarter = warp & 3;
        const int sl = e >> 2;                        // slab of an item
        const bool leader = elect_one();
        uint8_t* buf_s = smem_out + e * SLAB_BYTES;   // residual in, result out
        // the accumulator goes back to the MMA thread, which runs in the group's rank-0 CTA
        auto release_acc = [&](int b) {
            tc_fence_before_sync();
            __syncwarp();
            if (leader) {
                if (CG == 2) mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[b]), 0));
                else mbar_arrive(&acc_empty[b]);
            }
        };
        // In a launch that turns out to be void the accumulators still change hands, but this CTA has no rows.
        if (threadIdx.x == S::FIRST_EPI * 32) void_s[1] = launch_is_void(status) ? 1 : 0;
        named_barrier(1, EW * 32);
        const bool stores = void_s[1] == 0;
        int lt = 0;
        uint32_t res_ph = 0;
        bool ok = true;
        Item wi;
        for (uint32_t j = 0; ok && sched.at(j, wi); ++j) {
            if (wi.width <= 0) continue;
            const TcScalars& P = sc.p[wi.p];
            const TcMaps& T = L.m[wi.p];
            const int M = !stores ? 0 : (NPROB == 2 && wi.p) ? sched.M[NPROB - 1] : sched.M[0], N = P.N;
            const int buf = lt & 1;
            const uint32_t aph = (lt >> 1) & 1;
            ++lt;
            const int wrow0 = wi.m0 + quarter * 32;         // the warp's first row
            const int n0 = wi.ct0 + sl * SLAB;
            const bool active = wrow0 < M && sl * SLAB < wi.width;
            // the residual of 32 valid rows comes by TMA, mapped rows and those beside the last valid one are copied by the warp
            const bool res_tma = P.rm.res_mod <= 0 && wrow0 + 32 <= M;
            float2 b2[8], s2[8];                                       // bias and fold vector of this thread's columns
            float ln_a = 1.f, ln_b = 0.f;                              // of row `lane` of the warp
            if (active) {
                // what the slab needs besides the accumulator travels while the MMAs run
                // (the columns of a partial slab beyond N read the last ones; what is made of them is not stored)
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const int nb = min(n0 + 8 * c, N - 8) + 2 * (lane & 3);
                    b2[c] = __ldg(reinterpret_cast<const float2*>(P.bias ? P.bias + nb : g_no_bias));
                    if (EPI & EPI_LN) s2[c] = __ldg(reinterpret_cast<const float2*>(NPROB == 2 && !P.ln.s ? g_no_bias : P.ln.s + nb));
                }
                if (EPI & EPI_RES) {
                    if (leader) bulk_wait_group_read0();               // the last item's store has read the buffer
                    __syncwarp();
                    if (!res_tma) {
                        const int c = lane & 7;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int rr = i * 4 + (lane >> 3);
                            uint4 v = make_uint4(0, 0, 0, 0);
                            if (wrow0 + rr < M && n0 + c * 8 < N)
                                v = *reinterpret_cast<const uint4*>(P.res + map_res_row(P.rm, wrow0 + rr) * P.ldr + n0 + c * 8);
                            *reinterpret_cast<uint4*>(buf_s + rr * 128 + ((c ^ (rr & 7)) << 4)) = v;
                        }
                        __syncwarp();
                    } else if (leader) {
                        mbar_arrive_expect_tx(&res_full[e], SLAB_BYTES);
                        tma_load_2d(buf_s, &T.tr, &res_full[e], n0, wrow0);
                    }
                }
                if ((EPI & EPI_LN) && wrow0 + lane < M) row_fold(P.ln, wrow0 + lane, ln_a, ln_b);
            }
            ok = mbar_wait_warp(&acc_full[buf], aph, abort_flag, status, STATUS_GEMM_EPILOGUE);
            if (!ok) break;
            tc_fence_after_sync();
            if (!active) {
                release_acc(buf);
                continue;
            }
            if ((EPI & EPI_RES) && res_tma) {
                ok = mbar_wait_warp(&res_full[e], res_ph, abort_flag, status, STATUS_GEMM_EPILOGUE);
                res_ph ^= 1;
                if (!ok) break;
            }
            // A thread holds columns 8 c + 2 (lane % 4), + 1 of rows lane / 4 + 8 k: a bias or fold vector value serves four rows
            // of eight lanes.  (With a whole row to a thread every value of those vectors is a load of the whole warp, and the
            // sixteen warps' loads, four passes for 16 bytes each, took as long as the tile's MMAs.)
            const uint32_t tacc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * BN + sl * SLAB;
            float fa[4], fb[4];
            if (EPI & EPI_LN) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    fa[k] = __shfl_sync(0xffffffffu, ln_a, (lane >> 2) + 8 * k);
                    fb[k] = __shfl_sync(0xffffffffu, ln_b, (lane >> 2) + 8 * k);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {                      // 16 rows at a time
                uint32_t r[32];
                __syncwarp();                                  // tcgen05.ld is warp-collective
                tmem_ld_16x256b_x8(tacc + (static_cast<uint32_t>(16 * h) << 16), r);
                tmem_ld_wait();
                if (h == 1) release_acc(buf);                  // the warp's last columns are in registers
                // 16-byte cells for four 8 x 8 matrices at a time: rows 16 h + 0..7 and + 8..15 of chunks c and c + 1
                const int mrow = 16 * h + (lane & 15);
                const uint32_t cells = smem_u32(buf_s) + (uint32_t)mrow * 128u, cx = (uint32_t)(mrow & 7);
                if (h == 0 && !(EPI & EPI_RES) && !F32) {
                    if (leader) bulk_wait_group_read0();       // the last item's store has read the buffer
                    __syncwarp();
                }
                float p1[2][4], p2[2][4];                      // EPI_EMIT: sums and sums of squares, 16 columns each, of the two rows
#pragma unroll
                for (int c = 0; c < 8; c += 2) {
                    const uint32_t cell = cells + (((uint32_t)(c + (lane >> 4)) ^ cx) << 4);
                    uint32_t rv[4], o[4];
                    if (EPI & EPI_RES) ldmatrix_x4(cell, rv);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {              // matrix i: chunk c + i / 2, rows + 8 * (i % 2)
                        const int cc = c + (i >> 1), k = 2 * h + (i & 1);
                        const float a0 = __uint_as_float(r[4 * cc + 2 * (i & 1)]), a1 = __uint_as_float(r[4 * cc + 2 * (i & 1) + 1]);
                        float v0, v1;
                        if (EPI & EPI_LN) {
                            v0 = fmaf(fa[k], a0, fmaf(fb[k], s2[cc].x, b2[cc].x));
                            v1 = fmaf(fa[k], a1, fmaf(fb[k], s2[cc].y, b2[cc].y));
                        } else {
                            v0 = a0 + b2[cc].x;
                            v1 = a1 + b2[cc].y;
                        }
                        if (EPI & EPI_GELU) {
                            const uint32_t g = gelu_pair_f16(v0, v1);
                            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&g));
                            v0 = f.x;
                            v1 = f.y;
                        }
                        if (EPI & EPI_RES) {
                            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&rv[i]));
                            v0 += f.x;
                            v1 += f.y;
                        }
                        if (EPI & EPI_EMIT) {
                            const bool in = n0 + 8 * cc < N;
                            const float z0 = in ? v0 : 0.f, z1 = in ? v1 : 0.f;
                            const float q1 = z0 + z1, q2 = fmaf(z1, z1, __fmul_rn(z0, z0));
                            if (i < 2) { p1[i][c >> 1] = q1; p2[i][c >> 1] = q2; }
                            else { p1[i & 1][c >> 1] += q1; p2[i & 1][c >> 1] += q2; }
                        }
                        if (F32) {
                            const int rr = wrow0 + (lane >> 2) + 8 * k;
                            if (rr < M && n0 + 8 * cc < N)
                                *reinterpret_cast<float2*>(static_cast<float*>(P.y) + map_out_row(P.rm, rr) * P.ldy + n0 + 8 * cc + 2 * (lane & 3)) =
                                    make_float2(v0, v1);
                        } else {
                            const __nv_bfloat162 t = __floats2bfloat162_rn(v0, v1);
                            o[i] = *reinterpret_cast<const uint32_t*>(&t);
                        }
                    }
                    if (!F32) stmatrix_x4(cell, o);
                }
                if (EPI & EPI_EMIT) {
                    // (16 + 16) + (16 + 16) columns of a lane, then the four lanes of a row: (0 + 1) + (2 + 3)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        float e1 = (p1[i][0] + p1[i][1]) + (p1[i][2] + p1[i][3]), e2 = (p2[i][0] + p2[i][1]) + (p2[i][2] + p2[i][3]);
                        e1 += __shfl_xor_sync(0xffffffffu, e1, 1); e2 += __shfl_xor_sync(0xffffffffu, e2, 1);
                        e1 += __shfl_xor_sync(0xffffffffu, e1, 2); e2 += __shfl_xor_sync(0xffffffffu, e2, 2);
                        const int rr = wrow0 + 16 * h + 8 * i + (lane >> 2);
                        if ((lane & 3) == 0 && rr < M) P.ln.emit[(size_t)rr * P.ln.slots + n0 / SLAB] = make_float2(e1, e2);
                    }
                }
            }
            if (F32) continue;
            if (P.use_tma_store && wrow0 + 32 <= M) {
                fence_proxy_async_smem();
                __syncwarp();
                if (leader) {
                    tma_store_2d(&T.ty, buf_s, n0, wrow0);
                    bulk_commit_group();
                }
            } else {
                // rows beyond M among the warp's, or mapped rows: eight lanes copy a row's 128 bytes
                __syncwarp();
                const int c = lane & 7;
                bf16* y = static_cast<bf16*>(P.y) + n0 + c * 8;
                const bool in = n0 + c * 8 < N;
                const int rows = M - wrow0;
                const long long ldy = P.ldy;
                const bool mapped = P.rm.out_grp > 0;
                bf16* yr = y + (wrow0 + (lane >> 3)) * ldy;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int rr = i * 4 + (lane >> 3);
                    const uint4 v = lds_u4(smem_u32(buf_s) + rr * 128 + ((c ^ (rr & 7)) << 4));
                    if (mapped) yr = y + map_out_row(P.rm, wrow0 + rr) * ldy;
                    if (rr < rows && in) *reinterpret_cast<uint4*>(yr) = v;
                    yr += 4 * ldy;
                }
                fence_proxy_async_smem();                      // (a TMA residual may be the buffer's next content)
                __syncwarp();
            }
        }
        if (leader) bulk_wait_group0();               // every TMA store has landed before the CTA retires
        __syncwarp();
    }
    if (*abort_flag) {
        // Unwinding after a wait gave up: give copies still in flight time to land before
        // shared memory and TMEM are released.
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) { }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (CG == 2) cluster_sync_all();     // the partner no longer reads this CTA's operands or signals its barriers
    if (warp == PRODUCERS) {
        if (CG == 2) tmem_dealloc_pair(tmem_base, S::TMEM_COLS);
        else tmem_dealloc(tmem_base, S::TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------ small problems
// The same products for problems of no more 128 x 64 tiles than SMs, or 128 x 128 tiles (linear_tcgen05_pair), where a launch is a chain of
// latencies: one tile per CTA, which tile it is known before the wait for the kernel in front (the loads do not wait for the row
// count, only the stores do), sixteen epilogue warps with 16 columns of each 64 that go straight between registers and global memory.  Same MMA steps and
// sums in the same order as linear_tc_kernel: a row's bits do not depend on which of the two it comes from.
template <int BN_>
struct SmallConf {
    static constexpr int BN = BN_, STAGES = BN == 64 ? 8 : 6, PRODUCERS = 3, FIRST_EPI = 4, EW = 16, THREADS = (FIRST_EPI + EW) * 32;
    static constexpr int A_BYTES = TBM * TBK * 2, B_BYTES = BN * TBK * 2;
    static constexpr int RING = STAGES * (A_BYTES + B_BYTES);
    static constexpr int SUMS = TBM * 16 * 8;            // EPI_EMIT: (sum, sum of squares) of four columns of a row each
    static constexpr int USED = RING + SUMS + 256;
    static constexpr int TOTAL = USED + 1024;
    static_assert(TOTAL <= SMEM_MAX, "shared memory budget");
};
// n_tiles: tiles of a row; grid0: CTAs of the first problem; at_once: CTAs that are sure to start together
struct SmallLaunch { CUtensorMap ta[2], tw[2]; TcScalars p[2]; int grid0, at_once; };

template <int BN, int EPI, bool F32, int NPROB>
__global__ void __launch_bounds__(SmallConf<BN>::THREADS, 1)
linear_tc_small_kernel(const __grid_constant__ SmallLaunch L, int K, int* status) {
    using S = SmallConf<BN>;
    constexpr int H = BN / SLAB;                                       // 64-column halves of a tile
    static_assert(H == 1 || !(EPI & EPI_EMIT), "one half's row sums at a time");
    constexpr int STAGES = S::STAGES, PRODUCERS = S::PRODUCERS;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t ring_a = smem_u32(base), ring_b = ring_a + STAGES * S::A_BYTES;
    float2* sums = reinterpret_cast<float2*>(base + S::RING);
    uint64_t* full = reinterpret_cast<uint64_t*>(base + S::RING + S::SUMS);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* void_s = reinterpret_cast<int*>(tmem_slot + 2);               // [2] launch_is_void in front of the wait and behind it
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t full_a = smem_u32(full), empty_a = smem_u32(empty);

    const int prob = (NPROB == 2 && (int)blockIdx.x >= L.grid0) ? 1 : 0;
    const TcScalars& P = L.p[prob];
    const uint32_t tile = blockIdx.x - (prob ? L.grid0 : 0);
    const uint32_t mt = fast_div(tile, P.n_tiles);
    const int m0 = (int)mt * TBM, ct0 = (int)(tile - mt * P.n_tiles.d) * S::BN;
    const int nkb = K / TBK;

    if (warp == 0 && elect_one()) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1 && elect_one()) { prefetch_tmap(&L.ta[prob]); prefetch_tmap(&L.tw[prob]); }
    if (warp == PRODUCERS) { tmem_alloc(tmem_slot, BN); tmem_relinquish(); }
    if (threadIdx.x == S::FIRST_EPI * 32) void_s[0] = launch_is_void(status) ? 1 : 0;
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const bool known_void = void_s[0] != 0;
    pdl_begin();
    // a CTA that starts when others have ended looks first whether its rows exist
    const bool none = (int)blockIdx.x >= L.at_once && P.m_dev && m0 >= *reinterpret_cast<const volatile int32_t*>(P.m_dev);

    if (known_void || none) {
    } else if (warp < PRODUCERS) {
        if (elect_one()) {
            for (int kb = warp; kb < nkb; kb += PRODUCERS) {
                const int s = kb % STAGES;
                if (kb >= STAGES && !mbar_wait_a(empty_a + 8 * s, ((kb / STAGES) & 1) ^ 1, abort_flag, status, STATUS_GEMM_PRODUCER)) break;
                mbar_arrive_expect_tx_a(full_a + 8 * s, S::A_BYTES + S::B_BYTES);
                tma_load_2d_a<1>(ring_a + s * S::A_BYTES, &L.ta[prob], full_a + 8 * s, kb * TBK, m0);
                tma_load_2d_a<1>(ring_b + s * S::B_BYTES, &L.tw[prob], full_a + 8 * s, kb * TBK, ct0);
            }
        }
        __syncwarp();
    } else if (warp == PRODUCERS) {
        if (elect_one()) {
            const uint64_t adesc0 = smem_desc_sw128(ring_a), bdesc0 = smem_desc_sw128(ring_b);
            const uint32_t idesc = idesc_bf16_f32(TBM, S::BN, 0, 0);
            bool ok = true;
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = kb % STAGES;
                ok = mbar_wait_a(full_a + 8 * s, (kb / STAGES) & 1, abort_flag, status, STATUS_GEMM_MMA);
                if (!ok) break;
                tc_fence_after_sync();
                const uint64_t adesc = adesc0 + (uint64_t)(s * (S::A_BYTES >> 4)), bdesc = bdesc0 + (uint64_t)(s * (S::B_BYTES >> 4));
#pragma unroll
                for (int k = 0; k < TBK / 16; ++k) umma_ss(tmem_base, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
                if (kb + STAGES < nkb) umma_commit_a<1>(empty_a + 8 * s);
            }
            if (ok) umma_commit_a<1>(smem_u32(acc_full));
        }
        __syncwarp();
    } else {
        const int g = (warp - S::FIRST_EPI) >> 2;         // which 16 columns of a half
        const int row = (warp & 3) * 32 + lane;           // tile row = TMEM lane
        const int m = m0 + row, N = P.N;
        // (a launch that turns out to be void forms its products and has no rows to store)
        if (threadIdx.x == S::FIRST_EPI * 32) void_s[1] = launch_is_void(status) ? 1 : 0;
        int M = P.m_max;
        if (P.m_dev) M = min(max(*reinterpret_cast<const volatile int32_t*>(P.m_dev), 0), M);
        named_barrier(5, S::EW * 32);
        if (void_s[1] != 0) M = 0;
        // what the outputs need besides the accumulator travels while the operands are loaded and multiplied
        const bool live = m0 + (warp & 3) * 32 < M;       // the warp has rows
        const bool row_ok = m < M;
        float add[H][16], ln_a = 1.f, ln_b = 0.f;
        uint4 rv[H][2];
        if ((EPI & EPI_LN) && live && row_ok) row_fold(P.ln, m, ln_a, ln_b);
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int n0 = ct0 + h * SLAB + g * 16;
            const bool c1 = n0 + 8 < N;               // its columns exist, eight at a time
            if (live && n0 < N) {
                float sv[16];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int nb = min(n0 + 8 * (q >> 1), N - 8);
                    const float* bias = P.bias ? P.bias + nb : g_no_bias;
                    const float4 b4 = __ldg(reinterpret_cast<const float4*>(bias) + (q & 1));
                    add[h][4 * q] = b4.x; add[h][4 * q + 1] = b4.y; add[h][4 * q + 2] = b4.z; add[h][4 * q + 3] = b4.w;
                    if (EPI & EPI_LN) {
                        const float4 s4 = __ldg(reinterpret_cast<const float4*>(NPROB == 2 && !P.ln.s ? g_no_bias : P.ln.s + nb) + (q & 1));
                        sv[4 * q] = s4.x; sv[4 * q + 1] = s4.y; sv[4 * q + 2] = s4.z; sv[4 * q + 3] = s4.w;
                    }
                }
                if ((EPI & EPI_RES) && row_ok) {
                    const bf16* r = P.res + map_res_row(P.rm, m) * P.ldr + n0;
                    rv[h][0] = *reinterpret_cast<const uint4*>(r);
                    rv[h][1] = c1 ? *reinterpret_cast<const uint4*>(r + 8) : make_uint4(0, 0, 0, 0);
                }
                if (EPI & EPI_LN) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) add[h][i] = fmaf(ln_b, sv[i], add[h][i]);
                }
            }
        }
        const long long orow = map_out_row(P.rm, row_ok ? m : m0);
        const bool ok = mbar_wait_warp(acc_full, 0, abort_flag, status, STATUS_GEMM_EPILOGUE);
        if (ok && live) tc_fence_after_sync();
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int n0 = ct0 + h * SLAB + g * 16;
            const bool c1 = n0 + 8 < N;
            if (ok && live) {
                uint32_t r[16];
                float e1[4] = {0.f, 0.f, 0.f, 0.f}, e2[4] = {0.f, 0.f, 0.f, 0.f};
                __syncwarp();
                tmem_ld_32x16(tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + h * SLAB + g * 16, r);
                tmem_ld_wait();
                if (n0 < N) {
                    uint4 out[2];
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        float v[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float acc = __uint_as_float(r[8 * c + i]);
                            v[i] = (EPI & EPI_LN) ? fmaf(ln_a, acc, add[h][8 * c + i]) : acc + add[h][8 * c + i];
                        }
                        if (EPI & EPI_GELU) gelu8(v);
                        if (EPI & EPI_RES) {
                            Vec<bf16> w;
                            float rf[8];
                            w.raw = rv[h][c];
                            w.to_float(rf);
#pragma unroll
                            for (int i = 0; i < 8; ++i) v[i] += rf[i];
                        }
                        if (EPI & EPI_EMIT) {
                            // as in linear_tc_kernel: columns 2 q, 2 q + 1 of the first and of the second eight
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                const float z0 = (c == 0 || c1) ? v[2 * q] : 0.f, z1 = (c == 0 || c1) ? v[2 * q + 1] : 0.f;
                                const float q1 = z0 + z1, q2 = fmaf(z1, z1, __fmul_rn(z0, z0));
                                if (c == 0) { e1[q] = q1; e2[q] = q2; }
                                else { e1[q] += q1; e2[q] += q2; }
                            }
                        }
                        if (F32) {
                            if (row_ok && (c == 0 || c1)) {
                                float* y = static_cast<float*>(P.y) + orow * P.ldy + n0 + 8 * c;
                                reinterpret_cast<float4*>(y)[0] = make_float4(v[0], v[1], v[2], v[3]);
                                reinterpret_cast<float4*>(y)[1] = make_float4(v[4], v[5], v[6], v[7]);
                            }
                        } else {
                            Vec<bf16> ov;
                            ov.from_float(v);
                            out[c] = ov.raw;
                        }
                    }
                    if (!F32 && row_ok) {
                        bf16* y = static_cast<bf16*>(P.y) + orow * P.ldy + n0;
                        *reinterpret_cast<uint4*>(y) = out[0];
                        if (c1) *reinterpret_cast<uint4*>(y + 8) = out[1];
                    }
                }
                if (EPI & EPI_EMIT) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) sums[(g * 4 + q) * TBM + row] = make_float2(e1[q], e2[q]);
                }
            }
            if ((EPI & EPI_EMIT) && live) {
                // the four warps of these rows (all of them get here): a column pair's 16 columns of each, (0 + 1) + (2 + 3), then the
                // pairs, (0 + 1) + (2 + 3)
                named_barrier(1 + (warp & 3), 128);
                if (g == 0 && row_ok && ok) {
                    float t1[4], t2[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float2 a = sums[(0 * 4 + q) * TBM + row], b = sums[(1 * 4 + q) * TBM + row];
                        const float2 c = sums[(2 * 4 + q) * TBM + row], d = sums[(3 * 4 + q) * TBM + row];
                        t1[q] = (a.x + b.x) + (c.x + d.x);
                        t2[q] = (a.y + b.y) + (c.y + d.y);
                    }
                    P.ln.emit[(size_t)m * P.ln.slots + ct0 / SLAB] = make_float2((t1[0] + t1[1]) + (t1[2] + t1[3]), (t2[0] + t2[1]) + (t2[2] + t2[3]));
                }
            }
        }
    }
    if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) { }          // let copies in flight land before releasing memory
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == PRODUCERS) tmem_dealloc(tmem_base, BN);
}

// The same for a long reduction: a pair of CTAs shares a 128 x BN tile, 64 rows of A and half of the columns' W rows each.  A CTA's share of a
// k-block is 12 or 16 KB instead of 24, and what bounds a CTA is how fast its operands come (64 bytes a clock); the MMAs
// of a pair with 64 rows each take half of the cycles too.  Accumulator: lanes 0 to 63 hold the CTA's rows and the tile's
// first half of the columns, lanes 64 to 127 the same rows and the other half.
template <int BN_>
struct PairConf {
    static constexpr int BN = BN_, STAGES = BN == 64 ? 8 : 6, PRODUCERS = 3, FIRST_EPI = 4, EW = 16, THREADS = (FIRST_EPI + EW) * 32;
    static constexpr int ROWS = TBM / 2, A_BYTES = ROWS * TBK * 2, B_BYTES = BN / 2 * TBK * 2, STAGE = 2 * (A_BYTES + B_BYTES);      // 128 of K
    static constexpr int RING = STAGES * STAGE;
    static constexpr int SUMS = ROWS * 32 * 8;           // EPI_EMIT: (sum, sum of squares) of 32 column groups of a row
    static constexpr int USED = RING + SUMS + 256;
    static constexpr int TOTAL = USED + 1024;
    static constexpr int TMEM_COLS = 64;
    static constexpr int COLS = BN / 8;                  // columns of an epilogue warp
    static_assert(TOTAL <= SMEM_MAX && B_BYTES % 1024 == 0, "shared memory budget");
};

template <int BN, int EPI>
__global__ void __launch_bounds__(PairConf<BN>::THREADS, 1)
linear_tc_pair_kernel(const __grid_constant__ SmallLaunch L, int K, int* status) {
    using S = PairConf<BN>;
    constexpr int STAGES = S::STAGES, PRODUCERS = S::PRODUCERS, COLS = S::COLS;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t ring = smem_u32(base);
    float2* sums = reinterpret_cast<float2*>(base + S::RING);
    uint64_t* full = reinterpret_cast<uint64_t*>(base + S::RING + S::SUMS);     // rank 0's
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* void_s = reinterpret_cast<int*>(tmem_slot + 2);               // [2] launch_is_void in front of the wait and behind it
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank();
    const uint32_t full_a = smem_u32(full), empty_a = smem_u32(empty);

    const TcScalars& P = L.p[0];
    const uint32_t tile = blockIdx.x >> 1;
    const uint32_t mt = fast_div(tile, P.n_tiles);
    const int m0 = (int)mt * TBM, ct0 = (int)(tile - mt * P.n_tiles.d) * BN;
    const int n_stages = K / (2 * TBK);

    if (warp == 0 && elect_one()) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1 && elect_one()) { prefetch_tmap(&L.ta[0]); prefetch_tmap(&L.tw[0]); }
    if (warp == PRODUCERS) { tmem_alloc_pair(tmem_slot, S::TMEM_COLS); tmem_relinquish_pair(); }
    if (threadIdx.x == S::FIRST_EPI * 32) void_s[0] = launch_is_void(status) ? 1 : 0;
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();                  // the partner's barriers exist before anything arrives on them
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const bool known_void = lead_word<2>(void_s) != 0;
    pdl_begin();

    if (known_void) {
    } else if (warp < PRODUCERS) {
        if (elect_one()) {
            for (int i = warp; i < n_stages; i += PRODUCERS) {
                const int s = i % STAGES;
                if (i >= STAGES && !mbar_wait_a(empty_a + 8 * s, ((i / STAGES) & 1) ^ 1, abort_flag, status, STATUS_GEMM_PRODUCER)) break;
                // (both CTAs' bytes are counted on rank 0's barrier, which its MMA thread waits on)
                if (rank == 0) mbar_arrive_expect_tx_a(full_a + 8 * s, 2 * S::STAGE);
                const uint32_t lead = mapa_u32(full_a + 8 * s, 0), dst = ring + s * S::STAGE;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    tma_load_2d_a<2>(dst + k * S::A_BYTES, &L.ta[0], lead, (2 * i + k) * TBK, m0 + rank * S::ROWS);
                    tma_load_2d_a<2>(dst + 2 * S::A_BYTES + k * S::B_BYTES, &L.tw[0], lead, (2 * i + k) * TBK, ct0 + rank * (BN / 2));
                }
            }
        }
        __syncwarp();
    } else if (warp == PRODUCERS) {
        if (rank == 0 && elect_one()) {
            constexpr uint32_t idesc = idesc_bf16_f32(TBM, BN, 0, 0);
            const uint32_t desc0 = (uint32_t)smem_desc_sw128(ring);
            bool ok = true, peeked = false;
            int s = 0;
            uint32_t ph = 0;
            for (int i = 0; i < n_stages; ++i) {
                if (!peeked) ok = mbar_wait_a(full_a + 8 * s, ph, abort_flag, status, STATUS_GEMM_MMA);
                if (!ok) break;
                tc_fence_after_sync();
                const bool wrap = s + 1 == STAGES;
                // (a look behind the MMAs would wait until the tensor core has taken them)
                peeked = mbar_try_wait_a(wrap ? full_a : full_a + 8 * (s + 1), wrap ? ph ^ 1 : ph);
                const uint32_t a = desc0 + s * (S::STAGE >> 4), b = a + (2 * S::A_BYTES >> 4);
#pragma unroll
                for (int k = 0; k < 2 * TBK / 16; ++k) {
                    const uint32_t ad = a + (k >> 2) * (S::A_BYTES >> 4) + 2 * (k & 3), bd = b + (k >> 2) * (S::B_BYTES >> 4) + 2 * (k & 3);
                    if (k == 0 && i == 0) umma_ss_pair_lo<false>(tmem_base, ad, bd, idesc);
                    else umma_ss_pair_lo<true>(tmem_base, ad, bd, idesc);
                }
                if (i + STAGES < n_stages) umma_commit_a<2>(empty_a + 8 * s);
                if (wrap) { s = 0; ph ^= 1; }
                else ++s;
            }
            if (ok) umma_commit_a<2>(smem_u32(acc_full));
        }
        __syncwarp();
    } else {
        const int g = (warp - S::FIRST_EPI) >> 2, quarter = warp & 3;
        const int half = quarter >> 1, row = (quarter & 1) * 32 + lane;          // of the tile's columns; of the CTA's rows
        const int wm0 = m0 + rank * S::ROWS + (quarter & 1) * 32, m = wm0 + lane, N = P.N;
        const int c0 = half * (BN / 2) + g * COLS, n0 = ct0 + c0;
        // (a launch that turns out to be void forms its products and has no rows to store)
        if (threadIdx.x == S::FIRST_EPI * 32) void_s[1] = launch_is_void(status) ? 1 : 0;
        int M = P.m_max;
        if (P.m_dev) M = min(max(*reinterpret_cast<const volatile int32_t*>(P.m_dev), 0), M);
        named_barrier(5, S::EW * 32);
        if (void_s[1] != 0) M = 0;
        const bool live = wm0 < M, row_ok = m < M;        // the warp, the lane has rows
        float add[COLS], ln_a = 1.f, ln_b = 0.f;
        uint4 rv[COLS / 8];
        if (live) {
            if ((EPI & EPI_LN) && row_ok) row_fold(P.ln, m, ln_a, ln_b);
#pragma unroll
            for (int c = 0; c < COLS / 8; ++c) {
                const int nb = min(n0 + 8 * c, N - 8);
                const float* bias = P.bias ? P.bias + nb : g_no_bias;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float4 b4 = __ldg(reinterpret_cast<const float4*>(bias) + q);
                    float* d = add + 8 * c + 4 * q;
                    d[0] = b4.x; d[1] = b4.y; d[2] = b4.z; d[3] = b4.w;
                    if (EPI & EPI_LN) {
                        const float4 s4 = __ldg(reinterpret_cast<const float4*>(P.ln.s + nb) + q);
                        d[0] = fmaf(ln_b, s4.x, d[0]); d[1] = fmaf(ln_b, s4.y, d[1]); d[2] = fmaf(ln_b, s4.z, d[2]); d[3] = fmaf(ln_b, s4.w, d[3]);
                    }
                }
                rv[c] = make_uint4(0, 0, 0, 0);
                if ((EPI & EPI_RES) && row_ok && n0 + 8 * c < N)
                    rv[c] = *reinterpret_cast<const uint4*>(P.res + map_res_row(P.rm, m) * P.ldr + n0 + 8 * c);
            }
        }
        const long long orow = map_out_row(P.rm, row_ok ? m : m0);
        const bool ok = mbar_wait_warp(acc_full, 0, abort_flag, status, STATUS_GEMM_EPILOGUE);
        if (ok && live) {
            tc_fence_after_sync();
            uint32_t r[COLS];
            __syncwarp();
            const uint32_t at = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + g * COLS;
            if constexpr (COLS == 8) tmem_ld_32x8(at, r);
            else tmem_ld_32x16(at, r);
            tmem_ld_wait();
            float e1[4], e2[4];
#pragma unroll
            for (int c = 0; c < COLS / 8; ++c) {
                const bool in = n0 + 8 * c < N;
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float acc = __uint_as_float(r[8 * c + i]);
                    v[i] = (EPI & EPI_LN) ? fmaf(ln_a, acc, add[8 * c + i]) : acc + add[8 * c + i];
                }
                if (EPI & EPI_GELU) gelu8(v);
                if (EPI & EPI_RES) {
                    Vec<bf16> w;
                    float rf[8];
                    w.raw = rv[c];
                    w.to_float(rf);
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] += rf[i];
                }
                if (EPI & EPI_EMIT) {
                    // as in linear_tc_kernel: columns 2 q, 2 q + 1 of each eight
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float z0 = in ? v[2 * q] : 0.f, z1 = in ? v[2 * q + 1] : 0.f;
                        const float q1 = z0 + z1, q2 = fmaf(z1, z1, __fmul_rn(z0, z0));
                        if (c == 0) { e1[q] = q1; e2[q] = q2; }
                        else { e1[q] += q1; e2[q] += q2; }
                    }
                }
                if (row_ok && in) {
                    Vec<bf16> ov;
                    ov.from_float(v);
                    ov.store(static_cast<bf16*>(P.y) + orow * P.ldy + n0 + 8 * c);
                }
            }
            if (EPI & EPI_EMIT) {
#pragma unroll
                for (int q = 0; q < 4; ++q) sums[((half * 4 + g) * 4 + q) * S::ROWS + row] = make_float2(e1[q], e2[q]);
            }
        }
        if ((EPI & EPI_EMIT) && live) {
            // the eight warps of these rows (all of them get here): eights make sixteens, these (0 + 1) + (2 + 3), the column pairs the same
            named_barrier(1 + (quarter & 1), 256);
            if (g == 0 && (BN == 128 || half == 0) && row_ok && ok && ct0 + half * 64 < N) {
                float t1[4], t2[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float2 e[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (BN == 128) {
                            e[k] = sums[((half * 4 + k) * 4 + q) * S::ROWS + row];
                        } else {
                            const float2 a = sums[((2 * k) * 4 + q) * S::ROWS + row], b = sums[((2 * k + 1) * 4 + q) * S::ROWS + row];
                            e[k] = make_float2(a.x + b.x, a.y + b.y);
                        }
                    }
                    t1[q] = (e[0].x + e[1].x) + (e[2].x + e[3].x);
                    t2[q] = (e[0].y + e[1].y) + (e[2].y + e[3].y);
                }
                P.ln.emit[(size_t)m * P.ln.slots + ct0 / SLAB + half] = make_float2((t1[0] + t1[1]) + (t1[2] + t1[3]), (t2[0] + t2[1]) + (t2[2] + t2[3]));
            }
        }
    }
    if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) { }          // let copies in flight land before releasing memory
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();     // the partner no longer reads this CTA's operands
    if (warp == PRODUCERS) tmem_dealloc_pair(tmem_base, S::TMEM_COLS);
}

// ------------------------------------------------------------------------------ host

static EncodeTiledFn g_encode = nullptr;

EncodeTiledFn encode_tiled_fn() {
    if (g_encode) return g_encode;
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess || !fn) {
        cudaGetLastError();
        return nullptr;
    }
    g_encode = reinterpret_cast<EncodeTiledFn>(fn);
    return g_encode;
}

// Encoded maps are kept per thread, direct-mapped by a hash of everything they depend on: a forward asks for the
// same few hundred maps on every call, and encoding one costs more host time than the rest of a launch's set-up.
struct TmapKey {
    const void* base;
    unsigned long long dims[5], strides[4];
    unsigned box[5];
    int rank;
};
struct TmapSlot { TmapKey key; CUtensorMap map; };
constexpr int kTmapSlots = 1024;

int make_tmap_bf16(CUtensorMap* map, const void* base, int rank, const unsigned long long* dims,
                   const unsigned long long* strides_bytes, const unsigned* box) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return fail(VTP_ERR_DRIVER, "cuTensorMapEncodeTiled is not available from this driver");
    TmapKey key;
    memset(&key, 0, sizeof(key));
    key.base = base;
    key.rank = rank;
    for (int i = 0; i < rank; ++i) { key.dims[i] = dims[i]; key.box[i] = box[i]; }
    for (int i = 0; i + 1 < rank; ++i) key.strides[i] = strides_bytes[i];
    unsigned long long h = (unsigned long long)reinterpret_cast<uintptr_t>(base) * 0x9E3779B97F4A7C15ull;
    for (int i = 0; i < rank; ++i) h = (h ^ (key.dims[i] * 31 + key.box[i])) * 0xBF58476D1CE4E5B9ull;
    static thread_local std::unique_ptr<TmapSlot[]> slots;      // freed when the thread that launches ends
    static_assert(alignof(TmapSlot) >= alignof(CUtensorMap) && __STDCPP_DEFAULT_NEW_ALIGNMENT__ < alignof(CUtensorMap),
                  "an array from operator new starts on the alignment the driver asks of a map (an aligned new)");
    if (!slots) slots.reset(new (std::nothrow) TmapSlot[kTmapSlots]());
    TmapSlot* slot = slots ? &slots[(h >> 40) % kTmapSlots] : nullptr;
    if (slot && memcmp(&slot->key, &key, sizeof(key)) == 0) {
        *map = slot->map;
        return VTP_OK;
    }
    cuuint64_t gdim[5];
    cuuint64_t gstride[5];
    cuuint32_t bdim[5];
    cuuint32_t estride[5];
    for (int i = 0; i < rank; ++i) { gdim[i] = dims[i]; bdim[i] = box[i]; estride[i] = 1; }
    for (int i = 0; i + 1 < rank; ++i) gstride[i] = strides_bytes[i];
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), gdim,
                           gstride, bdim, estride, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
        return (int)r;
    }
    if (slot) { slot->key = key; slot->map = *map; }
    return VTP_OK;
}

static int pick_bn(int N) {
    // widest tile that does not pad N more than a narrower one would
    auto padded = [&](int bn) { return ceil_div(N, bn) * bn; };
    int bn = 256;
    if (padded(192) < padded(bn)) bn = 192;
    if (padded(128) < padded(bn)) bn = 128;
    return bn;
}

int linear_stat_slots(int N) { return (int)round_up(ceil_div(N, SLAB), 2); }

static void fill_scalars(TcScalars& q, const LinearArgs& p, bool f32, int bn) {
    q.bias = p.bias; q.res = (const bf16*)p.res; q.ldr = p.ldr; q.y = p.y; q.ldy = p.ldy;
    q.m_max = p.m_max; q.m_dev = p.m_dev; q.N = p.N;
    q.n_tiles = make_fast_div((uint32_t)ceil_div(p.N, bn));
    q.use_tma_store = (!f32 && p.out_grp == 0) ? 1 : 0;
    q.rm = RowMap{p.out_grp, p.out_skip, p.res_mod, p.res_off};
    q.ln = LnFold{p.ln_stats, p.ln_s, p.ln_mode, p.ln_dim, p.ln_eps, p.emit_stats,
                  p.emit_stats ? linear_stat_slots(p.N) : p.ln_slots, ceil_div(p.ln_dim, SLAB)};
}

template <int BN, int CG>
static int fill_problem(TcMaps& t, TcScalars& q, const LinearArgs& p, bool f32) {
    fill_scalars(q, p, f32, BN);
    // W boxes: a whole tile, and 64 columns of a strip or a narrow last tile (each CTA of a group loads its share)
    if (int rc = operand_maps(&t.ta, &t.tw, p, BN / CG)) return rc;
    if (int rc = operand_maps(nullptr, &t.tws, p, SLAB / CG)) return rc;
    // Output and residual maps: 32 rows of a slab (bf16 output, rows not remapped).
    t.ty = t.tw;
    t.tr = t.tw;
    const unsigned box[2] = {SLAB, 32};
    const unsigned long long dims[2] = {(unsigned long long)p.N, (unsigned long long)p.m_max};
    if (q.use_tma_store) {
        const unsigned long long strides[1] = {(unsigned long long)p.ldy * 2ull};
        if (int rc = make_tmap_bf16(&t.ty, p.y, 2, dims, strides, box)) return rc;
    }
    if (p.res && p.res_mod <= 0) {
        const unsigned long long strides[1] = {(unsigned long long)p.ldr * 2ull};
        if (int rc = make_tmap_bf16(&t.tr, p.res, 2, dims, strides, box)) return rc;
    }
    return VTP_OK;
}

// p1 = null: one problem.  Otherwise two problems of the same K and epilogue kind in one launch.
template <int BN, int CG, int EPI, bool F32, int NPROB>
static int launch_tc(const LinearArgs& p, const LinearArgs* p1, cudaStream_t st) {
    using S = TcConf<BN, CG>;
    TcLaunch L;
    if (int rc = fill_problem<BN, CG>(L.m[0], L.s.p[0], p, F32)) return rc;
    if (NPROB == 2) {
        if (int rc = fill_problem<BN, CG>(L.m[1], L.s.p[1], *p1, F32)) return rc;
    } else {
        L.m[1] = L.m[0];
        L.s.p[1] = L.s.p[0];
    }
    auto kern = linear_tc_kernel<BN, CG, EPI, F32, NPROB>;
    static bool reserved[64] = {};   // per instantiation and device
    if (int rc = reserve_smem(kern, S::TOTAL, reserved)) return rc;
    long long tiles = (long long)ceil_div(p.N, BN) * ceil_div(p.m_max, TBM * CG);
    if (NPROB == 2) tiles += (long long)ceil_div(p1->N, BN) * ceil_div(p1->m_max, TBM * CG);
    const int groups = sm_count() / CG;
    // few tiles are cut into column strips, one per CTA group (see Schedule): launch a group for each of those
    tiles *= BN / SLAB;
    const int used = (int)(tiles < groups ? tiles : groups);
    L.s.groups = make_fast_div((uint32_t)used);
    // Every launch starts early (launch_kernel): a CTA takes an SM by itself and sets itself up while the kernel in front ends
    // (DeiT-S, 256 images: 3.35 -> 3.31 ms; DeiT-B, 33 images: 1.55 -> 1.47; PVT-small, 96 images: 2.78 -> 2.69).
    return launched(launch_kernel(kern, true, CG, dim3(CG * used), dim3(S::THREADS), (size_t)S::TOTAL, st, L, p.K, device_status_ptr()));
}

// 128 x bn tiles of a problem.  As many of 64 columns as SMs at most run as linear_tc_small_kernel: all at once, one per SM.  (DeiT-Ti, one
// image: 505 us per forward with the persistent kernel alone, 395 with both; DeiT-S, 7 images: 662 and 586.  Launches on both
// sides of the line, us, small / persistent kernel:  1536, K = 384, GELU: 96 tiles 4.6 / 6.2, 144 4.7 / 6.8, 216 8.5 / 7.0, 288
// 8.9 / 7.3;  384, K = 1536, residual: 108 tiles 7.8 / 8.9, 144 7.8 / 9.5, 222 14.7 / 11.5;  768, K = 192, GELU: 108 tiles 3.9 / 4.7,
// 144 4.1 / 4.8, 216 7.4 / 5.4.)
// Two problems in one launch also run that way as 128 x 128 tiles, if those of all of one's rows and of seven tenths of the rows that
// the other's count on the device allows are no more than SMs (q and kv of DeiT-S, 7 images: 7.0 -> 5.8 us).  Blocks, us, at a fifth /
// half / three quarters / all of the regions on the finest grain, this way and by the persistent kernel: DeiT-S, 7 images 43.2 43.7 44.4
// 45.5 and 44.0 44.5 45.0 47.4; 8 images 42.4 43.5 46.1 49.4 and 44.8 45.2 48.0 48.3; DeiT-Ti, 16 images 37.3 37.9 41.1 43.4 and 38.0
// 39.9 42.4 41.3; DeiT-B, 4 images 54.2 55.2 60.5 62.9 and 56.1 58.4 61.9 61.9; PVT stage 3, 18 images 53.7 55.8 57.9 61.7 and 54.7 57.1
// 59.9 60.2.  Up to here it gains more than it loses: with all regions on the finest grain the tiles are some more than SMs,
// and each of those waits until one is free.  Beyond the line that costs more than the rest gains: DeiT-S, 9 images 43.2 45.0 51.1
// 52.0 and 43.8 46.2 48.5 49.7; PVT stage 3, 25 images 58.0 61.2 66.3 67.3 and 58.9 61.9 64.8 65.6.
// Where the queries are most of the rows and have no more columns than a tile (PVT stage 1, 8 images 63.2 65.9 73.9 74.7 and 62.1
// 66.0 72.0 72.6) it gains nothing.  One problem gains nothing either: 1536, K = 384, 539 of 1799 rows 6.6 / 6.5, all of them 11.4 / 8.4.
static long long small_tiles(const LinearArgs& p, int bn, bool likely = false) {
    const int rows = likely && p.m_dev ? (int)((7ll * p.m_max + 9) / 10) : p.m_max;
    return (long long)ceil_div(rows, TBM) * ceil_div(p.N, bn);
}

template <int BN, int EPI, bool F32, int NPROB>
static int launch_small(const LinearArgs& p, const LinearArgs* p1, cudaStream_t st) {
    using S = SmallConf<BN>;
    SmallLaunch L;
    for (int i = 0; i < 2; ++i) {
        const LinearArgs& q = (NPROB == 2 && i) ? *p1 : p;
        if (int rc = operand_maps(&L.ta[i], &L.tw[i], q, BN)) return rc;
        fill_scalars(L.p[i], q, F32, BN);
    }
    L.grid0 = (int)small_tiles(p, BN);
    L.at_once = sm_count();
    const int grid = L.grid0 + (NPROB == 2 ? (int)small_tiles(*p1, BN) : 0);
    auto kern = linear_tc_small_kernel<BN, EPI, F32, NPROB>;
    static bool reserved[64] = {};   // per instantiation and device
    if (int rc = reserve_smem(kern, S::TOTAL, reserved)) return rc;
    return launched(launch_kernel(kern, true, 1, dim3(grid), dim3(S::THREADS), (size_t)S::TOTAL, st, L, p.K, device_status_ptr()));
}

// Which tiles of linear_tc_pair_kernel a problem takes, 0: none.  All of them run at once, a pair of SMs each: as many tiles as pairs at most.
// us, this form with 64 and with 128 columns / the forms above (rows valid of those the host has to allow for):
//   64 x 4096, 192 rows (PVT's first reduction, 3 images)    7.1         / 13.2      128 x 2048, 192 rows          5.0  5.9  /  8.0
//   320 x 1280, 192 rows                                     4.5  5.3    /  6.1      320 x 1280, 2048 rows (80)   10.0  6.2  /  6.8
//   192 x 768, 92 of 257 rows (DeiT-Ti fc2, one image)       3.9  4.7    /  4.6      384 x 1536, 92 of 257         4.8  5.8  /  6.8
//   384 x 1536, 644 of 1799 (90)                             8.0  6.6    /  8.2      768 x 3072, 92 of 257         6.6  7.8  / 11.0
//   768 x 3072, 368 of 1028 (108)                           10.1  9.7    / 12.6      768 x 3072, 920 of 2570 (252) 16.5 12.3 / 12.6
//   768 x 768, 92 of 257                                     4.0  4.8    /  4.8      768 x 768, 368 of 1028 (108)  7.2  5.5  /  5.9
//   384 x 384, 92 of 257                                     3.3  4.2    /  3.6      1536 x 384, 92 of 257 (72)    4.3  4.4  /  4.2
//   384 x 384, 644 of 1799 (90)                              6.2  4.6    /  4.5      3072 x 768, 92 of 257 (144)   7.8  5.9  /  6.0
// (In brackets the 128 x 64 tiles, where they come near the 74 pairs or exceed them.)
// Rows that a router picks (m_dev) are a third to a half of those allowed for, and a pair without any has ended early.  Where all rows are
// valid every pair stores a tile, and the forms above win earlier.  Time of this form over theirs, no router, by K and number of tiles:
//   64 columns   K = 384   45 tiles 0.97   48 0.99..1.03   56 1.05     K = 512   56 0.99   60 1.00   64 1.02   72 1.00..1.07   K = 640   72 0.98..1.02
//   128 columns  K = 768   40 0.98..1.05   54 1.08   72 1.14           K = 1024  45 0.99..1.01   51 1.00   57 1.01..1.03   72 1.06   K = 1280   72 1.02
static int long_reduction_pairs(const LinearArgs& p) {
    if (p.K % (2 * TBK) != 0) return 0;
    const long long pairs = sm_count() / 2;
    const bool routed = p.m_dev != nullptr;
    if (small_tiles(p, 64) <= (p.K >= (routed ? 512 : 640) ? pairs : routed || p.K >= 512 ? pairs * 4 / 5 : pairs * 2 / 3)) return p.K >= 384 ? 64 : 0;
    const long long most = p.K >= (routed ? 768 : 1280) ? pairs : p.K >= 1024 ? pairs * 2 / 3 : 0;
    return p.N > 64 && small_tiles(p, 128) <= most ? 128 : 0;
}

template <int BN, int EPI>
static int launch_pair(const LinearArgs& p, cudaStream_t st) {
    using S = PairConf<BN>;
    SmallLaunch L;
    if (int rc = operand_maps(nullptr, &L.tw[0], p, BN / 2)) return rc;
    const unsigned long long da[2] = {(unsigned long long)p.K, (unsigned long long)p.m_max}, sa[1] = {(unsigned long long)p.lda * 2ull};
    const unsigned ba[2] = {TBK, S::ROWS};
    if (int rc = make_tmap_bf16(&L.ta[0], p.a, 2, da, sa, ba)) return rc;
    fill_scalars(L.p[0], p, false, BN);
    L.ta[1] = L.ta[0]; L.tw[1] = L.tw[0]; L.p[1] = L.p[0];
    const int grid = 2 * (int)small_tiles(p, BN);
    L.grid0 = L.at_once = grid;          // (all of them run at once: long_reduction_pairs)
    auto kern = linear_tc_pair_kernel<BN, EPI>;
    static bool reserved[64] = {};   // per instantiation and device
    if (int rc = reserve_smem(kern, S::TOTAL, reserved)) return rc;
    return launched(launch_kernel(kern, true, 2, dim3(grid), dim3(S::THREADS), (size_t)S::TOTAL, st, L, p.K, device_status_ptr()));
}

// Two independent Linears of the same K (the q and kv projections of a block) in ONE launch: the tiles of the second problem fill
// the last, partial round of the first, and one launch's ramp and tail is saved.  Both: bf16 output, bias, no residual, no row
// remap, N a multiple of 64; one or both fold a LayerNorm (ln_mode 1: a block that reduces its keys folds only q's).
bool linear_pair_supported(const LinearArgs& a, const LinearArgs& b) {
    auto ok = [](const LinearArgs& p) {
        return p.dtype == VTP_BF16 && (p.ln_mode == 1 || (p.ln_mode == 0 && !p.ln_s)) && !p.res && !p.emit_stats && p.out_grp == 0 && p.flags == 0 &&
               p.m_max > 0 && p.N >= 64 && p.N % 64 == 0;
    };
    return ok(a) && ok(b) && a.K == b.K && a.ln_mode + b.ln_mode > 0;
}

// Whether two CTAs should share 256-row tiles (cta_group::2).  Each then loads and multiplies half of the tile's W rows, which
// pays once a tile has several k-blocks: 65792 x 768 with K = 384 48.1 -> 41.2 us, 23040 x 384 with K = 1536 37.1 -> 30.8.  With
// K = 64, or tiles of 128 columns, the pair's longer set-up costs more than that: 393216 x 64 with K = 64 19.5 -> 21.7,
// 172000 x 64 with K = 512 37.6 -> 39.6, 172000 x 512 with K = 64 42.5 -> 43.9.  From K = 128 to 256 it depends on the launch: many
// rounds of tiles gain, one or two lose (K = 192: 65792 x 576 24.6 -> 21.2, 65792 x 384 14.4 -> 14.2, 22000 x 192 6.1 -> 6.8, 22000 x
// 768 12.7 -> 13.8, 8000 x 768 8.0 -> 8.8; K = 256: 65792 x 768 36.1 -> 30.3, 65792 x 512 25.8 -> 21.7, 22000 x 1024 15.4 -> 15.8, 8000 x
// 1024 8.9 -> 9.7).  The line keeps K = 192 (DeiT-Ti) on single CTAs, and K = 128 (stage 2 of PVT, where 43000 x 512
// would go 12.4 -> 11.7 and 100000 x 256 13.5 -> 13.0); no model has K = 256 with tiles this wide.
static bool pairs_pay(int bn, int K) { return bn >= 192 && K >= 256; }

int linear_tcgen05_pair(const LinearArgs& a, const LinearArgs& b, cudaStream_t st) {
    if (int rc = linear_validate(a)) return rc;
    if (int rc = linear_validate(b)) return rc;
    if (int rc = check_tc_args(a)) return rc;
    if (int rc = check_tc_args(b)) return rc;
    VTP_REQUIRE(linear_pair_supported(a, b), VTP_ERR_UNSUPPORTED, "linear (tcgen05): these two problems cannot share a launch");
    if (small_tiles(a, 64) + small_tiles(b, 64) <= sm_count()) return launch_small<64, EPI_LN, false, 2>(a, &b, st);
    const bool narrow = pick_bn((a.m_max > b.m_max ? a : b).N) == 128;
    if ((!narrow || a.m_max == b.m_max) && small_tiles(a, 128, true) + small_tiles(b, 128, true) <= sm_count())
        return launch_small<128, EPI_LN, false, 2>(a, &b, st);
    // (narrow tiles where most of the work, the problem of more rows, has no more than 128 columns: the queries of PVT's first two stages,
    // whose keys are few; PVT-tiny, 96 images, 1470 us)
    if (narrow) return launch_tc<128, 1, EPI_LN, false, 2>(a, &b, st);
    if (pairs_pay(256, a.K)) return launch_tc<256, 2, EPI_LN, false, 2>(a, &b, st);
    return launch_tc<256, 1, EPI_LN, false, 2>(a, &b, st);
}

int linear_tcgen05(const LinearArgs& p, cudaStream_t st) {
    if (p.m_max == 0) return VTP_OK;
    if (int rc = check_tc_args(p)) return rc;
    const int bn = pick_bn(p.N);
    const bool pairs = pairs_pay(bn, p.K);
    const bool small = small_tiles(p, 64) <= sm_count();
    const bool f32 = (p.flags & VTP_FLAG_OUT_F32) != 0;
    const int epi = ((p.flags & VTP_FLAG_GELU) ? EPI_GELU : 0) | (p.ln_mode ? EPI_LN : 0) | (p.emit_stats ? EPI_EMIT : 0) |
                    (p.res ? EPI_RES : 0);
    // rare kinds in one tile width (a row's bits do not depend on it)
    if (f32) {
        if (small && epi == 0) return launch_small<64, 0, true, 1>(p, nullptr, st);
        if (small && epi == EPI_RES) return launch_small<64, EPI_RES, true, 1>(p, nullptr, st);
        if (epi == 0) return launch_tc<128, 1, 0, true, 1>(p, nullptr, st);
        if (epi == EPI_RES) return launch_tc<128, 1, EPI_RES, true, 1>(p, nullptr, st);
        return fail(VTP_ERR_UNSUPPORTED, "linear (tcgen05): fp32 output supports bias and residual only");
    }
    const int pair_bn = long_reduction_pairs(p);
    if (pair_bn) {
#define VTP_PAIR_CASE(E) if (epi == (E)) return pair_bn == 64 ? launch_pair<64, (E)>(p, st) : launch_pair<128, (E)>(p, st);
        VTP_PAIR_CASE(0)
        VTP_PAIR_CASE(EPI_GELU)
        VTP_PAIR_CASE(EPI_RES)
        VTP_PAIR_CASE(EPI_LN)
        VTP_PAIR_CASE(EPI_LN | EPI_GELU)
        VTP_PAIR_CASE(EPI_EMIT | EPI_RES)
#undef VTP_PAIR_CASE
    }
    if (small && epi == (EPI_GELU | EPI_RES)) return launch_small<64, EPI_GELU | EPI_RES, false, 1>(p, nullptr, st);
    if (epi == (EPI_GELU | EPI_RES)) return launch_tc<128, 1, EPI_GELU | EPI_RES, false, 1>(p, nullptr, st);
#define VTP_TC_CASE(E)                                                                   \
    if (epi == (E)) {                                                                    \
        if (small) return launch_small<64, (E), false, 1>(p, nullptr, st);               \
        if (pairs && bn == 256) return launch_tc<256, 2, (E), false, 1>(p, nullptr, st); \
        if (pairs && bn == 192) return launch_tc<192, 2, (E), false, 1>(p, nullptr, st); \
        if (bn == 256) return launch_tc<256, 1, (E), false, 1>(p, nullptr, st);          \
        if (bn == 192) return launch_tc<192, 1, (E), false, 1>(p, nullptr, st);          \
        return launch_tc<128, 1, (E), false, 1>(p, nullptr, st);                         \
    }
    VTP_TC_CASE(0)
    VTP_TC_CASE(EPI_GELU)
    VTP_TC_CASE(EPI_RES)
    VTP_TC_CASE(EPI_LN)
    VTP_TC_CASE(EPI_LN | EPI_GELU)
    VTP_TC_CASE(EPI_EMIT | EPI_RES)
#undef VTP_TC_CASE
    return fail(VTP_ERR_UNSUPPORTED, "linear (tcgen05): epilogue combination %d is not instantiated", epi);
}

}  // namespace vtp
