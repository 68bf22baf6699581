// Variable-length-query attention on tcgen05 tensor cores (bf16 in, fp32 accumulate).
//
// Work item = 128 packed queries of one (image, head).  Persistent CTAs (two per SM) walk
// the items with a fixed stride; the item list is derived on the device from the per-image
// offsets, so images with few queries cost nothing and nothing is read back to the host.
// Keys are split into a tensor-core part (the largest multiple of 16, walked in chunks of
// up to 256 keys) and a tail of at most 15 keys done on CUDA cores: token grids with one
// cls token have 16k+1 keys, so 257 keys are ONE 256-key chunk plus one tail key.
//   S = Q K_c^T        tcgen05.mma, A = Q tile, B = K chunk, both K-major from TMA (128B
//                      swizzle); accumulator S in TMEM columns [0, KC)
//   P = exp2(scale*log2e*(S - rowmax))   four softmax warps, one thread per query row: read S
//                      with tcgen05.ld, write bf16 P back into TMEM over the S columns
//                      already consumed (the first 128 keys to columns [0, 64), the others from 128 on)
//   O_c = P V_c        tcgen05.mma with A = P from TMEM and B = V chunk as an MN-major operand
//                      straight from the TMA image of the [keys, d] rows; accumulator in TMEM
//                      columns [64, 128), which are free once the first 128 keys are consumed: their
//                      products run while the exp2 of the rest does (DeiT-Ti, one image: 526 -> 522 us;
//                      from 7 images on the gain is within the 1 % that two runs differ by)
//   O  = O*alpha + O_c in registers of the softmax threads (online-softmax rescale), then the
//                      tail keys, the 1/rowsum and the bf16 store.
// Warp 0 issues TMA (Q is double-buffered so the next item's Q and K stream in during
// the current softmax), warp 1 issues MMA, warps 2-5 do softmax and output.
// q, k, v are read in place from the Linear outputs through strided tensor maps.
// Every mbarrier wait is bounded (sm100.cuh).
//
// An item (128 queries, 257 keys) is a chain of scores, maximum, exp2, P V and output: 1400 + 1500 + 5300 + 1500 + 3000 cycles
// (clock64) with two items on the SM, hardly less alone.  Two threads a row (eight softmax warps) measured 68 us where this
// takes 59 (256 images x 6 heads) and 73 where it takes 56 (1025 keys).  What a chunk costs beside the sweeps: one arrival per warp
// instead of one per thread, loads and MMAs from an elected thread, offsets kept in shared memory and scanned a run of images per
// lane: DeiT-S at 512 px 1830 -> 1770 us, 256 images 3384 -> 3357, DeiT-Ti with one image 396 -> 392.
//
// Replaces batched_sparse_attention_forward
// (vtpack/layers/csrc/batched_sparse_gemm/batched_sparse_gemm.cu:219-305: per image two
// cuBLAS strided-batched GEMMs around a cuDNN softmax, scores round-tripping through HBM).
#include "attention.h"
#include "attention_items.cuh"
#include "runtime.h"
#include "sm100.cuh"

namespace vtp {

using namespace sm100;

constexpr int KC_MAX = 256;        // keys per tensor-core chunk, upper bound
constexpr int O_COL = 64;          // TMEM column of the P*V accumulator
constexpr int P_SPLIT = 128;       // keys of a chunk's first part of P, in columns [0, 64); the rest of P from column 128 on
constexpr int ATT_TMEM_COLS = 256;
constexpr int SOFTMAX_WARPS = 4;
constexpr int OFFSETS_KEPT = 512;  // images whose offsets are copied to shared memory beside the tile prefix

constexpr int SM_Q = 0;                               // two Q buffers
constexpr int SM_K = SM_Q + 2 * QT * HD * 2;          // 32768
constexpr int SM_V = SM_K + KC_MAX * HD * 2;          // 65536
constexpr int SM_BAR = SM_V + KC_MAX * HD * 2;        // 98304
constexpr int SM_ITEM = SM_BAR + 256;                 // two work items (one per Q buffer), written by the producer
constexpr int SM_TAIL = SM_ITEM + 256;                // per Q buffer: up to 15 tail K rows, then 15 tail V rows
constexpr int TAIL_ROWS = 15;
constexpr int SM_PREFIX = SM_TAIL + 2 * 2 * TAIL_ROWS * HD * 2;   // int32 [B + 1] tile prefix

// 2^x on the special-function unit; arguments here are <= 0 (or -inf, giving 0).
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Plain bulk copy global -> shared of `bytes` (a multiple of 16, both ends 16-byte aligned), counted on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

template <int PER>
__global__ void __launch_bounds__(192, 2)
attn_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
               const __grid_constant__ CUtensorMap tmap_v, const bf16* __restrict__ kptr,
               const bf16* __restrict__ vptr, long long q_hs, long long kv_bs, long long kv_rs, long long kv_hs,
               bf16* __restrict__ out, long long o_rs, long long o_hs, int B, int heads, int n_keys, int KC,
               int n_chunks, const int32_t* __restrict__ offsets, int l_max, int max_q, float scale_log2e,
               int* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + SM_BAR);
    uint64_t* q_full = bars + 0;    // [2]
    uint64_t* q_free = bars + 2;    // [2]
    uint64_t* k_full = bars + 4;
    uint64_t* k_free = bars + 5;
    uint64_t* v_full = bars + 6;
    uint64_t* v_free = bars + 7;
    uint64_t* s_full = bars + 8;
    uint64_t* p_full = bars + 9;
    uint64_t* o_full = bars + 10;
    uint64_t* o_free = bars + 11;
    uint64_t* p_half = bars + 12;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* void_s = reinterpret_cast<int*>(tmem_slot + 2);
    int* tile_prefix = reinterpret_cast<int*>(base + SM_PREFIX);
    int32_t* offs_s = tile_prefix + B + 1;
    AttnItem* items = reinterpret_cast<AttnItem*>(base + SM_ITEM);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (warp == 1 && elect_one()) {
        for (int i = 0; i < 2; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_free[i], SOFTMAX_WARPS); }
        mbar_init(k_full, 1); mbar_init(k_free, 1);
        mbar_init(v_full, 1); mbar_init(v_free, 1);
        mbar_init(s_full, 1); mbar_init(p_full, SOFTMAX_WARPS); mbar_init(p_half, SOFTMAX_WARPS);
        mbar_init(o_full, 1); mbar_init(o_free, SOFTMAX_WARPS);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmap_q);
        prefetch_tmap(&tmap_k);
        prefetch_tmap(&tmap_v);
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, ATT_TMEM_COLS);
        tmem_relinquish();
    }
    const int n_main = (n_keys / 16) * 16;          // keys handled by the tensor cores
    const int tail = n_keys - n_main;               // 0..15 keys handled on CUDA cores
    const uint32_t kv_bytes = (uint32_t)KC * HD * 2;
    // Loads of one thread of warp 0: an item, its Q tile and the K and V rows of the tail keys all arrive on q_full
    auto load_q = [&](const AttnItem& it, int qb) {
        items[qb] = it;
        mbar_arrive_expect_tx(&q_full[qb], QT * HD * 2 + 2 * tail * HD * 2);
        tma_load_2d(base + SM_Q + qb * (QT * HD * 2), &tmap_q, &q_full[qb], (int)(it.h * q_hs), it.row0);
        for (int t = 0; t < tail; ++t) {
            const size_t koff = (size_t)it.b * kv_bs + (size_t)(n_main + t) * kv_rs + (size_t)it.h * kv_hs;
            uint8_t* tb = base + SM_TAIL + qb * (2 * TAIL_ROWS * HD * 2) + t * (HD * 2);
            bulk_load(tb, kptr + koff, HD * 2, &q_full[qb]);
            bulk_load(tb + TAIL_ROWS * HD * 2, vptr + koff, HD * 2, &q_full[qb]);
        }
    };
    auto load_k = [&](const AttnItem& it, int c) {
        mbar_arrive_expect_tx(k_full, kv_bytes);
        tma_load_3d(base + SM_K, &tmap_k, k_full, (int)(it.h * kv_hs), c * KC, it.b);
    };
    auto load_v = [&](const AttnItem& it, int c) {
        mbar_arrive_expect_tx(v_full, kv_bytes);
        tma_load_3d(base + SM_V, &tmap_v, v_full, (int)(it.h * kv_hs), c * KC, it.b);
    };
    __syncthreads();                                // (the barriers exist)
    // Nothing above depends on the kernel in front of this one on the stream; the packed-row
    // offsets, q, k and v below do.
    pdl_begin();
    // The items.  Of up to 256 images warp 0 lists them alone and sends for the first one's operands before the others know the list
    // (all threads listing them first / this): DeiT-Ti, one image, 8.3 / 7.9 us a launch, DeiT-S, 7 images, 10.1 / 9.3; the forward of
    // PVT-tiny, 48 images, 986 / 975 us, DeiT-Ti, 96 images, 1015 / 1011, 200 images, 1679 / 1657.
    const bool few = PER == 1 || B <= FEW_IMAGES, keep = B <= OFFSETS_KEPT;
    FewImages<PER> images;
    if (few && warp == 0) images.load(offsets, B);
    if (threadIdx.x == (few ? 0 : blockDim.x - 1)) *void_s = launch_is_void(status) ? 1 : 0;
    AttnItem first_item;
    if (!few) {
        list_tiles(offsets, B, max_q, l_max, status, tile_prefix, keep ? offs_s : nullptr);
    } else if (warp == 0) {
        __syncwarp();
        const int n_tiles = images.list(B, max_q, l_max, status, tile_prefix, offs_s, blockIdx.x, heads, first_item);
        if (*void_s == 0 && (int)blockIdx.x < n_tiles * heads && elect_one()) {
            load_q(first_item, 0);
            load_k(first_item, 0);
            load_v(first_item, 0);
        }
        __syncwarp();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const int n_work = *void_s ? 0 : tile_prefix[B] * heads;

    if (warp == 0) {
        if (elect_one()) {
            // ------------------------------------------------------------ TMA producer
            const int32_t* offs = keep ? offs_s : offsets;
            int li = 0, g = 0;
            bool ok = true;
            for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++li) {
                const bool sent = few && li == 0;              // (its Q and first chunk are under way)
                const AttnItem it = sent ? first_item : attn_item(w, heads, B, tile_prefix, offs);
                const int qb = li & 1;
                if (!sent) {
                    ok = mbar_wait(&q_free[qb], ((li >> 1) & 1) ^ 1, abort_flag, status, STATUS_ATTN_LOAD);
                    if (!ok) break;
                    load_q(it, qb);
                }
                for (int c = 0; c < n_chunks; ++c, ++g) {
                    if (sent && c == 0) continue;
                    const uint32_t ph = g & 1;
                    ok = mbar_wait(k_free, ph ^ 1, abort_flag, status, STATUS_ATTN_LOAD);
                    if (!ok) break;
                    load_k(it, c);
                    ok = mbar_wait(v_free, ph ^ 1, abort_flag, status, STATUS_ATTN_LOAD);
                    if (!ok) break;
                    load_v(it, c);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            // -------------------------------------------------------------- MMA issuer
            const uint32_t idesc_s = idesc_bf16_f32(QT, KC, 0, 0);
            const uint32_t idesc_o = idesc_bf16_f32(QT, HD, 0, 1);     // B = V, MN-major
            const uint64_t kdesc = smem_desc_sw128(smem_u32(base + SM_K));
            const uint64_t vdesc = smem_desc_sw128(smem_u32(base + SM_V));
            int li = 0, g = 0;
            bool ok = true;
            for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++li) {
                const int qb = li & 1;
                const uint64_t qdesc = smem_desc_sw128(smem_u32(base + SM_Q + qb * (QT * HD * 2)));
                ok = mbar_wait(&q_full[qb], (li >> 1) & 1, abort_flag, status, STATUS_ATTN_MMA);
                for (int c = 0; c < n_chunks && ok; ++c, ++g) {
                    const uint32_t ph = g & 1;
                    // S columns double as the P and O columns of the previous chunk: wait until
                    // the softmax threads have taken O out
                    ok = mbar_wait(k_full, ph, abort_flag, status, STATUS_ATTN_MMA) &&
                         mbar_wait(o_free, ph ^ 1, abort_flag, status, STATUS_ATTN_MMA);
                    if (!ok) break;
                    tc_fence_after_sync();
#pragma unroll
                    for (int k = 0; k < HD / 16; ++k)
                        umma_ss(tmem_base, qdesc + 2 * k, kdesc + 2 * k, idesc_s, k != 0 ? 1u : 0u);
                    umma_commit(s_full);
                    umma_commit(k_free);
                    ok = mbar_wait(p_half, ph, abort_flag, status, STATUS_ATTN_MMA) &&
                         mbar_wait(v_full, ph, abort_flag, status, STATUS_ATTN_MMA);
                    if (!ok) break;
                    tc_fence_after_sync();
                    const int ksteps = KC / 16;
                    for (int t = 0; t < ksteps; ++t) {
                        if (t == P_SPLIT / 16) {
                            ok = mbar_wait(p_full, ph, abort_flag, status, STATUS_ATTN_MMA);
                            if (!ok) break;
                            tc_fence_after_sync();
                        }
                        // P: 16 keys = 8 TMEM columns of bf16 pairs.  V: 16 keys = 16 rows of 128 bytes.
                        umma_ts(tmem_base + O_COL, tmem_base + 8 * t + (t < P_SPLIT / 16 ? 0 : 64),
                                vdesc + (uint64_t)(t * (16 * 128 >> 4)), idesc_o, t != 0 ? 1u : 0u);
                    }
                    if (!ok) break;
                    umma_commit(o_full);
                    umma_commit(v_free);
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------- softmax + output warps
        const int r = (warp & 3) * 32 + lane;                     // query row = TMEM lane
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        auto arrive = [&](uint64_t* bar) {
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        int li = 0, g = 0;
        bool ok = true;
        for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++li) {
            const int qb = li & 1;
            // the producer worked out which (image, head, rows) this item is; it arrives with the Q tile
            ok = mbar_wait_warp(&q_full[qb], (li >> 1) & 1, abort_flag, status, STATUS_ATTN_SOFTMAX);
            if (!ok) break;
            const AttnItem it = items[qb];
            // a warp whose 32 rows all lie beyond the item's queries only keeps the barriers moving: its rows
            // of P and O are never stored, so what the tensor core computes for them does not matter, and
            // the special-function unit and the issue slots go to the warps that have rows to compute
            const bool live = (warp & 3) * 32 < it.nq;
            float m = -INFINITY, l = 0.f;
            float o[HD];
#pragma unroll
            for (int i = 0; i < HD; ++i) o[i] = 0.f;
            const uint8_t* qrow = base + SM_Q + qb * (QT * HD * 2) + r * 128;
            // ---- the last n_keys % 16 keys run on CUDA cores.  Their scores (one fmaf chain in channel order each) are
            // formed here: the rows arrived with Q, and the scores of the chunk are still being loaded and multiplied
            // (behind the chunk: DeiT-Ti, one image, 529 instead of 521 us; DeiT-S, 7 images, 687 instead of 680 us).
            const uint8_t* tb = base + SM_TAIL + qb * (2 * TAIL_ROWS * HD * 2);
            float tail_s[TAIL_ROWS];
            if (live) {
#pragma unroll 1
                for (int t = 0; t < tail; ++t) {
                    const uint4* krow = reinterpret_cast<const uint4*>(tb + t * (HD * 2));
                    float sdot = 0.f;
#pragma unroll
                    for (int ch = 0; ch < HD / 8; ++ch) {
                        Vec<bf16> qv, kv;
                        float qf[8], kf[8];
                        qv.raw = *reinterpret_cast<const uint4*>(qrow + ((ch ^ (r & 7)) << 4));
                        kv.raw = krow[ch];
                        qv.to_float(qf);
                        kv.to_float(kf);
#pragma unroll
                        for (int i = 0; i < 8; ++i) sdot = fmaf(qf[i], kf[i], sdot);
                    }
                    tail_s[t] = sdot;
                }
            }
            for (int c = 0; c < n_chunks && ok; ++c, ++g) {
                const uint32_t ph = g & 1;
                ok = mbar_wait_warp(s_full, ph, abort_flag, status, STATUS_ATTN_SOFTMAX);
                if (!ok) break;
                tc_fence_after_sync();
                if (!live) {
                    arrive(p_half);
                    arrive(p_full);
                    ok = mbar_wait_warp(o_full, ph, abort_flag, status, STATUS_ATTN_SOFTMAX);
                    if (!ok) break;
                    arrive(o_free);
                    continue;
                }
                const int n_valid = min(KC, n_main - c * KC);
                const bool full = n_valid == KC && (KC & 31) == 0;     // no column needs masking
                // Two sweeps over the S columns, 32 at a time: row maximum, then exp2 + P.  The
                // TMEM load of the next block is always in flight while the current one is used.
                const int nblk = (KC + 31) >> 5;
                uint32_t s[32];
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                __syncwarp();
                tmem_ld_32x32(lane_base, s);
                for (int blk = 0; blk < nblk; ++blk) {
                    tmem_ld_wait();
                    float f[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(s[i]);
                    __syncwarp();
                    tmem_ld_32x32(lane_base + (blk + 1 < nblk ? (blk + 1) * 32 : 0), s);   // wraps to sweep 2
                    const int c0 = blk * 32;
                    if (full) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], f[i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (c0 + i < n_valid) mx4[i & 3] = fmaxf(mx4[i & 3], f[i]);
                    }
                }
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                const float m_new = fmaxf(m, mx);
                const float m_at = m_new == -INFINITY ? 0.f : m_new;            // (scores of -inf have weight zero)
                const float alpha = fast_exp2((m - m_at) * scale_log2e);        // 0 while m is -inf
                const float mb = m_at * scale_log2e;
                float ls4[4] = {0.f, 0.f, 0.f, 0.f};
                for (int blk = 0; blk < nblk; ++blk) {
                    tmem_ld_wait();
                    float f[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(s[i]);
                    if (blk + 1 < nblk) {
                        __syncwarp();
                        tmem_ld_32x32(lane_base + (blk + 1) * 32, s);
                    }
                    const int c0 = blk * 32;
                    uint32_t pk[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float p0 = fast_exp2(fmaf(f[2 * i], scale_log2e, -mb));
                        float p1 = fast_exp2(fmaf(f[2 * i + 1], scale_log2e, -mb));
                        if (!full) {
                            p0 = (c0 + 2 * i < n_valid) ? p0 : 0.f;
                            p1 = (c0 + 2 * i + 1 < n_valid) ? p1 : 0.f;
                        }
                        ls4[i & 3] += p0 + p1;
                        const __nv_bfloat162 h2 = __floats2bfloat162_rn(p0, p1);   // low half = even key
                        pk[i] = *reinterpret_cast<const uint32_t*>(&h2);
                    }
                    __syncwarp();
                    // over S columns already consumed; the accumulator takes columns [64, 128) once the first part is full
                    tmem_st_32x16(lane_base + (c0 >> 1) + (c0 < P_SPLIT ? 0 : 64), pk);
                    if (c0 + 32 == P_SPLIT || (blk + 1 == nblk && c0 < P_SPLIT)) {
                        tmem_st_wait();
                        tc_fence_before_sync();
                        arrive(p_half);
                    }
                }
                const float lsum = (ls4[0] + ls4[1]) + (ls4[2] + ls4[3]);
                tmem_st_wait();
                tc_fence_before_sync();
                arrive(p_full);
                l = l * alpha + lsum;
                m = m_new;
                ok = mbar_wait_warp(o_full, ph, abort_flag, status, STATUS_ATTN_SOFTMAX);
                if (!ok) break;
                tc_fence_after_sync();
#pragma unroll
                for (int c0 = 0; c0 < HD; c0 += 32) {
                    uint32_t t[32];
                    __syncwarp();
                    tmem_ld_32x32(lane_base + O_COL + c0, t);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[c0 + i] = fmaf(o[c0 + i], alpha, __uint_as_float(t[i]));
                }
                tc_fence_before_sync();
                arrive(o_free);
            }
            if (!ok) break;
            if (!live) {
                arrive(&q_free[qb]);
                continue;
            }
            // ---- one online-softmax step per tail key, behind the chunks: a row's terms are added in the order of its keys
#pragma unroll 1
            for (int t = 0; t < tail; ++t) {
                const uint4* vrow = reinterpret_cast<const uint4*>(tb + (TAIL_ROWS + t) * (HD * 2));
                const float sdot = tail_s[t];
                const float m_new = fmaxf(m, sdot);
                const float m_at = m_new == -INFINITY ? 0.f : m_new;
                const float alpha = fast_exp2((m - m_at) * scale_log2e);
                const float p = fast_exp2((sdot - m_at) * scale_log2e);
                l = l * alpha + p;
                m = m_new;
#pragma unroll
                for (int ch = 0; ch < HD / 8; ++ch) {
                    Vec<bf16> vv;
                    float vf[8];
                    vv.raw = vrow[ch];
                    vv.to_float(vf);
#pragma unroll
                    for (int i = 0; i < 8; ++i) o[8 * ch + i] = fmaf(o[8 * ch + i], alpha, p * vf[i]);
                }
            }
            // ---- normalise, then out through the warp's own 32 rows of the Q tile (no longer needed) so that
            // eight lanes write one full 128-byte line of a row instead of every lane a piece of its own row
            {
                const float inv = 1.0f / l;
                __syncwarp();                                   // every lane has read its Q row (tail scores)
                uint8_t* my = const_cast<uint8_t*>(qrow);
#pragma unroll
                for (int ch = 0; ch < HD / 8; ++ch) {
                    float v8[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) v8[i] = o[8 * ch + i] * inv;
                    Vec<bf16> ov;
                    ov.from_float(v8);
                    *reinterpret_cast<uint4*>(my + ((ch ^ (r & 7)) << 4)) = ov.raw;
                }
                __syncwarp();
                const uint8_t* wq = base + SM_Q + qb * (QT * HD * 2) + (warp & 3) * 32 * 128;
                const int ch = lane & 7;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int rr = i * 4 + (lane >> 3);          // row within the warp's 32
                    const int row = (warp & 3) * 32 + rr;
                    const uint4 v = *reinterpret_cast<const uint4*>(wq + rr * 128 + ((ch ^ (rr & 7)) << 4));
                    if (row < it.nq && it.row0 + row < l_max)
                        *reinterpret_cast<uint4*>(out + (size_t)(it.row0 + row) * o_rs + it.h * o_hs + ch * 8) = v;
                }
                __syncwarp();
                fence_proxy_async_smem();                       // the next Q tile is written by TMA
            }
            arrive(&q_free[qb]);
        }
    }
    if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) { }     // let copies in flight land before releasing memory
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, ATT_TMEM_COLS);
}

constexpr int MOST_IMAGES = 16384, SM_MOST = SM_PREFIX + (MOST_IMAGES + 1) * 4 + 1024;
static_assert(SM_MOST <= 232448, "shared memory budget");
int attention_tcgen05_max_images() { return MOST_IMAGES; }

int attention_tcgen05(const AttnArgs& p, cudaStream_t st) {
    VTP_REQUIRE(p.dtype == VTP_BF16, VTP_ERR_DTYPE, "attention (tcgen05): bf16 only");
    VTP_REQUIRE(p.head_dim == HD, VTP_ERR_UNSUPPORTED, "attention (tcgen05): head_dim %d (only %d)", p.head_dim, HD);
    VTP_REQUIRE(p.n_keys >= 16, VTP_ERR_UNSUPPORTED, "attention (tcgen05): needs at least 16 keys, got %d", p.n_keys);
    VTP_REQUIRE(p.B <= MOST_IMAGES, VTP_ERR_SHAPE, "attention (tcgen05): %d images (at most %d)", p.B, MOST_IMAGES);
    VTP_REQUIRE(p.q_rs % 8 == 0 && p.q_hs % 8 == 0 && p.kv_rs % 8 == 0 && p.kv_hs % 8 == 0 && p.kv_bs % 8 == 0 &&
                    p.o_rs % 8 == 0 && p.o_hs % 8 == 0,
                VTP_ERR_ALIGN, "attention (tcgen05): strides must be multiples of 16 bytes");
    VTP_REQUIRE(aligned16(p.q) && aligned16(p.k) && aligned16(p.v) && aligned16(p.out), VTP_ERR_ALIGN,
                "attention (tcgen05): pointers must be 16-byte aligned");
    const int n_main = (p.n_keys / 16) * 16;
    const int n_chunks = ceil_div(n_main, KC_MAX);
    const int KC = (int)round_up(ceil_div(n_main, n_chunks), 16);
    CUtensorMap tq, tk, tv;
    {
        const unsigned long long dims[2] = {(unsigned long long)((p.heads - 1) * p.q_hs + HD),
                                            (unsigned long long)p.l_max};
        const unsigned long long strides[1] = {(unsigned long long)p.q_rs * 2ull};
        const unsigned box[2] = {HD, QT};
        if (int rc = make_tmap_bf16(&tq, p.q, 2, dims, strides, box)) return rc;
    }
    {
        const unsigned long long dims[3] = {(unsigned long long)((p.heads - 1) * p.kv_hs + HD),
                                            (unsigned long long)p.n_keys, (unsigned long long)p.B};
        const unsigned long long strides[2] = {(unsigned long long)p.kv_rs * 2ull, (unsigned long long)p.kv_bs * 2ull};
        const unsigned box[3] = {HD, (unsigned)KC, 1};
        if (int rc = make_tmap_bf16(&tk, p.k, 3, dims, strides, box)) return rc;
        if (int rc = make_tmap_bf16(&tv, p.v, 3, dims, strides, box)) return rc;
    }
    const int smem = SM_PREFIX + (p.B + 1) * 4 * (p.B <= OFFSETS_KEPT ? 2 : 1) + 1024;
    // (batches of up to 32 images have a kernel of their own, whose code a small launch is through sooner: FewImages)
    const bool one_each = p.B <= 32;
    auto kern = one_each ? attn_tc_kernel<1> : attn_tc_kernel<FEW_PER>;
    // (what the largest launch takes, whatever this one does: two threads may get here with different batches)
    static bool reserved[2][64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !reserved[one_each][dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_MOST);
        if (e != cudaSuccess) {
            set_error("attention (tcgen05): cannot reserve %d bytes of shared memory: %s", SM_MOST, cudaGetErrorString(e));
            return (int)e;
        }
        if (dev >= 0 && dev < 64) reserved[one_each][dev] = true;
    }
    const long long worst = (long long)p.B * ceil_div(p.max_q, QT) * p.heads;
    const int grid = (int)(worst < 2ll * sm_count() ? worst : 2ll * sm_count());
    const cudaError_t le = launch_kernel(kern, worst <= sm_count(), 1, dim3(grid), dim3(192), (size_t)smem, st, tq, tk, tv,
                                      (const bf16*)p.k, (const bf16*)p.v, p.q_hs, p.kv_bs, p.kv_rs, p.kv_hs, (bf16*)p.out,
                                      p.o_rs, p.o_hs, p.B, p.heads, p.n_keys, KC, n_chunks, p.offsets, p.l_max, p.max_q,
                                      p.scale * 1.4426950408889634f, device_status_ptr());
    if (le != cudaSuccess) {
        cudaGetLastError();
        set_error("attention (tcgen05): %s", cudaGetErrorString(le));
        return (int)le;
    }
    return check_launch("attention (tcgen05)");
}

}  // namespace vtp
