// Variable-length-query attention of fp32 blocks on tcgen05 tensor cores, operands as terms (f32_terms.cuh).
//
// The products are formed like those of the fp32 Linears: six bf16 products of terms, smallest first, into a fresh TMEM
// accumulator per 64 channels (scores) or 64 keys (P V), which fp32 registers add up; the softmax is fp32 with expf.  A row with a
// score or an output that is not finite is worked out again from the decoded operands (redo_rows).
//
// Work item = 128 packed queries of one (image, head) (attention_items.cuh); persistent, one CTA per SM; keys in chunks of up to
// 320, five blocks of 64:
//   warp 0      (one lane) TMA: the three terms of Q, and of K and V in slots of 128 keys
//   warp 1      (one lane) MMA: S = Q K^T into TMEM columns [0, 320); per block O_i = P_i V_i into [384, 448) or [448, 512)
//   8 warps     two per TMEM lane quarter, a thread per query row and half of every block's keys: maximum over the chunk, then
//               p = expf(s - max), split into terms and written back to TMEM, h and m over the scores the thread has just read, l to
//               [320, 384); adds the O_i of its half of the channels
//
// What bounds it: an item is a chain of loads (2800 cycles), scores (4300 for 257 keys), maximum, exponentials and splits (22
// instructions a score, 7000 with P V beside them) and output.
// Replaces batched_sparse_attention_forward (vtpack/layers/csrc/batched_sparse_gemm/batched_sparse_gemm.cu:219-305) in fp32 blocks.
#include "attention.h"
#include "attention_items.cuh"
#include "f32_terms.cuh"
#include "runtime.h"
#include "sm100.cuh"

namespace vtp {

using namespace sm100;

constexpr int AF_BLOCKS = 5;                             // 64-key blocks of a chunk at most
constexpr int AF_SLOT_KEYS = 128, AF_SLOTS = 3;
constexpr int AF_PLANE = 128 * HD * 2;                   // one term of 128 rows
constexpr int AF_WARPS = 8, AF_FIRST = 2, AF_THREADS = (AF_FIRST + AF_WARPS) * 32;
constexpr int AF_PL = 320, AF_O = 384;                   // TMEM columns: low terms of P (two blocks), O (two blocks)
constexpr int AF_SM_KV = 3 * AF_PLANE;
constexpr int AF_SM_BAR = AF_SM_KV + AF_SLOTS * 3 * AF_PLANE;
constexpr int AF_SM_ITEM = AF_SM_BAR + 256;              // two items
constexpr int AF_SM_ROW = AF_SM_ITEM + 64;               // float [2][2 halves][128 rows], exchanged between the two threads of a row
constexpr int AF_SM_PREFIX = AF_SM_ROW + 2048;           // int32 [B + 1] tile prefix, [B + 1] offsets
constexpr int AF_MOST_IMAGES = 4000;
constexpr int AF_SM_MOST = AF_SM_PREFIX + 2 * (AF_MOST_IMAGES + 1) * 4 + 1024;
static_assert(AF_SM_MOST <= 232448, "shared memory budget");

struct AfArgs {
    const bf16* q; const bf16* kv; float* out;           // q [l_max][3][C], kv [B n_keys][3][2 C], out [l_max][3][C] terms
    int B, heads, C, n_keys, n_blocks, n_chunks, l_max, max_q;
    const int32_t* offsets; float scale;
};

// 32 channels from d0 on of a query row per lane, as chains of fused multiply-adds over the decoded operands; `put`: whether the lane
// stores its row (the others come along, with a row that exists).  A key and its value are decoded once, two channels and
// one a lane, and go round by shuffles.  (A DeiT-S block, 12 images, with a NaN among the biases of v, us: 1360; each lane decoding all of
// the keys 4000; the CUDA-core attention and fp32 Linears 3200.)
__device__ __noinline__ void redo_rows(const AfArgs& g, int b, int h, long long row, int d0, int lane, bool put) {
    const bf16* k = g.kv + (long long)b * g.n_keys * 6 * g.C + h * HD;
    const bf16* v = k + g.C + d0;
    float q[HD];
    {
        const bf16* at = g.q + row * 3 * g.C + h * HD;
#pragma unroll
        for (int d = 0; d < HD; d += 8) {
            float x[8];
            join8(at + d, g.C, x);
#pragma unroll
            for (int i = 0; i < 8; ++i) q[d + i] = x[i];
        }
    }
    auto score = [&](int key) {
        const bf16* kr = k + (long long)key * 6 * g.C + 2 * lane;
        uint32_t t[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) t[i] = __ldg(reinterpret_cast<const uint32_t*>(kr + (size_t)i * 2 * g.C));
        const float y[2] = {join_terms(t[0] & 0xFFFFu, t[1] & 0xFFFFu, t[2] & 0xFFFFu), join_terms(t[0] >> 16, t[1] >> 16, t[2] >> 16)};
        float s = 0.f;
#pragma unroll
        for (int d = 0; d < HD; ++d) s = fmaf(q[d], __shfl_sync(0xffffffffu, y[d & 1], d >> 1), s);
        return s * g.scale;
    };
    float m = -INFINITY, l = 0.f, o[32];
#pragma unroll 1
    for (int key = 0; key < g.n_keys; ++key) m = fmaxf(m, score(key));
    const float m_at = m == -INFINITY ? 0.f : m;
#pragma unroll
    for (int i = 0; i < 32; ++i) o[i] = 0.f;
#pragma unroll 1
    for (int key = 0; key < g.n_keys; ++key) {
        const float p = expf(score(key) - m_at);
        l += p;
        const unsigned short* vr = reinterpret_cast<const unsigned short*>(v + (long long)key * 6 * g.C) + lane;
        const float x = join_terms(__ldg(vr), __ldg(vr + 2 * g.C), __ldg(vr + 4 * (size_t)g.C));
#pragma unroll
        for (int c = 0; c < 32; ++c) o[c] = fmaf(p, __shfl_sync(0xffffffffu, x, c), o[c]);
    }
    if (!put) return;
    const float inv = 1.f / l;
    bf16* dst = reinterpret_cast<bf16*>(g.out) + row * 3 * g.C + h * HD + d0;
#pragma unroll
    for (int c = 0; c < 32; c += 4) {
        const float r[4] = {o[c] * inv, o[c + 1] * inv, o[c + 2] * inv, o[c + 3] * inv};
        store_terms4(dst + c, (size_t)g.C, r);
    }
}

template <bool V> struct Masked { static constexpr bool value = V; };

template <int PER>
__global__ void __launch_bounds__(AF_THREADS, 1)
attn_f32_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kv,
                   const __grid_constant__ AfArgs g, int* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + AF_SM_BAR);
    uint64_t* q_full = bars;           // the item is known and its Q has landed
    uint64_t* q_free = bars + 1;       // its scores are formed and the softmax warps know the item
    uint64_t* kv_full = bars + 2;      // [3] per slot
    uint64_t* kv_free = bars + 5;      // [3]
    uint64_t* s_full = bars + 8;       // [3] scores of 128 keys of a chunk
    uint64_t* p_full = bars + 11;      // [2] P of a block, blocks in turn
    uint64_t* o_full = bars + 13;      // [2]
    uint64_t* o_free = bars + 15;      // [2]
    uint64_t* pair = bars + 17;        // [4] per lane quarter: both warps have put down a value for the other
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* void_s = reinterpret_cast<int*>(tmem_slot + 2);
    AttnItem* items = reinterpret_cast<AttnItem*>(base + AF_SM_ITEM);
    float* row_x = reinterpret_cast<float*>(base + AF_SM_ROW);
    int* tile_prefix = reinterpret_cast<int*>(base + AF_SM_PREFIX);
    int32_t* offs = tile_prefix + g.B + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (warp == 1 && elect_one()) {
        mbar_init(q_full, 1);
        mbar_init(q_free, 1 + AF_WARPS);
        for (int i = 0; i < AF_SLOTS; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_free[i], 1); mbar_init(&s_full[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&p_full[i], AF_WARPS); mbar_init(&o_full[i], 1); mbar_init(&o_free[i], AF_WARPS); }
        for (int i = 0; i < 4; ++i) mbar_init(&pair[i], 2);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmap_q);
        prefetch_tmap(&tmap_kv);
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    if (warp == 2 && lane < (int)(sizeof(AfArgs) / 4)) asm volatile("" ::"r"(reinterpret_cast<const uint32_t*>(&g)[lane]));
    // Loads of one thread of warp 0: an item and its Q; a slot of K (which = 0) or V of blocks blk and, where there is one, blk + 1
    auto load_q = [&](const AttnItem& it, int slot) {
        items[slot] = it;
        mbar_arrive_expect_tx(q_full, 3 * AF_PLANE);
        for (int t = 0; t < 3; ++t) tma_load_3d_a(smem_u32(base + t * AF_PLANE), &tmap_q, smem_u32(q_full), it.h * HD, t, it.row0);
    };
    auto load_kv = [&](const AttnItem& it, int s, int which, int blk, int halves) {
        mbar_arrive_expect_tx(&kv_full[s], 3 * halves * (AF_PLANE / 2));
        for (int t = 0; t < 3; ++t)
            for (int i = 0; i < halves; ++i)
                tma_load_4d_a(smem_u32(base + AF_SM_KV + (s * 3 + t) * AF_PLANE + i * (AF_PLANE / 2)), &tmap_kv, smem_u32(&kv_full[s]),
                              which * g.C + it.h * HD, t, (blk + i) * 64, it.b);
    };
    __syncthreads();                                 // (the barriers exist)
    pdl_begin();
    // (of up to 256 images warp 0 lists the items alone and sends for the first one's Q and first keys before the others know the list)
    const bool few = PER == 1 || g.B <= FEW_IMAGES;
    FewImages<PER> images;
    if (few && warp == 0) images.load(g.offsets, g.B);
    if (threadIdx.x == (few ? 0 : blockDim.x - 1)) *void_s = launch_is_void(status) ? 1 : 0;
    AttnItem first_item;
    if (!few) {
        list_tiles(g.offsets, g.B, g.max_q, g.l_max, status, tile_prefix, offs);
    } else if (warp == 0) {
        __syncwarp();
        const int n_tiles = images.list(g.B, g.max_q, g.l_max, status, tile_prefix, offs, blockIdx.x, g.heads, first_item);
        if (*void_s == 0 && (int)blockIdx.x < n_tiles * g.heads && elect_one()) {
            load_q(first_item, 0);
            load_kv(first_item, 0, 0, 0, min(2, g.n_blocks / g.n_chunks));       // (the first chunk has so many blocks)
        }
        __syncwarp();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const int n_work = *void_s ? 0 : tile_prefix[g.B] * g.heads;
    constexpr int TA[6] = {2, 0, 1, 1, 0, 0}, TB[6] = {0, 2, 1, 0, 1, 0};        // terms of the products, smallest first
    // blocks [first_block(c), first_block(c + 1)) are chunk c
    auto first_block = [&](int c) { return g.n_blocks * c / g.n_chunks; };
    bool ok = true;
    int li = 0;                                      // items so far

    if (warp == 0) {
        if (elect_one()) {
            // ------------------------------------------------------------ TMA producer
            int n = 0, s = 0;                        // slots filled; the next one
            uint32_t ph = 1;
            for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++li) {
                const bool sent = few && li == 0;         // (its Q and first slot of K are under way)
                const AttnItem it = sent ? first_item : attn_item(w, g.heads, g.B, tile_prefix, offs);
                if (!sent) {
                    ok = mbar_wait(q_free, (li & 1) ^ 1, abort_flag, status, STATUS_ATTN_LOAD);
                    if (!ok) break;
                    load_q(it, li & 1);
                }
                for (int c = 0; c < g.n_chunks && ok; ++c) {
                    const int b0 = first_block(c), b1 = first_block(c + 1);
                    for (int v = 0; v < 2 && ok; ++v) {
                        for (int blk = b0; blk < b1; blk += 2, ++n) {
                            if (!sent || n > 0) {
                                ok = mbar_wait(&kv_free[s], ph, abort_flag, status, STATUS_ATTN_LOAD);
                                if (!ok) break;
                                load_kv(it, s, v, blk, min(2, b1 - blk));
                            }
                            if (++s == AF_SLOTS) { s = 0; ph ^= 1; }
                        }
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            // -------------------------------------------------------------- MMA issuer
            const uint64_t qdesc = smem_desc_sw128(smem_u32(base)), kvdesc = smem_desc_sw128(smem_u32(base + AF_SM_KV));
            constexpr uint64_t PLANE = AF_PLANE >> 4;
            const uint32_t idesc_o = idesc_bf16_f32(QT, HD, 0, 1);     // B = V, MN-major
            int s = 0, pn = 0;                       // slot; blocks of P so far
            uint32_t ph = 0;
            for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++li) {
                ok = mbar_wait(q_full, li & 1, abort_flag, status, STATUS_ATTN_MMA);
                for (int c = 0; c < g.n_chunks && ok; ++c) {
                    const int b0 = first_block(c), b1 = first_block(c + 1);
                    const int nk = min(g.n_keys, b1 * 64) - b0 * 64;
                    for (int j = 0; 2 * j < b1 - b0; ++j) {
                        ok = mbar_wait(&kv_full[s], ph, abort_flag, status, STATUS_ATTN_MMA);
                        if (!ok) break;
                        tc_fence_after_sync();
                        const int N = (min(nk - j * AF_SLOT_KEYS, AF_SLOT_KEYS) + 15) & ~15;
                        const uint32_t idesc_s = idesc_bf16_f32(QT, N, 0, 0);
                        const uint64_t kd = kvdesc + (uint64_t)s * 3 * PLANE;
#pragma unroll
                        for (int p = 0; p < 6; ++p)
#pragma unroll
                            for (int k = 0; k < HD / 16; ++k)
                                umma_ss(tmem_base + j * AF_SLOT_KEYS, qdesc + TA[p] * PLANE + 2 * k, kd + TB[p] * PLANE + 2 * k, idesc_s,
                                        (p | k) != 0 ? 1u : 0u);
                        umma_commit(&kv_free[s]);
                        umma_commit(&s_full[j]);
                        if (++s == AF_SLOTS) { s = 0; ph ^= 1; }
                    }
                    if (!ok) break;
                    if (c + 1 == g.n_chunks) umma_commit(q_free);
                    for (int i = 0; i < b1 - b0; ++i, ++pn) {
                        const int par = pn & 1;
                        const uint32_t use = (uint32_t)(pn >> 1) & 1;
                        if ((i & 1) == 0) ok = mbar_wait(&kv_full[s], ph, abort_flag, status, STATUS_ATTN_MMA);
                        ok = ok && mbar_wait(&p_full[par], use, abort_flag, status, STATUS_ATTN_MMA) &&
                             mbar_wait(&o_free[par], use ^ 1, abort_flag, status, STATUS_ATTN_MMA);
                        if (!ok) break;
                        tc_fence_after_sync();
                        const int ksteps = (min(nk - i * 64, 64) + 15) / 16;
                        // (16 keys = 16 rows of 128 bytes; the second block of a slot starts at row 64)
                        const uint64_t vd = kvdesc + (uint64_t)s * 3 * PLANE + (uint64_t)((i & 1) * (64 * 128 >> 4));
#pragma unroll
                        for (int p = 0; p < 6; ++p) {
                            for (int k = 0; k < ksteps; ++k) {
                                const uint32_t pcol = TA[p] == 2 ? AF_PL + par * 32 + (k >> 1) * 16 + (k & 1) * 8
                                                                 : i * 64 + (k >> 1) * 32 + TA[p] * 16 + (k & 1) * 8;
                                umma_ts(tmem_base + AF_O + par * HD, tmem_base + pcol, vd + TB[p] * PLANE + (uint64_t)(k * (16 * 128 >> 4)),
                                        idesc_o, (p | k) != 0 ? 1u : 0u);
                            }
                        }
                        umma_commit(&o_full[par]);
                        if ((i & 1) == 1 || i + 1 == b1 - b0) {
                            umma_commit(&kv_free[s]);
                            if (++s == AF_SLOTS) { s = 0; ph ^= 1; }
                        }
                    }
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------- softmax + output warps
        const int quarter = warp & 3, hf = (warp - AF_FIRST) >> 2;
        const int r = quarter * 32 + lane;                        // query row = TMEM lane
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        const float sc = g.scale * F_UNSCALE;                     // (the scores come out times 2^32)
        auto arrive = [&](uint64_t* bar) {
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        // a value of the row's other thread (two places in turn: who puts down the next but one has seen the next)
        uint32_t swaps = 0;
        auto swap_row = [&](float v) {
            float* at = row_x + (swaps & 1) * 2 * QT;
            at[hf * QT + r] = v;
            arrive(&pair[quarter]);
            ok = mbar_wait_warp(&pair[quarter], swaps & 1, abort_flag, status, STATUS_ATTN_SOFTMAX);
            ++swaps;
            return at[(hf ^ 1) * QT + r];
        };
        int pn = 0;                                                // blocks of P so far
        uint32_t s_ph = 0;                                         // phases of s_full
        for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++li) {
            ok = mbar_wait_warp(q_full, li & 1, abort_flag, status, STATUS_ATTN_SOFTMAX);
            if (!ok) break;
            const AttnItem it = items[li & 1];
            arrive(q_free);
            const bool live = quarter * 32 < it.nq;                // (both warps of a quarter alike)
            float m = -INFINITY, l = 0.f, bad = 0.f;
            float o[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0.f;
            // O_i of this thread's channels, the block number `n`th of all
            auto take_o = [&](int n) {
                ok = mbar_wait_warp(&o_full[n & 1], (uint32_t)(n >> 1) & 1, abort_flag, status, STATUS_ATTN_SOFTMAX);
                if (!ok) return;
                tc_fence_after_sync();
                if (live) {
                    uint32_t t[32];
                    __syncwarp();
                    tmem_ld_32x32(lane_base + AF_O + (n & 1) * HD + hf * 32, t);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] += __uint_as_float(t[i]);
                }
                tc_fence_before_sync();
                arrive(&o_free[n & 1]);
            };
            for (int c = 0; c < g.n_chunks && ok; ++c) {
                const int b0 = first_block(c), nb = first_block(c + 1) - b0;
                const int nk = min(g.n_keys, (b0 + nb) * 64) - b0 * 64;
                // this thread's scores of block i: columns 64 i + 32 hf + 0 .. valid - 1
                auto valid_of = [&](int i) { return min(max(nk - i * 64 - hf * 32, 0), 32); };
                float mx = -INFINITY;
                for (int i = 0; i < nb; ++i) {
                    if ((i & 1) == 0) {
                        ok = mbar_wait_warp(&s_full[i >> 1], (s_ph >> (i >> 1)) & 1, abort_flag, status, STATUS_ATTN_SOFTMAX);
                        if (!ok) break;
                        s_ph ^= 1u << (i >> 1);
                        tc_fence_after_sync();
                    }
                    const int valid = valid_of(i);
                    if (!live || valid == 0) continue;
                    uint32_t t[32];
                    __syncwarp();
                    tmem_ld_32x32(lane_base + i * 64 + hf * 32, t);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) {
                        // (columns beyond the keys hold anything)
                        const float x = e < valid ? __uint_as_float(t[e]) : 0.f;
                        mx = fmaxf(mx, e < valid ? x * sc : -INFINITY);
                        bad = fmaf(x, 0.f, bad);                   // NaN once a score is infinite or NaN
                    }
                }
                if (!ok) break;
                float m_at = 0.f;
                if (live) {
                    mx = fmaxf(mx, swap_row(mx));
                    if (!ok) break;
                    const float m_new = fmaxf(m, mx);
                    m_at = m_new == -INFINITY ? 0.f : m_new;
                    const float alpha = expf(m - m_at);            // 0 while m is -inf
                    m = m_new;
                    l *= alpha;
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] *= alpha;
                }
                for (int i = 0; i < nb; ++i, ++pn) {
                    const int valid = valid_of(i);
                    if (live && valid > 0) {
                        uint32_t t[32];
                        __syncwarp();
                        tmem_ld_32x32(lane_base + i * 64 + hf * 32, t);
                        tmem_ld_wait();
                        float sum[4] = {0.f, 0.f, 0.f, 0.f};
                        // sixteen keys: no branch among them, every step of the sixteen exponentials is independent of the others'
                        auto unit = [&](int u, auto masked) {
                            uint32_t w3[3][8];
#pragma unroll
                            for (int e = 0; e < 16; e += 2) {
                                uint32_t tt[3][2];
#pragma unroll
                                for (int x = 0; x < 2; ++x) {
                                    const int col = u * 16 + e + x;
                                    float p = expf(fmaf(__uint_as_float(t[col]), sc, -m_at));
                                    if (masked.value) p = col < valid ? p : 0.f;
                                    sum[(e >> 1) & 3] += p;
                                    split_scaled(p * F_SCALE, tt[0][x], tt[1][x], tt[2][x]);
                                }
#pragma unroll
                                for (int q = 0; q < 3; ++q) w3[q][e >> 1] = __byte_perm(tt[q][0], tt[q][1], 0x7632);
                            }
                            __syncwarp();
                            const uint32_t at = lane_base + i * 64 + hf * 32 + u * 8;
                            tmem_st_32x8(at, w3[0]);
                            tmem_st_32x8(at + 16, w3[1]);
                            tmem_st_32x8(lane_base + AF_PL + (pn & 1) * 32 + hf * 16 + u * 8, w3[2]);
                        };
                        if (valid == 32) {
                            unit(0, Masked<false>());
                            unit(1, Masked<false>());
                        } else {
                            unit(0, Masked<true>());
                            if (valid > 16) unit(1, Masked<true>());
                        }
                        l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
                        tmem_st_wait();
                    }
                    tc_fence_before_sync();
                    arrive(&p_full[pn & 1]);
                    if (i > 0) take_o(pn - 1);
                    if (!ok) break;
                }
                if (!ok) break;
                take_o(pn - 1);
            }
            if (!ok) break;
            if (!live) continue;
            l += swap_row(l);
            if (!ok) break;
            const float inv = F_UNSCALE / l;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                o[i] *= inv;
                bad = fmaf(o[i], 0.f, bad);
            }
            bad += swap_row(bad);
            if (!ok) break;
            const bool exists = r < it.nq && it.row0 + r < g.l_max, again = exists && bad != bad;
            const long long row = it.row0 + (exists ? r : 0);
            if (exists && !again) {
                bf16* dst = reinterpret_cast<bf16*>(g.out) + row * 3 * g.C + it.h * HD + hf * 32;
#pragma unroll
                for (int e = 0; e < 32; e += 16) {
                    uint32_t w3[3][8];
#pragma unroll
                    for (int x = 0; x < 16; x += 2) {
                        uint32_t tt[3][2];
#pragma unroll
                        for (int y = 0; y < 2; ++y) split_scaled(o[e + x + y] * F_SCALE, tt[0][y], tt[1][y], tt[2][y]);      // (below 2^96)
#pragma unroll
                        for (int q = 0; q < 3; ++q) w3[q][x >> 1] = __byte_perm(tt[q][0], tt[q][1], 0x7632);
                    }
                    // (32 bytes a store: each touches a line per lane, which is what a store costs here)
#pragma unroll
                    for (int q = 0; q < 3; ++q) stg_u8(dst + (size_t)q * g.C + e, w3[q]);
                }
            }
            // (behind the stores, where a call has no outputs to keep)
            if (__any_sync(0xffffffffu, again)) redo_rows(g, it.b, it.h, row, hf * 32, lane, again);
        }
    }
    if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) { }     // let copies in flight land before releasing memory
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, 512);
}

// Whether blocks with this many keys should take this kernel.  By the keys only: an image's bits must not depend on how many come
// with it.  us, this one / CUDA cores, n_keys / 4 to n_keys / 2 queries, 6 heads: 64 keys 8.4 / 5.8; 145 keys, 2 images 12.1 / 13.4, 16
// 13.0 / 19.7; 257 keys, 1 image 16.2 / 15.2, 4 16.6 / 23.2, 16 17.8 / 43.3; 577 keys, 1 image 27.6 / 32.1, 32 80 / 244; 1025 keys, 1
// image 44 / 83, 32 211 / 651.  Relative error against float64 at 257 keys 2.0e-7 / 4.0e-7, at 1025 2.2e-7 / 6.4e-7.
bool attention_f32_terms_pays(int n_keys) { return n_keys >= 128; }

int attention_f32_terms(const AttnArgs& p, cudaStream_t st) {
    const int C = p.heads * HD;
    VTP_REQUIRE(p.dtype == VTP_F32 && p.head_dim == HD && p.n_keys >= 1, VTP_ERR_UNSUPPORTED, "attention (fp32 terms): head_dim %d, %d keys",
                p.head_dim, p.n_keys);
    VTP_REQUIRE(aligned16(p.q) && aligned16(p.k) && (reinterpret_cast<uintptr_t>(p.out) & 31u) == 0, VTP_ERR_ALIGN,
                "attention (fp32 terms): unaligned pointer");
    if (p.l_max == 0 || p.max_q == 0) return VTP_OK;
    if (p.B > AF_MOST_IMAGES) {
        // (the tile table of a launch holds so many images)
        AttnArgs part = p;
        for (int b = 0; b < p.B; b += AF_MOST_IMAGES) {
            part.B = p.B - b < AF_MOST_IMAGES ? p.B - b : AF_MOST_IMAGES;
            part.offsets = p.offsets + b;
            part.k = static_cast<const bf16*>(p.k) + (size_t)b * p.n_keys * 6 * C;
            if (int rc = attention_f32_terms(part, st)) return rc;
        }
        return VTP_OK;
    }
    AfArgs g;
    g.q = (const bf16*)p.q; g.kv = (const bf16*)p.k; g.out = (float*)p.out; g.B = p.B; g.heads = p.heads; g.C = C; g.n_keys = p.n_keys;
    g.n_blocks = ceil_div(p.n_keys, 64);
    g.n_chunks = ceil_div(g.n_blocks, AF_BLOCKS);
    g.l_max = p.l_max; g.max_q = p.max_q; g.offsets = p.offsets; g.scale = p.scale;
    CUtensorMap tq, tkv;
    {
        const unsigned long long dims[3] = {(unsigned long long)C, 3, (unsigned long long)p.l_max};
        const unsigned long long strides[2] = {(unsigned long long)C * 2, (unsigned long long)C * 6};
        const unsigned box[3] = {HD, 1, QT};
        if (int rc = make_tmap_bf16(&tq, p.q, 3, dims, strides, box)) return rc;
    }
    {
        const unsigned long long dims[4] = {(unsigned long long)C * 2, 3, (unsigned long long)p.n_keys, (unsigned long long)p.B};
        const unsigned long long strides[3] = {(unsigned long long)C * 4, (unsigned long long)C * 12, (unsigned long long)C * 12 * p.n_keys};
        const unsigned box[4] = {HD, 1, 64, 1};
        if (int rc = make_tmap_bf16(&tkv, p.k, 4, dims, strides, box)) return rc;
    }
    const int smem = AF_SM_PREFIX + 2 * (p.B + 1) * 4 + 1024;
    // (batches of up to 32 images have a kernel of their own, whose code a small launch is through sooner: FewImages)
    const bool one_each = p.B <= 32;
    auto kern = one_each ? attn_f32_tc_kernel<1> : attn_f32_tc_kernel<FEW_PER>;
    // (what the largest launch takes, whatever this one does: two threads may get here with different batches)
    static bool reserved[2][64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !reserved[one_each][dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, AF_SM_MOST);
        if (e != cudaSuccess) {
            set_error("attention (fp32 terms): cannot reserve %d bytes of shared memory: %s", AF_SM_MOST, cudaGetErrorString(e));
            return (int)e;
        }
        if (dev >= 0 && dev < 64) reserved[one_each][dev] = true;
    }
    const long long worst = (long long)p.B * ceil_div(p.max_q, QT) * p.heads;
    const int grid = (int)(worst < sm_count() ? worst : sm_count());
    const cudaError_t le = launch_kernel(kern, true, 1, dim3(grid), dim3(AF_THREADS), (size_t)smem, st, tq, tkv, g,
                                         device_status_ptr());
    if (le != cudaSuccess) {
        cudaGetLastError();
        set_error("attention (fp32 terms): %s", cudaGetErrorString(le));
        return (int)le;
    }
    return check_launch("attention (fp32 terms)");
}

}  // namespace vtp
