// Whole-block and whole-model eval forwards: the host-side sequencing of the kernels on
// one stream, with every intermediate in a caller-provided workspace and every
// data-dependent size (the number of packed queries L) left on the device.
//
// Replaces Block.forward and VisionTransformer.forward
// (vtpack/models/dge/deit_dge.py:123-130, 267-299) and, for the comparison baseline,
// Block.forward of vtpack/models/standard/deit.py:79-83.
#include "attention.h"
#include "linear.h"
#include "region_ops.h"

namespace vtp {

int token_im2col(const void* x, int dtype, int B, int H, int W, int C, int sr, void* cols, cudaStream_t st);  // patch_embed.cu

int patch_im2col(const void* images, int image_dtype, int B, int S, int P, int dtype, void* cols, int ld,
                 const void* cls_token, const void* pos_embed, int C, void* x, int32_t* counts, cudaStream_t st);   // patch_embed.cu

// Slices of a workspace, on 32-byte boundaries (the fp32 attention stores 32 bytes at a time): a workspace only has to lie on a
// 16-byte one, and the 16 bytes that may be skipped for it are counted in its size.
struct Carver {
    char* base;
    long long off = 0;
    explicit Carver(void* p) : base(static_cast<char*>(p)) {
        if (reinterpret_cast<uintptr_t>(p) % 32 == 16) base += 16;
    }
    long long bytes() const { return off + 16; }
    void* take(long long bytes) {
        void* r = base ? base + off : nullptr;
        off += round_up(bytes, 256);
        return r;
    }
};

struct BlockScratch {
    int32_t *idx[2], *counts[2], *offsets, *patches, *region_first; // idx / counts / logits / stats_x: this block's and the
    float* logits[2];                                              // next block's (written by this block's unpool)
    float2 *stats_x[2], *stats_q, *stats_acc;
    void *comp, *xn, *qn, *qp, *kv, *ao, *q1, *hid;
    void *sr_cols, *sr_out, *sr_norm;       // spatial reduction (PVT blocks): im2col rows, reduced tokens, their LayerNorm
    void *q_wt, *kv_wt, *proj_wt, *fc1_wt, *fc2_wt, *sr_wt;     // the matrices as terms (block_terms)
    long long bytes;
};

// keys per image: the tokens, or the grid reduced by sr_ratio in each direction
static int keys_per_image(const vtp_dge_shape& s) {
    return s.sr_ratio > 1 ? (s.H / s.sr_ratio) * (s.W / s.sr_ratio) : s.num_extra + s.H * s.W;
}

static RegionGeom region_geom(const vtp_dge_shape& s) {
    RegionGeom g;
    g.B = s.B; g.Hr = s.H / s.region; g.Wr = s.W / s.region; g.W = s.W; g.N = s.num_extra + s.H * s.W; g.C = s.C;
    g.num_extra = s.num_extra; g.region = s.region;
    return g;
}

// Whether the Linears of an fp32 block take their operands as terms (f32_terms.cuh): their inputs are written that way by the
// kernels in front, and the matrices are split beside the pooling.
static bool block_terms(const vtp_dge_shape& s) {
    const long long reduced = (long long)s.B * s.H * s.W * s.C / 8;
    return s.dtype == VTP_F32 && !(s.flags & VTP_FLAG_CUDA_CORES) && s.C % 8 == 0 && s.hidden % 8 == 0 && s.region > 0 &&
           region_ops_supported(region_geom(s), s.dtype) && (s.sr_ratio <= 1 || reduced < (1ll << 32));
}

// ... and its attention too.
static bool attn_terms(const vtp_dge_shape& s) {
    return block_terms(s) && s.C == s.heads * 64 && attention_f32_terms_pays(keys_per_image(s));
}

static BlockScratch carve_block(const vtp_dge_shape& s, void* ws) {
    const long long e = (long long)elem_size(s.dtype);
    const int N = s.num_extra + s.H * s.W;
    const long long rows = (long long)s.B * N;            // worst case: every region at the finest grain
    const int R = (s.H / s.region) * (s.W / s.region);
    Carver c(ws);
    BlockScratch b;
    b.idx[0] = (int32_t*)c.take((long long)s.B * R * 4);
    b.idx[1] = (int32_t*)c.take((long long)s.B * R * 4);
    b.counts[0] = (int32_t*)c.take((long long)s.B * 4);
    b.counts[1] = (int32_t*)c.take((long long)s.B * 4);
    b.offsets = (int32_t*)c.take((long long)(s.B + 1) * 4);
    b.patches = (int32_t*)c.take(rows * 16);
    b.region_first = (int32_t*)c.take((long long)s.B * R * 4);
    b.logits[0] = (float*)c.take((long long)s.B * R * s.n_splits * 4);
    b.logits[1] = (float*)c.take((long long)s.B * R * s.n_splits * 4);
    b.stats_x[0] = (float2*)c.take(rows * 8);
    b.stats_x[1] = (float2*)c.take(rows * 8);
    b.stats_q = (float2*)c.take(rows * 8);
    b.stats_acc = (float2*)c.take(rows * 8 * linear_stat_slots(s.C));
    const bool terms = block_terms(s);
    const long long et = terms ? 6 : e;     // of what a Linear reads
    b.comp = c.take(rows * s.C * e);
    b.xn = c.take(rows * s.C * et);
    b.qn = c.take(rows * s.C * et);
    const long long ea = attn_terms(s) ? 6 : e;     // of what the attention reads
    b.qp = c.take(rows * s.C * ea);
    b.kv = c.take(rows * 2 * s.C * ea);
    b.ao = c.take(rows * s.C * et);
    b.q1 = c.take(rows * s.C * e);
    b.hid = c.take(rows * s.hidden * et);
    b.sr_cols = b.sr_out = b.sr_norm = nullptr;
    if (s.sr_ratio > 1) {
        const long long krows = (long long)s.B * keys_per_image(s);
        b.sr_cols = c.take(rows * s.C * et);            // [B*keys, sr*sr*C] = as many elements as the tokens
        b.sr_out = c.take(krows * s.C * e);
        b.sr_norm = c.take(krows * s.C * et);
    }
    b.q_wt = b.kv_wt = b.proj_wt = b.fc1_wt = b.fc2_wt = b.sr_wt = nullptr;
    if (terms) {
        const long long cc = (long long)s.C * s.C * 6, ch = (long long)s.C * s.hidden * 6;
        b.q_wt = c.take(cc);
        b.kv_wt = c.take(2 * cc);
        b.proj_wt = c.take(cc);
        b.fc1_wt = c.take(ch);
        b.fc2_wt = c.take(ch);
        if (s.sr_ratio > 1) b.sr_wt = c.take(cc * s.sr_ratio * s.sr_ratio);
    }
    b.bytes = c.bytes();
    return b;
}

static int check_shape(const vtp_dge_shape* s) {
    VTP_REQUIRE(s, VTP_ERR_NULL, "block: null shape");
    VTP_REQUIRE(s->dtype == VTP_F32 || s->dtype == VTP_BF16, VTP_ERR_DTYPE, "block: dtype %d", s->dtype);
    VTP_REQUIRE(s->B > 0 && s->H > 0 && s->W > 0 && s->C > 0 && s->heads > 0 && s->hidden > 0 && s->num_extra >= 0,
                VTP_ERR_SHAPE, "block: bad shape");
    VTP_REQUIRE(s->C % s->heads == 0, VTP_ERR_SHAPE, "block: C=%d not divisible by %d heads", s->C, s->heads);
    VTP_REQUIRE(s->region > 0 && s->H % s->region == 0 && s->W % s->region == 0, VTP_ERR_SHAPE,
                "block: grid %dx%d not divisible by region %d", s->H, s->W, s->region);
    VTP_REQUIRE(s->n_splits >= 1 && s->n_splits <= 8, VTP_ERR_SHAPE, "block: n_splits %d", s->n_splits);
    VTP_REQUIRE((long long)s->B * (s->num_extra + s->H * s->W) < (1ll << 30), VTP_ERR_SHAPE, "block: too many tokens");
    if (s->sr_ratio > 1) {
        // the reference reshapes the tokens to [B, C, H, W] before the reduction (pvt_dge.py:82)
        VTP_REQUIRE(s->num_extra == 0, VTP_ERR_SHAPE, "block: spatial reduction needs a grid without extra tokens");
        VTP_REQUIRE(s->H % s->sr_ratio == 0 && s->W % s->sr_ratio == 0, VTP_ERR_SHAPE,
                    "block: grid %dx%d not divisible by the reduction ratio %d", s->H, s->W, s->sr_ratio);
    }
    return VTP_OK;
}

// Records events[i] on the stream after stage i when the caller asked for stage timing.
struct StageMarks {
    void* const* events = nullptr;
    int n = 0;
    cudaStream_t st = nullptr;
    // An event is wanted behind stage i alone, so it cannot share a launch with stage i + 1.
    bool apart(int i) const { return events && i < n && events[i]; }
    int mark(int i) const {
        if (!events || i >= n || !events[i]) return VTP_OK;
        const cudaError_t e = cudaEventRecord(static_cast<cudaEvent_t>(events[i]), st);
        return e == cudaSuccess ? VTP_OK : fail((int)e, "stage event %d: %s", i, cudaGetErrorString(e));
    }
};

static bool has_folded_weights(const vtp_block_weights& w) {
    return w.q_wf && w.q_s && w.q_c && w.kv_wf && w.kv_s && w.kv_c && w.fc1_wf && w.fc1_s && w.fc1_c;
}

static bool has_folded_q_fc1(const vtp_block_weights& w) {
    return w.q_wf && w.q_s && w.q_c && w.fc1_wf && w.fc1_s && w.fc1_c;
}

// Whether a block of this shape runs with norm1 folded into q and norm2 into fc1 (bf16 tensor-core path,
// region-parallel token movers, prepared weights).  A block without a spatial reduction folds kv too.
static bool block_folds(const vtp_dge_shape& s, const vtp_block_weights& w) {
    if (!region_ops_supported(region_geom(s), s.dtype) || s.dtype != VTP_BF16 || (s.flags & VTP_FLAG_CUDA_CORES))
        return false;
    return s.sr_ratio > 1 ? has_folded_q_fc1(w) : has_folded_weights(w);
}

// Whether a block can hand the next one its gate decisions (and, where both fold, the token statistics) from its
// unpool.  The sums behind a decision are the stand-alone gate's, in the same order, on the values it would read.
static bool block_chains(const vtp_dge_shape& s, const vtp_block_weights& w, const vtp_block_weights& next) {
    if (!region_ops_supported(region_geom(s), s.dtype)) return false;
    return block_folds(s, w) == block_folds(s, next);
}

// Whether the pool of a block that nothing prepared works out the packed rows itself: every warp of its B * R CTAs then
// adds up the counts of the images in front and the grains of the regions in front.  From B * R * (B + R) of about
// 500,000 on that costs more than the two launches of the patch-list kernels (one block with 64 channels, derived
// against listed: 256 regions, 8 images 110.5 / 109.3 us, 32 images 242 / 234, 256 images 1442 / 1384; 576 regions, 128
// images 1778 / 1627; 64 regions of 128 channels, 16 images 91.0 / 92.2, 96 images 283 / 281).  Where the gate has counted
// already, deriving saves a launch more.  An image's regions are listed from shared memory (48 KB), so more than 8192 of
// them are always derived.
static bool pool_derives_rows(long long B, long long R, bool counted) {
    return R > 8192 || B * R * (B + R) < (counted ? 2000000 : 500000);
}

// Position of a block inside a model forward: whether the previous block's unpool already
// produced this block's gate decisions and token statistics (in scratch slot `parity`), and
// the block that follows, whose gate and statistics this block's unpool can produce.
struct BlockChain {
    bool have_gate = false;
    bool counts_started = false;         // not chained: an earlier kernel set this block's counts to num_extra
    int32_t* counts_next = nullptr;      // where the next block's counts go (null: scratch)
    int parity = 0;
    const vtp_block_weights* next = nullptr;
    const float* image_bias = nullptr;   // fp32 [B, n_splits] added to this and the next block's router logits
};

// softmax scale of the attention: the shape's attn_scale, or head_dim^-0.5 when it is 0
static float attn_scale(const vtp_dge_shape& s) {
    return s.attn_scale != 0.f ? s.attn_scale : 1.0f / sqrtf((float)(s.C / s.heads));
}

static int block_forward(const vtp_dge_shape& s, const vtp_block_weights& w, const void* x_in, void* x_out,
                         const float* forced_logits, int32_t* counts_out, void* ws, cudaStream_t st,
                         const StageMarks& marks = StageMarks(), const BlockChain& chain = BlockChain()) {
    const int N = s.num_extra + s.H * s.W;
    const int rows = s.B * N;
    const int Hr = s.H / s.region, Wr = s.W / s.region;
    const int C = s.C, d = C / s.heads;
    const unsigned kflag = s.flags & VTP_FLAG_CUDA_CORES;
    BlockScratch b = carve_block(s, ws);
    const int32_t* L_dev = b.offsets + s.B;
    int rc;
    if ((rc = marks.mark(0))) return rc;

    Splits sp;
    if ((rc = make_splits(&sp, s.splits, s.n_splits, s.region))) return rc;
    const RegionGeom g = region_geom(s);
    // Region-parallel gate / pool / unpool when the region is 4x4 tokens, else one warp per patch.
    const bool by_region = region_ops_supported(g, s.dtype);
    const bool reduce = s.sr_ratio > 1;        // PVT block: keys from spatially reduced tokens (explicit LayerNorm rows)
    VTP_REQUIRE(!reduce || (w.sr_w && w.sr_norm_w && w.sr_norm_b), VTP_ERR_NULL,
                "block: spatial reduction needs the sr and sr_norm parameters");
    const int n_keys = keys_per_image(s);
    // LayerNorm folded into the GEMM epilogues (bf16 tensor-core path with prepared weights): norm1 into q and
    // norm2 into fc1.  A PVT block's keys need LayerNorm rows all the same; the pool kernel writes them as the rows of the reducing
    // convolution.  Without a reduction kv folds norm1 too.
    const bool fold_q = block_folds(s, w);
    const bool fold = fold_q && !reduce;
    // norm2 into fc1 only where the reduction is long enough to hide it: with K <= 128 the Linear is bound by its
    // epilogue, the fold adds a quarter to that, and the narrow-row LayerNorm pass costs less than it adds
    const bool fold_fc1 = fold_q && s.C > 128;
    const int par = chain.parity & 1;
    int32_t* idx = b.idx[par];
    int32_t* counts = counts_out ? counts_out : b.counts[par];      // worked out in place: no copy afterwards
    int32_t* counts_next = chain.counts_next ? chain.counts_next : b.counts[par ^ 1];
    float2* stats_x = b.stats_x[par];
    bool stats_x_ready = false;
    // chained: gate decisions, per-image counts and token statistics came from the previous
    // block's unpool; the pool kernel then also derives the row offsets itself
    const bool chained = chain.have_gate && by_region && !forced_logits;
    const bool terms = block_terms(s), terms_attn = attn_terms(s);
    if (terms)
        VTP_REQUIRE(aligned16(w.q_w) && aligned16(w.kv_w) && aligned16(w.proj_w) && aligned16(w.fc1_w) && aligned16(w.fc2_w) &&
                        aligned16(w.sr_w), VTP_ERR_ALIGN, "block: matrices must be 16-byte aligned");
    auto run_linear = [&](LinearArgs& p, const void* w_terms, bool out_terms) {
        if (!terms) return linear(p, st);
        p.w = w_terms;
        p.out_terms = out_terms;
        return linear_f32_terms(p, st);
    };
    const bool derive = by_region && (chained || pool_derives_rows(s.B, Hr * Wr, chain.counts_started));
    VTP_REQUIRE(!chain.image_bias || by_region, VTP_ERR_UNSUPPORTED,
                "block: a per-image gate bias needs the region-parallel gate (4x4-token regions)");

    if (chained) {
        stats_x_ready = fold_q;
        rc = VTP_OK;
    } else if (forced_logits) {
        rc = derive ? count_queries(forced_logits, idx, sp, s.B, Hr * Wr, s.num_extra, counts, st)
                       : vtp_gate_argmax(forced_logits, s.B * Hr * Wr, s.n_splits, idx, st);
    } else if (by_region) {
        RegionGateArgs ga;
        ga.g = g; ga.x = x_in; ga.gw = w.gate_w; ga.gb = w.gate_b; ga.S = s.n_splits; ga.logits_out = b.logits[par];
        ga.idx_out = idx; ga.eps = s.eps; ga.image_bias = chain.image_bias;
        if (fold_q) { ga.stats_x = stats_x; stats_x_ready = true; }
        ga.sp = sp;
        if (chain.counts_started) ga.counts = counts;
        rc = region_gate(ga, s.dtype, st);
    } else {
        rc = vtp_router_gate(x_in, s.dtype, s.B, s.H, s.W, C, s.num_extra, s.region, w.gate_w, w.gate_b,
                             s.n_splits, b.logits[par], idx, st);
    }
    if (rc || (rc = marks.mark(1))) return rc;
    if (!derive)
        rc = index_to_patch(idx, 0, sp, s.B, Hr, Wr, s.region, s.num_extra, counts, b.offsets,
                            by_region ? nullptr : b.patches, nullptr, by_region ? b.region_first : nullptr, st);
    else if (!chained && !forced_logits && !chain.counts_started)
        rc = count_queries(nullptr, idx, sp, s.B, Hr * Wr, s.num_extra, counts, st);
    if (rc || (rc = marks.mark(2))) return rc;
    if (by_region) {
        RegionPoolArgs pa;
        pa.g = g; pa.sp = sp; pa.x = x_in; pa.idx = idx; pa.comp = b.comp; pa.eps = s.eps;
        pa.offsets = b.offsets; pa.region_first = derive ? nullptr : b.region_first;
        pa.counts = counts; pa.offsets_out = b.offsets; pa.region_first_out = b.region_first;
        const bool will_chain = chain.next && block_chains(s, w, *chain.next);
        pa.counts_next = will_chain ? counts_next : nullptr;
        if (fold_q) {
            pa.stats_x = stats_x; pa.stats_q = b.stats_q;
            pa.stats_x_ready = stats_x_ready;
            // (the rows of the reducing convolution come with it)
            if (reduce) { pa.sr = s.sr_ratio; pa.cols = b.sr_cols; pa.lnw = w.norm1_w; pa.lnb = w.norm1_b; }
        }
        else { pa.lnw = w.norm1_w; pa.lnb = w.norm1_b; pa.xn = b.xn; pa.qn = b.qn; }
        if (terms) {
            pa.qn_terms = true;
            pa.xn_terms = !reduce;           // (the gather of a reduction splits its rows itself)
            pa.split.add(w.q_w, b.q_wt, C, C);
            pa.split.add(w.kv_w, b.kv_wt, 2 * C, C);
            pa.split.add(w.proj_w, b.proj_wt, C, C);
            pa.split.add(w.fc1_w, b.fc1_wt, s.hidden, C);
            pa.split.add(w.fc2_w, b.fc2_wt, C, s.hidden);
            if (reduce) pa.split.add(w.sr_w, b.sr_wt, C, s.sr_ratio * s.sr_ratio * C);
        }
        rc = region_pool(pa, s.dtype, st);
    } else {
        rc = vtp_pool(x_in, s.dtype, s.B, N, C, s.W, s.num_extra, b.patches, L_dev, rows, b.comp, w.norm1_w,
                      w.norm1_b, s.eps, b.xn, b.qn, st);
    }
    if (rc || (rc = marks.mark(3))) return rc;

    LinearArgs lq;   // q = LN(comp) Wq^T + b
    lq.a = fold_q ? b.comp : b.qn; lq.lda = C; lq.w = fold_q ? w.q_wf : w.q_w; lq.bias = fold_q ? w.q_c : w.q_b;
    lq.y = b.qp; lq.ldy = C; lq.dtype = s.dtype; lq.m_max = rows; lq.m_dev = L_dev; lq.N = C; lq.K = C; lq.flags = kflag;
    if (fold_q) { lq.ln_mode = 1; lq.ln_stats = b.stats_q; lq.ln_s = w.q_s; }

    LinearArgs lkv;  // kv = LN(x) Wkv^T + b, rows stay [b, key, {k,v}, head, d]
    lkv.a = reduce ? b.sr_norm : fold ? x_in : b.xn; lkv.lda = C; lkv.w = fold ? w.kv_wf : w.kv_w; lkv.bias = fold ? w.kv_c : w.kv_b;
    lkv.y = b.kv; lkv.ldy = 2 * C; lkv.dtype = s.dtype; lkv.m_max = s.B * n_keys; lkv.N = 2 * C; lkv.K = C; lkv.flags = kflag;
    if (fold) { lkv.ln_mode = 1; lkv.ln_stats = stats_x; lkv.ln_s = w.kv_s; }
    // The two projections do not depend on each other: one launch, the q tiles fill the kv tail.  Behind a reduction as well, where q
    // waits for the keys although it need not (apart / together: PVT-tiny, 3 / 33 / 96 images, 460 / 803 / 1493 us and 440 / 791 / 1470;
    // PVT-small, 1 and 96 images, 783 / 2704 and 751 / 2657; in fp32, 1 image, 1228 and 1149).
    const bool pair_bf16 = fold_q && !marks.apart(4) && linear_pair_supported(lkv, lq), pair_f32 = terms && !marks.apart(4);
    if (!pair_bf16 && !pair_f32 && ((rc = run_linear(lq, b.q_wt, terms_attn)) || (rc = marks.mark(4)))) return rc;

    if (reduce) {
        // x_ = norm(sr(LN1(x) as [B,C,H,W])): the stride-sr convolution as im2col rows times a matrix
        const int krows = s.B * n_keys, KS = s.sr_ratio * s.sr_ratio * C;
        if (terms) rc = token_im2col_terms(b.xn, s.B, s.H, s.W, C, s.sr_ratio, b.sr_cols, st);
        else if (!fold_q) rc = token_im2col(b.xn, s.dtype, s.B, s.H, s.W, C, s.sr_ratio, b.sr_cols, st);
        if (rc) return rc;
        LinearArgs lsr;
        lsr.a = b.sr_cols; lsr.lda = KS; lsr.w = w.sr_w; lsr.bias = w.sr_b; lsr.y = b.sr_out; lsr.ldy = C;
        lsr.dtype = s.dtype; lsr.m_max = krows; lsr.N = C; lsr.K = KS; lsr.flags = kflag;
        if ((rc = run_linear(lsr, b.sr_wt, false))) return rc;
        rc = terms ? layernorm_terms(b.sr_out, krows, nullptr, C, w.sr_norm_w, w.sr_norm_b, s.sr_eps, b.sr_norm, st)
                   : vtp_layernorm(b.sr_out, s.dtype, krows, nullptr, C, C, w.sr_norm_w, w.sr_norm_b, s.sr_eps, b.sr_norm, st);
        if (rc) return rc;
    }
    if (pair_bf16) {
        rc = linear_tcgen05_pair(lkv, lq, st);
    } else if (pair_f32) {
        lq.w = b.q_wt; lkv.w = b.kv_wt;
        lq.out_terms = lkv.out_terms = terms_attn;
        rc = linear_f32_terms_pair(lkv, lq, st);
    } else {
        rc = run_linear(lkv, b.kv_wt, terms_attn);
    }
    if (rc || (rc = marks.mark(5))) return rc;

    AttnArgs at;
    const long long e = (long long)elem_size(s.dtype);
    at.q = b.qp; at.q_rs = C; at.q_hs = d;
    at.k = b.kv; at.v = static_cast<const char*>(b.kv) + (long long)C * e;
    at.kv_bs = (long long)n_keys * 2 * C; at.kv_rs = 2 * C; at.kv_hs = d;
    at.out = b.ao; at.o_rs = terms ? 3 * C : C; at.o_hs = d;
    at.o_terms = terms ? C : 0;
    at.dtype = s.dtype; at.B = s.B; at.n_keys = n_keys; at.heads = s.heads; at.head_dim = d;
    at.offsets = b.offsets; at.l_max = rows; at.max_q = N; at.scale = attn_scale(s); at.flags = kflag;
    if ((rc = terms_attn ? attention_f32_terms(at, st) : attention(at, st)) || (rc = marks.mark(6))) return rc;

    LinearArgs lp;   // q1 = comp + attn_out Wp^T + b   (and, when folding, the row sums LN2 needs)
    lp.a = b.ao; lp.lda = C; lp.w = w.proj_w; lp.bias = w.proj_b; lp.res = b.comp; lp.ldr = C; lp.y = b.q1;
    lp.ldy = C; lp.dtype = s.dtype; lp.m_max = rows; lp.m_dev = L_dev; lp.N = C; lp.K = C; lp.flags = kflag;
    if (fold_fc1) lp.emit_stats = b.stats_acc;
    if ((rc = run_linear(lp, b.proj_wt, false)) || (rc = marks.mark(7))) return rc;

    if (!fold_fc1) {
        rc = terms ? layernorm_terms(b.q1, rows, L_dev, C, w.norm2_w, w.norm2_b, s.eps, b.qn, st)
                   : vtp_layernorm(b.q1, s.dtype, rows, L_dev, C, C, w.norm2_w, w.norm2_b, s.eps, b.qn, st);
        if (rc) return rc;
    }
    if ((rc = marks.mark(8))) return rc;

    LinearArgs l1;   // hid = GELU(LN2(q1) W1^T + b)
    l1.a = fold_fc1 ? b.q1 : b.qn; l1.lda = C; l1.w = fold_fc1 ? w.fc1_wf : w.fc1_w; l1.bias = fold_fc1 ? w.fc1_c : w.fc1_b;
    l1.y = b.hid; l1.ldy = s.hidden; l1.dtype = s.dtype; l1.m_max = rows; l1.m_dev = L_dev; l1.N = s.hidden; l1.K = C;
    l1.flags = kflag | VTP_FLAG_GELU;
    if (fold_fc1) { l1.ln_mode = 2; l1.ln_stats = b.stats_acc; l1.ln_s = w.fc1_s; l1.ln_dim = C; l1.ln_eps = s.eps;
                l1.ln_slots = linear_stat_slots(C); }
    LinearArgs l2;   // q2 = q1 + hid W2^T + b   (into the q-projection buffer, dead by now)
    l2.a = b.hid; l2.lda = s.hidden; l2.w = w.fc2_w; l2.bias = w.fc2_b; l2.res = b.q1; l2.ldr = C; l2.y = b.qp;
    l2.ldy = C; l2.dtype = s.dtype; l2.m_max = rows; l2.m_dev = L_dev; l2.N = C; l2.K = s.hidden; l2.flags = kflag;
    if (!marks.apart(9) && mlp_tcgen05_supported(l1, l2) && mlp_tcgen05_pays(l1)) {
        rc = mlp_tcgen05(l1, l2, st);
    } else {
        if ((rc = run_linear(l1, b.fc1_wt, true)) || (rc = marks.mark(9))) return rc;
        rc = run_linear(l2, b.fc2_wt, false);
    }
    if (rc || (rc = marks.mark(10))) return rc;

    if (by_region) {
        RegionUnpoolArgs ua;
        ua.g = g; ua.sp = sp; ua.q = b.qp; ua.comp = b.comp; ua.ref = x_in; ua.out = x_out; ua.idx = idx;
        ua.region_first = b.region_first; ua.offsets = b.offsets;
        if (chain.next && block_chains(s, w, *chain.next)) {
            // the rows being written are the next block's input: leave its LayerNorm statistics and
            // its router gate's decisions in the other scratch slot
            if (fold_q) ua.next.stats_x = b.stats_x[par ^ 1];
            ua.next.eps = s.eps;
            ua.next.gw = chain.next->gate_w; ua.next.gb = chain.next->gate_b; ua.next.S = s.n_splits;
            ua.next.logits = b.logits[par ^ 1]; ua.next.idx = b.idx[par ^ 1];
            ua.next.counts = counts_next;
            ua.next.image_bias = chain.image_bias;
        }
        rc = region_unpool(ua, s.dtype, st);
    } else {
        rc = vtp_unpool_add(b.qp, b.comp, s.dtype, s.B, N, C, s.W, s.num_extra, b.patches, L_dev, rows, x_in,
                            x_out, st);
    }
    if (rc) return rc;
    return marks.mark(11);
}

__global__ void dense_offsets_kernel(int32_t* offsets, int B, int N) {
    pdl_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= B) offsets[i] = i * N;
}

static int dense_block_forward(const vtp_dge_shape& s, const vtp_block_weights& w, const void* x_in, void* x_out,
                               void* ws, cudaStream_t st) {
    const int N = s.num_extra + s.H * s.W;
    const int rows = s.B * N;
    const int C = s.C, d = C / s.heads;
    const unsigned kflag = s.flags & VTP_FLAG_CUDA_CORES;
    BlockScratch b = carve_block(s, ws);
    int rc;
    launch_chain(dense_offsets_kernel, dim3(ceil_div(s.B + 1, 128)), dim3(128), 0, st, b.offsets, s.B, N);
    if ((rc = check_launch("dense offsets"))) return rc;
    rc = vtp_layernorm(x_in, s.dtype, rows, nullptr, C, C, w.norm1_w, w.norm1_b, s.eps, b.xn, st);
    if (rc) return rc;
    LinearArgs lq;
    lq.a = b.xn; lq.lda = C; lq.w = w.q_w; lq.bias = w.q_b; lq.y = b.qp; lq.ldy = C; lq.dtype = s.dtype;
    lq.m_max = rows; lq.N = C; lq.K = C; lq.flags = kflag;
    if ((rc = linear(lq, st))) return rc;
    LinearArgs lkv;
    lkv.a = b.xn; lkv.lda = C; lkv.w = w.kv_w; lkv.bias = w.kv_b; lkv.y = b.kv; lkv.ldy = 2 * C;
    lkv.dtype = s.dtype; lkv.m_max = rows; lkv.N = 2 * C; lkv.K = C; lkv.flags = kflag;
    if ((rc = linear(lkv, st))) return rc;
    AttnArgs at;
    const long long e = (long long)elem_size(s.dtype);
    at.q = b.qp; at.q_rs = C; at.q_hs = d;
    at.k = b.kv; at.v = static_cast<const char*>(b.kv) + (long long)C * e;
    at.kv_bs = (long long)N * 2 * C; at.kv_rs = 2 * C; at.kv_hs = d;
    at.out = b.ao; at.o_rs = C; at.o_hs = d;
    at.dtype = s.dtype; at.B = s.B; at.n_keys = N; at.heads = s.heads; at.head_dim = d;
    at.offsets = b.offsets; at.l_max = rows; at.max_q = N; at.scale = attn_scale(s); at.flags = kflag;
    if ((rc = attention(at, st))) return rc;
    LinearArgs lp;
    lp.a = b.ao; lp.lda = C; lp.w = w.proj_w; lp.bias = w.proj_b; lp.res = x_in; lp.ldr = C; lp.y = b.q1;
    lp.ldy = C; lp.dtype = s.dtype; lp.m_max = rows; lp.N = C; lp.K = C; lp.flags = kflag;
    if ((rc = linear(lp, st))) return rc;
    rc = vtp_layernorm(b.q1, s.dtype, rows, nullptr, C, C, w.norm2_w, w.norm2_b, s.eps, b.qn, st);
    if (rc) return rc;
    LinearArgs l1;
    l1.a = b.qn; l1.lda = C; l1.w = w.fc1_w; l1.bias = w.fc1_b; l1.y = b.hid; l1.ldy = s.hidden;
    l1.dtype = s.dtype; l1.m_max = rows; l1.N = s.hidden; l1.K = C; l1.flags = kflag | VTP_FLAG_GELU;
    if ((rc = linear(l1, st))) return rc;
    LinearArgs l2;
    l2.a = b.hid; l2.lda = s.hidden; l2.w = w.fc2_w; l2.bias = w.fc2_b; l2.res = b.q1; l2.ldr = C; l2.y = x_out;
    l2.ldy = C; l2.dtype = s.dtype; l2.m_max = rows; l2.N = C; l2.K = s.hidden; l2.flags = kflag;
    return linear(l2, st);
}

struct ModelScratch {
    void *cols, *x, *cls_n;
    void* block_ws;
    long long bytes;
};

static ModelScratch carve_model(const vtp_dge_shape& s, const vtp_model_weights& m, void* ws) {
    const long long e = (long long)elem_size(s.dtype);
    const int N = s.num_extra + s.H * s.W;
    Carver c(ws);
    ModelScratch r;
    r.cols = c.take((long long)s.B * s.H * s.W * 3 * m.patch * m.patch * e);
    r.x = c.take((long long)s.B * N * s.C * e);
    r.cls_n = c.take((long long)s.B * s.C * e);
    r.block_ws = c.take(carve_block(s, nullptr).bytes);
    r.bytes = c.bytes();
    return r;
}

// Patch embedding Linear, blocks and final LayerNorm: everything between the im2col and the head.
static int deit_trunk(const vtp_dge_shape& s, const vtp_model_weights& m, const vtp_block_weights* blocks,
                      int32_t* counts_out, const vtp_forward_options* opt, const ModelScratch& ms, const BlockScratch& bs,
                      cudaStream_t st) {
    const int HW = s.H * s.W, N = HW + 1, C = s.C;
    const int KP = 3 * m.patch * m.patch;
    const long long e = (long long)elem_size(s.dtype);
    int rc;
    LinearArgs pe;   // token (b, 1+t) = cols(b,t) Wp^T + bias + pos_embed[1+t]
    pe.a = ms.cols; pe.lda = KP; pe.w = m.patch_w; pe.bias = m.patch_b; pe.res = m.pos_embed; pe.ldr = C;
    pe.y = ms.x; pe.ldy = C; pe.dtype = s.dtype; pe.m_max = s.B * HW; pe.N = C; pe.K = KP;
    pe.flags = s.flags & VTP_FLAG_CUDA_CORES;
    pe.out_grp = HW; pe.out_skip = 1; pe.res_mod = HW; pe.res_off = 1;
    if ((rc = linear(pe, st))) return rc;
    bool chained = false;      // block i-1's unpool prepared block i's gate
    const long long R = (long long)(s.H / s.region) * (s.W / s.region);
    for (int i = 0; i < m.depth; ++i) {
        BlockChain chain;
        chain.have_gate = chained;
        chain.parity = i & 1;
        chain.next = (i + 1 < m.depth) ? &blocks[i + 1] : nullptr;
        chain.counts_next = (counts_out && chain.next) ? counts_out + (size_t)(i + 1) * s.B : nullptr;
        chain.counts_started = i == 0;
        chain.image_bias = opt ? opt->gate_image_bias : nullptr;
        if (opt && opt->tokens_trace) {
            const size_t nb = (size_t)s.B * N * C * e;
            const cudaError_t ce = cudaMemcpyAsync(static_cast<char*>(opt->tokens_trace) + (size_t)i * nb, ms.x, nb,
                                                   cudaMemcpyDeviceToDevice, st);
            if (ce != cudaSuccess) return fail((int)ce, "model: tokens trace copy: %s", cudaGetErrorString(ce));
        }
        rc = block_forward(s, blocks[i], ms.x, ms.x, nullptr, counts_out ? counts_out + (size_t)i * s.B : nullptr,
                           ms.block_ws, st, StageMarks(), chain);
        if (rc) return rc;
        if (opt && opt->grain_trace) {
            // the block's grain indices stay in its slot of the scratch (its unpool writes the other slot)
            const size_t nb = (size_t)s.B * R * sizeof(int32_t);
            const cudaError_t ce = cudaMemcpyAsync(opt->grain_trace + (size_t)i * s.B * R, bs.idx[i & 1], nb,
                                                   cudaMemcpyDeviceToDevice, st);
            if (ce != cudaSuccess) return fail((int)ce, "model: grain trace copy: %s", cudaGetErrorString(ce));
        }
        chained = chain.next && block_chains(s, blocks[i], *chain.next);
    }
    return vtp_layernorm(ms.x, s.dtype, s.B, nullptr, C, (long long)N * C, m.norm_w, m.norm_b, s.eps, ms.cls_n, st);
}

}  // namespace vtp

using namespace vtp;

extern "C" long long vtp_block_workspace_bytes(const vtp_dge_shape* s) {
    if (check_shape(s)) return -1;
    return carve_block(*s, nullptr).bytes;
}

extern "C" int vtp_dge_block_forward(const vtp_dge_shape* s, const vtp_block_weights* w, const void* x_in,
                                     void* x_out, const float* forced_logits, int32_t* counts_out,
                                     void* workspace, long long workspace_bytes, void* stream) {
    if (int rc = check_shape(s)) return rc;
    VTP_REQUIRE(w && x_in && x_out && workspace, VTP_ERR_NULL, "block: null pointer");
    VTP_REQUIRE(aligned16(workspace), VTP_ERR_ALIGN, "block: workspace must be 16-byte aligned");
    VTP_REQUIRE(workspace_bytes >= carve_block(*s, nullptr).bytes, VTP_ERR_SHAPE,
                "block: workspace of %lld bytes is smaller than the %lld needed", workspace_bytes,
                carve_block(*s, nullptr).bytes);
    return block_forward(*s, *w, x_in, x_out, forced_logits, counts_out, workspace,
                         static_cast<cudaStream_t>(stream));
}

extern "C" int vtp_dge_blocks_forward(const vtp_dge_shape* s, const vtp_block_weights* w, int n_blocks,
                                      const void* x_in, void* x_out, int32_t* counts_out, void* workspace,
                                      long long workspace_bytes, void* stream) {
    if (int rc = check_shape(s)) return rc;
    VTP_REQUIRE(w && x_in && x_out && workspace, VTP_ERR_NULL, "blocks: null pointer");
    VTP_REQUIRE(n_blocks > 0, VTP_ERR_SHAPE, "blocks: n_blocks=%d", n_blocks);
    VTP_REQUIRE(aligned16(workspace), VTP_ERR_ALIGN, "blocks: workspace must be 16-byte aligned");
    VTP_REQUIRE(workspace_bytes >= carve_block(*s, nullptr).bytes, VTP_ERR_SHAPE,
                "blocks: workspace of %lld bytes is smaller than the %lld needed", workspace_bytes,
                carve_block(*s, nullptr).bytes);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    bool chained = false;      // block i-1's unpool prepared block i's gate
    for (int i = 0; i < n_blocks; ++i) {
        BlockChain chain;
        chain.have_gate = chained;
        chain.parity = i & 1;
        chain.next = (i + 1 < n_blocks) ? &w[i + 1] : nullptr;
        chain.counts_next = (counts_out && chain.next) ? counts_out + (size_t)(i + 1) * s->B : nullptr;
        if (int rc = block_forward(*s, w[i], i == 0 ? x_in : x_out, x_out, nullptr,
                                   counts_out ? counts_out + (size_t)i * s->B : nullptr, workspace, st, StageMarks(),
                                   chain))
            return rc;
        chained = chain.next && block_chains(*s, w[i], *chain.next);
    }
    return VTP_OK;
}

extern "C" int vtp_dge_block_forward_timed(const vtp_dge_shape* s, const vtp_block_weights* w, const void* x_in,
                                           void* x_out, const float* forced_logits, int32_t* counts_out,
                                           void* workspace, long long workspace_bytes, void* const* events,
                                           int n_events, void* stream) {
    if (int rc = check_shape(s)) return rc;
    VTP_REQUIRE(w && x_in && x_out && workspace && events, VTP_ERR_NULL, "block: null pointer");
    VTP_REQUIRE(aligned16(workspace), VTP_ERR_ALIGN, "block: workspace must be 16-byte aligned");
    VTP_REQUIRE(workspace_bytes >= carve_block(*s, nullptr).bytes, VTP_ERR_SHAPE, "block: workspace too small");
    StageMarks marks;
    marks.events = events; marks.n = n_events; marks.st = static_cast<cudaStream_t>(stream);
    return block_forward(*s, *w, x_in, x_out, forced_logits, counts_out, workspace, marks.st, marks);
}

extern "C" int vtp_dense_block_forward(const vtp_dge_shape* s, const vtp_block_weights* w, const void* x_in,
                                       void* x_out, void* workspace, long long workspace_bytes, void* stream) {
    if (int rc = check_shape(s)) return rc;
    VTP_REQUIRE(w && x_in && x_out && workspace, VTP_ERR_NULL, "dense block: null pointer");
    VTP_REQUIRE(x_in != x_out, VTP_ERR_UNSUPPORTED, "dense block: x_out must not alias x_in");
    VTP_REQUIRE(workspace_bytes >= carve_block(*s, nullptr).bytes, VTP_ERR_SHAPE, "dense block: workspace too small");
    return dense_block_forward(*s, *w, x_in, x_out, workspace, static_cast<cudaStream_t>(stream));
}

extern "C" long long vtp_model_workspace_bytes(const vtp_dge_shape* s, const vtp_model_weights* m) {
    if (check_shape(s) || !m) return -1;
    return carve_model(*s, *m, nullptr).bytes;
}

extern "C" int vtp_deit_dge_forward(const vtp_dge_shape* s, const vtp_model_weights* m,
                                    const vtp_block_weights* blocks, const void* images, float* logits,
                                    int32_t* counts_out, void* workspace, long long workspace_bytes,
                                    void* stream) {
    return vtp_deit_dge_forward_ex(s, m, blocks, images, logits, counts_out, nullptr, workspace, workspace_bytes,
                                   stream);
}

extern "C" int vtp_deit_dge_forward_ex(const vtp_dge_shape* s, const vtp_model_weights* m,
                                       const vtp_block_weights* blocks, const void* images, float* logits,
                                       int32_t* counts_out, const vtp_forward_options* opt, void* workspace,
                                       long long workspace_bytes, void* stream) {
    return vtp_deit_dge_forward_part(s, m, blocks, images, logits, counts_out, opt,
                                     VTP_PART_FRONT | VTP_PART_TRUNK | VTP_PART_HEAD, workspace, workspace_bytes, stream);
}

extern "C" int vtp_deit_dge_forward_part(const vtp_dge_shape* s, const vtp_model_weights* m,
                                         const vtp_block_weights* blocks, const void* images, float* logits,
                                         int32_t* counts_out, const vtp_forward_options* opt, unsigned parts,
                                         void* workspace, long long workspace_bytes, void* stream) {
    if (int rc = check_shape(s)) return rc;
    VTP_REQUIRE(m && blocks && workspace, VTP_ERR_NULL, "model: null pointer");
    VTP_REQUIRE(parts != 0 && (parts & ~7u) == 0, VTP_ERR_SHAPE, "model: parts %u", parts);
    VTP_REQUIRE((images || !(parts & VTP_PART_FRONT)) && (logits || !(parts & VTP_PART_HEAD)), VTP_ERR_NULL, "model: null pointer");
    VTP_REQUIRE(m->depth > 0 && m->patch > 0 && m->num_classes > 0, VTP_ERR_SHAPE, "model: bad shape");
    VTP_REQUIRE(m->img_size == s->H * m->patch && s->H == s->W && s->num_extra == 1, VTP_ERR_SHAPE,
                "model: image %d does not match a %dx%d grid of %d-pixel patches with one cls token",
                m->img_size, s->H, s->W, m->patch);
    VTP_REQUIRE(aligned16(workspace), VTP_ERR_ALIGN, "model: workspace must be 16-byte aligned");
    const ModelScratch ms = carve_model(*s, *m, workspace);
    VTP_REQUIRE(workspace_bytes >= ms.bytes, VTP_ERR_SHAPE, "model: workspace of %lld bytes, %lld needed",
                workspace_bytes, ms.bytes);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int C = s->C, KP = 3 * m->patch * m->patch;
    const BlockScratch bs = carve_block(*s, ms.block_ws);
    int rc = VTP_OK;
    if (parts & VTP_PART_FRONT) {
        // (the kernel that writes the cls rows also starts the first block's query counts)
        rc = patch_im2col(images, m->image_dtype, s->B, m->img_size, m->patch, s->dtype, ms.cols, KP, m->cls_token,
                          m->pos_embed, C, ms.x, counts_out ? counts_out : bs.counts[0], st);
        if (rc) return rc;
    }
    if (parts & VTP_PART_TRUNK) {
        if ((rc = deit_trunk(*s, *m, blocks, counts_out, opt, ms, bs, st))) return rc;
    }
    if (!(parts & VTP_PART_HEAD)) return VTP_OK;
    LinearArgs hd;
    hd.a = ms.cls_n; hd.lda = C; hd.w = m->head_w; hd.bias = m->head_b; hd.y = logits; hd.ldy = m->num_classes;
    hd.dtype = s->dtype; hd.m_max = s->B; hd.N = m->num_classes; hd.K = C;
    hd.flags = (s->flags & VTP_FLAG_CUDA_CORES) | VTP_FLAG_OUT_F32;
    return linear(hd, st);
}
