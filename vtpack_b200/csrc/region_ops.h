// Internal interface of the region-parallel kernels (router gate, pooling, unpooling).
#pragma once

#include "f32_terms.cuh"

namespace vtp {

struct Splits { int v[8]; int n; };

struct RegionGeom {
    int B, Hr, Wr;      // images, regions per column / row
    int W, N, C;        // token grid width, tokens per image (extra + H*W), channels
    int num_extra;      // cls tokens in front of the grid
    int region;         // tokens per region side
    int l_max = 0;      // rows of the packed array where the caller supplies each region's first row
                        // (0: the rows come from this library's own compaction and are not checked)
};

struct RegionPoolArgs {
    RegionGeom g; Splits sp;
    const void* x = nullptr;
    const int32_t* idx = nullptr;            // grain index per region
    const int32_t* region_first = nullptr;   // packed row of each region's first query; null: derive it
                                             //   in the kernel from `counts` and write `offsets_out`
    const int32_t* offsets = nullptr;        // packed row of each image's first query (with region_first)
    const int32_t* counts = nullptr;         // queries per image (without region_first)
    int32_t* offsets_out = nullptr;          // [B+1], written when region_first is null
    int32_t* region_first_out = nullptr;     // [B*R], written when region_first is null (for the unpool)
    int32_t* counts_next = nullptr;          // [B], reset to num_extra for the next block's gate
    void* comp = nullptr;
    // LayerNorm applied later, in a GEMM epilogue: per-row (mean, rstd) of x and of comp, and a
    // per-query accumulator to clear.  Leave null for explicit LayerNorm rows instead.
    float2* stats_x = nullptr; float2* stats_q = nullptr; float2* stats_acc = nullptr;
    bool stats_x_ready = false;              // stats_x was already written (by the previous block's unpool)
    const float* lnw = nullptr; const float* lnb = nullptr; float eps = 1e-6f;
    void* xn = nullptr; void* qn = nullptr;
    bool xn_terms = false, qn_terms = false; // fp32: these rows as terms (f32_terms.cuh)
    TermSplit split;                         // with qn_terms: matrices to split beside the pooling
    // With the statistics and sr > 1 (a divisor of both grid sides, no extra tokens): also LayerNorm(x) (lnw, lnb) in `cols`, as rows of
    // the stride-sr convolution, [B * (H / sr) * (W / sr), sr * sr * C] with column (dy, dx, c).
    int sr = 1; void* cols = nullptr;
    // With neither statistics nor LayerNorm rows asked for: plain pooled rows, as means or (sum_only) as the
    // sums of each patch's tokens, which is the gradient of the replicate-unpool for its packed rows.
    bool sum_only = false;
};

// What the unpool kernel can prepare for the block that follows, from the rows it has just
// written: their LayerNorm statistics and the next router gate's decisions.
struct NextBlock {
    float2* stats_x = nullptr; float eps = 1e-6f;
    const float* gw = nullptr; const float* gb = nullptr; int S = 0;
    float* logits = nullptr; int32_t* idx = nullptr;
    int32_t* counts = nullptr;               // [B] per-image query counts, accumulated with atomics
    const float* image_bias = nullptr;       // [B, S] added to the logits of every region of image b, or null
};

struct RegionUnpoolArgs {
    RegionGeom g; Splits sp;
    const void* q = nullptr; const void* comp = nullptr; const void* ref = nullptr; void* out = nullptr;
    const int32_t* idx = nullptr; const int32_t* region_first = nullptr; const int32_t* offsets = nullptr;
    NextBlock next;
};

struct RegionGateArgs {
    RegionGeom g;
    const void* x = nullptr;
    const float* gw = nullptr; const float* gb = nullptr; int S = 0;
    float* logits_out = nullptr; int32_t* idx_out = nullptr;
    float2* stats_x = nullptr; float eps = 1e-6f;     // optional: also the token rows' (mean, rstd)
    const float* image_bias = nullptr;                // [B, S] added to the logits of every region of image b, or null
    // optional: per-image query counts, started at num_extra by an earlier kernel; every region adds its own
    int32_t* counts = nullptr; Splits sp;
};

// Gated decompress of the training path, or (grad_out) its gradients; rows in one dtype, `gate` [B * R, sp.n] too.
struct GatedArgs {
    RegionGeom g; Splits sp;
    const void *x = nullptr, *comp = nullptr, *gate = nullptr, *ref = nullptr, *grad_out = nullptr;
    const int32_t *idx = nullptr, *region_first = nullptr, *offsets = nullptr;
    void *out = nullptr, *grad_x = nullptr, *grad_comp = nullptr, *grad_gate = nullptr;
    int* status = nullptr;
};

bool region_ops_supported(const RegionGeom& g, int dtype);
int region_gated_unpool(const GatedArgs& a, int dtype, cudaStream_t st);
int region_pool(const RegionPoolArgs& a, int dtype, cudaStream_t st);
int region_unpool(const RegionUnpoolArgs& a, int dtype, cudaStream_t st);
int region_gate(const RegionGateArgs& a, int dtype, cudaStream_t st);

// Patch list + per-region first rows (internal form of vtp_index_to_patch).
int index_to_patch(const void* indices, int idx_is_i64, const Splits& sp, int B, int Hr, int Wr, int region,
                   int num_extra, int32_t* counts, int32_t* offsets, int32_t* patches, int64_t* patches64,
                   int32_t* region_first, cudaStream_t st, int32_t* idx32 = nullptr);

// Per-image query counts of the grain indices `idx` [B, R]; with `logits` [B, R, n_splits] the indices are their
// argmax (lowest index wins) and are written.  One warp per image.
int count_queries(const float* logits, int32_t* idx, const Splits& sp, int B, int R, int num_extra, int32_t* counts,
                  cudaStream_t st);

int make_splits(Splits* sp, const int* splits, int n_splits, int region);

}  // namespace vtp
