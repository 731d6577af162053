// MoE layer and dense gated FFN entry points.
#include <string.h>

#include <algorithm>
#include <new>

#include "internal.h"
#include "moe_aux.cuh"
#include "moe_small.cuh"

struct iq_moe {
    iq_ctx* ctx = nullptr;
    iq_moe_desc d;
    int32_t fmt = 0;
    int32_t ld = 0;  // logits row stride
    const uint32_t* ext_inds = nullptr;
    const float* ext_wts = nullptr;
    // largest row norm of a bf16 router (0: not computed), for the error bound of the tensor-core logits
    float router_wnorm_max = 0.f;
};

namespace iq {

namespace {

struct MoeWs {
    float* logits;
    uint32_t* inds;
    float* wts;
    uint32_t* counts;
    uint32_t* offsets;
    uint32_t* row_map;
    uint32_t* pos;
    uint32_t* ntiles;
    uint32_t* chunk_hist;
    Tile* tiles_a;
    Tile* tiles_b;
    __half* h;
    void* yd;
    __half* xs;  // activations in expert order, fp16 [P, d_model] (tensor-core path)
    FixedRows fx, fh;  // the activations as block fixed point and h likewise, as far as the int8 kernels go
    // shared expert (only when the layer has one): fp16 copy of x, h, output, per-token weight, tile list
    __half* s_x16;
    __half* s_h;
    void* s_yd;
    float* s_w;
    QmmSplit split;  // what the workspace holds beyond `bytes`: partial sums of the shared expert's GEMMs
    size_t bytes;
};

constexpr int kDecodeTileRows = 8;  // token rows per tile of the int8 expert kernels
constexpr int kRouterSmemMax = 200 * 1024;
constexpr int kGroupChunkedMinPairs = 4096;  // from here on the permutation runs as a chunked counting sort
constexpr int kFixedTokens = 512;  // up to here the grouping kernel leaves the activations as fixed point for the int8 kernels
// Affine experts run on the decode tiles (csrc/qmv_tile.cuh) while they see a few rows each on average; everything else, MXFP4 experts at any number of
// rows, runs on the grouped GEMM. The tiles take the token rows as two digits (16 bits of a group's largest input), with the sums and so the bits of the
// expert-parallel pieces' kernel, in the widths that this one takes and 4096: a power of two from 256, up to six rows per expert. In other widths the
// pieces run on the GEMM, which takes bf16 activations whole, and so do three digits (23 bits): with a few input channels 100 times the rest, or one of
// every 64 300 times, two are 4.3e-4 to 5.2e-4 off the 64-bit result (40 and 64 tokens of 2048 x 768), GEMM and three digits 3.0e-4 (24 tokens of 2880 x
// 768). MoE block, us, tiles / GEMM (eight, four, six and eight experts per token):
//   128 experts of 2048 x 768, two digits    20 tokens 77 / 102, 64 98 / 128, 96 (6 rows) 116 / 134, 112 (7 rows) 127 / 135
//   32 of 4096 x 2048, two digits            20 tokens 117 / 152, 48 (6 rows) 142 / 168, 64 (8 rows) 168 / 165
//   64 of 3072 x 1408, three digits          8 tokens 107 / 110, 20 149 / 150, 40 (3.8 rows) 166 / 168, 64 (6 rows) 183 / 169
//   128 of 2880 x 768, three digits          8 tokens 89 / 94, 20 130 / 147, 64 (4 rows) 171 / 183, 80 (5 rows) 193 / 191
// Likewise h: two digits in the widths that the pieces' kernel takes, three (up to four rows per expert, two below 1024 features, then the GEMM) in the
// others, where it has been whole halves. With one feature of every 64 256 times the rest, that do not count in the outputs, two digits are 5e-3 to 7e-3
// off the 64-bit result, three as much as the GEMM, 2.9e-4. h's three digits, tiles / GEMM: 64 of 2048 x 1408 at 4 tokens 55.1 / 58.9, 30 103 / 104,
// 45 (4.2 rows) 108.1 / 108.4, 64 (6) 121 / 116, 32 of 2880 x 2880 at 16 153 / 159, 32 (4) 171 / 182, 256 of 1024 x 704 at 8 46.3 / 47.6, 64 (2) 96.6 / 94.9,
// 190 (5.9) 149 / 140, 64 of 4096 x 704 at 16 (1.5) 95.0 / 97.2, 40 (3.8) 130 / 127.
constexpr int kInt8RowsPerExpert = 6, kWideRowsPerExpert = 4;
bool two_digit_h(const iq_moe* l) { return qmv_grouped_slices(l->d.d_ff, 1) > 0; }
bool two_digit_inputs(const iq_moe* l) { return l->d.d_model >= 256 && l->d.d_model <= 4096 && (l->d.d_model & (l->d.d_model - 1)) == 0; }
// Router products (tokens x experts x inputs) up to which a block takes eight tokens against a few experts in float64 (about
// 0.35 us per million): beyond, the tensor cores with exact refinement (22 us at 27 to 400 million) where they apply, else the
// tiled float64 GEMM. 128 experts x 2048 inputs, router and top-k: 128 tokens 22.8 -> 14.4 us, 200 tokens 22.5 -> 20.4, 400
// tokens 22.5 against 37.6; 32 experts x 2880 inputs, 257 tokens 30.9 -> 10.8, 1000 tokens 41.0 against 38.6.
constexpr int64_t kRouterBlockWork = 56000000, kRouterTiledWork = 90000000;
int64_t router_work(const iq_moe* l, int tokens) { return (int64_t)tokens * l->d.experts * l->d.d_model; }

// Expert outputs between the down projection and the combine: fp16 for affine experts, fp32 for MXFP4 ones, whose
// outputs can pass half's range (the reference makes the same choice, MoEPrefill.swift:159-160).
int32_t yd_dtype_of(const iq_moe* l) { return l->fmt == kFmtMxfp4 ? kF32 : kF16; }

MoeWs carve(const iq_moe* l, void* base, int tokens) {
    const iq_moe_desc& d = l->d;
    const size_t P = (size_t)tokens * d.top_k;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        void* p = base ? static_cast<char*>(base) + off : nullptr;
        off += round_up_sz(bytes, 256);
        return p;
    };
    MoeWs w;
    w.logits = static_cast<float*>(take((size_t)tokens * l->ld * 4));
    w.inds = static_cast<uint32_t*>(take(P * 4));
    w.wts = static_cast<float*>(take(P * 4));
    w.counts = static_cast<uint32_t*>(take((size_t)d.experts * 4));
    w.offsets = static_cast<uint32_t*>(take((size_t)(d.experts + 1) * 4));
    w.row_map = static_cast<uint32_t*>(take(P * 4));
    w.pos = static_cast<uint32_t*>(take(P * 4));
    w.ntiles = static_cast<uint32_t*>(take(16));
    w.chunk_hist = static_cast<uint32_t*>(take((P / kGroupChunk + 1) * (size_t)d.experts * 4));
    w.tiles_a = static_cast<Tile*>(take((d.experts + P / 8 + 1) * sizeof(Tile)));
    w.tiles_b = static_cast<Tile*>(take((d.experts + P / 32 + 1) * sizeof(Tile)));
    w.h = static_cast<__half*>(take(P * d.d_ff * 2));
    w.yd = take(P * d.d_model * (yd_dtype_of(l) == kF16 ? 2 : 4));
    w.xs = static_cast<__half*>(take(P * d.d_model * 2));
    const size_t few = tokens < kSmallTokens ? tokens : kSmallTokens;
    // (of any format and number of owned experts: layers of one shape share a workspace)
    const size_t pairs = std::min(P, (size_t)d.experts * kInt8RowsPerExpert);
    const size_t fixed = std::max(few, std::min((size_t)tokens, (size_t)d.experts * kInt8RowsPerExpert / d.top_k));
    w.fx.digits = static_cast<unsigned char*>(take(fixed * 192 * (d.d_model / 64)));  // (the wide form)
    w.fx.scale = static_cast<float2*>(take(fixed * (d.d_model / 64) * 8));
    w.fh.digits = static_cast<unsigned char*>(take(std::max(pairs, few * d.top_k) * 192 * (d.d_ff / 64)));
    w.fh.scale = static_cast<float2*>(take(std::max(pairs, few * d.top_k) * (d.d_ff / 64) * 8));
    w.s_x16 = nullptr; w.s_h = nullptr; w.s_yd = nullptr; w.s_w = nullptr;
    if (d.shared != IQ_SHARED_NONE) {
        const size_t T = (size_t)tokens;
        w.s_x16 = static_cast<__half*>(take(T * d.d_model * 2));
        w.s_h = static_cast<__half*>(take(T * d.shared_up.n * 2));
        w.s_yd = take(T * d.d_model * 4);
        w.s_w = static_cast<float*>(take(T * 4));
    }
    w.bytes = off;
    return w;
}

typedef void (*RouteKernel)(const RouteParams);
template <bool REFINE, int WPT>
RouteKernel route_kernel_of(int experts) {
    switch ((experts + 31) / 32) {
        case 1: return route_topk_kernel<1, REFINE, WPT>;
        case 2: return route_topk_kernel<2, REFINE, WPT>;
        case 3: return route_topk_kernel<3, REFINE, WPT>;
        case 4: return route_topk_kernel<4, REFINE, WPT>;
        case 5: case 6: return route_topk_kernel<6, REFINE, WPT>;
        case 7: case 8: return route_topk_kernel<8, REFINE, WPT>;
        case 9: case 10: case 11: case 12: return route_topk_kernel<12, REFINE, WPT>;
        default: return route_topk_kernel<16, REFINE, WPT>;
    }
}
// wide: four warps per token share the refinement's exact dot products (few tokens: the chain per token is the time)
RouteKernel route_kernel_for(int experts, bool refine, bool wide) {
    if (!refine) return route_kernel_of<false, 1>(experts);
    return wide ? route_kernel_of<true, 4>(experts) : route_kernel_of<true, 1>(experts);
}
constexpr int kRouteWideMaxTokens = 2048;

// Many tokens with a bf16 router and bf16 activations: the logits come from the tensor cores (bf16 products are exact,
// the fp32 accumulation is not), and the route kernel recomputes exactly, in float64, the few logits per token that
// can still be among the k largest. Indices and weights are then the same bits as with float64 logits throughout, at
// a fifth of the time: the float64 GEMM was 135 us of a 4096-token layer.
// Error bound of an approximate logit: K accumulations, each assumed to lose at most 2^-21 of the running magnitude
// (eight times what round-to-nearest fp32 would), over sum_k |x_k w_k| <= ||x||_2 ||w||_2.
bool tensor_router(const iq_moe* l, int tokens, int32_t x_dtype) {
    const iq_moe_desc& d = l->d;
    return l->router_wnorm_max > 0.f && l->ext_inds == nullptr && d.router_kind == IQ_ROUTER_BF16 &&
           d.router_score == IQ_SCORE_SOFTMAX && x_dtype == kBF16 && router_work(l, tokens) > kRouterBlockWork;
}
float router_err_coef(const iq_moe* l) { return (float)l->d.d_model * 4.76837158e-7f * 1.05f * l->router_wnorm_max; }

RouteParams route_params(const iq_moe* l, const float* logits, int ld, int tokens, uint32_t* inds, float* wts) {
    RouteParams rp;
    rp.logits = logits;
    rp.logits_rw = const_cast<float*>(logits);
    rp.x = nullptr;
    rp.ldx = 0;
    rp.wr = static_cast<const uint16_t*>(l->d.router_w);
    rp.D = l->d.d_model;
    rp.err_coef = router_err_coef(l);
    rp.logit_bias = l->d.router_logit_bias;
    rp.pes = l->d.per_expert_scale;
    rp.inds = inds;
    rp.wts = wts;
    rp.T = tokens; rp.E = l->d.experts; rp.ld = ld; rp.topk = l->d.top_k;
    rp.scale = l->d.routed_scale;
    rp.sigmoid = l->d.router_score == IQ_SCORE_SIGMOID ? 1 : 0;
    rp.select_bias = l->d.router_select_bias;
    rp.eps = l->d.route_eps;
    return rp;
}

int32_t launch_route(iq_moe* l, cudaStream_t st, const float* logits, int ld, int tokens, uint32_t* inds, float* wts,
                     const void* refine_x = nullptr, int64_t ldx = 0) {
    RouteParams rp = route_params(l, logits, ld, tokens, inds, wts);
    rp.x = static_cast<const uint16_t*>(refine_x);
    rp.ldx = ldx;
    const bool wide = refine_x != nullptr && tokens <= kRouteWideMaxTokens;
    return check_cuda(l->ctx, launch_dependent(route_kernel_for(l->d.experts, refine_x != nullptr, wide), dim3(wide ? tokens : (tokens + 3) / 4), 128, 0, st, rp),
                      "route_topk launch");
}

// On the int8 kernels; 1: the shape does not fit them. Gate + up + activation of every tile: h[row, :] = half(act(x W_gate^T + b_g, x W_up^T + b_u)). Expert e's weights live
// at local slot e - expert_lo: the offset is folded into the base pointers. row_map == nullptr: x rows are in place.
int32_t run_gateup(iq_moe* l, cudaStream_t cs, const void* x, int32_t x_dtype, int64_t ldx, const uint32_t* row_map,
                   const Tile* tiles, const uint32_t* ntiles, int max_tiles, __half* h) {
    const iq_moe_desc& d = l->d;
    const int64_t lo = d.expert_lo;
    GqmvCall c;
    c.mode = kModeGateUp;
    c.fmt = l->fmt;
    c.w_estride = (int64_t)d.d_ff * (d.d_model / 8);
    c.s_estride = (int64_t)d.d_ff * (d.d_model / d.gate.group);
    const size_t sb = l->fmt == kFmtMxfp4 ? 1 : 2;
    c.w[0] = static_cast<const uint32_t*>(d.gate.w) - lo * c.w_estride;
    c.w[1] = static_cast<const uint32_t*>(d.up.w) - lo * c.w_estride;
    c.s[0] = static_cast<const char*>(d.gate.scales) - lo * c.s_estride * (int64_t)sb;
    c.s[1] = static_cast<const char*>(d.up.scales) - lo * c.s_estride * (int64_t)sb;
    if (d.gate.biases) {
        c.b[0] = static_cast<const char*>(d.gate.biases) - lo * c.s_estride * 2;
        c.b[1] = static_cast<const char*>(d.up.biases) - lo * c.s_estride * 2;
    }
    c.expert_lo = d.expert_lo; c.expert_count = d.expert_count;
    c.N = d.d_ff; c.K = d.d_model;
    c.x = x; c.x_dtype = x_dtype; c.ldx = ldx;
    c.row_map = row_map;
    c.tiles = tiles; c.ntiles = ntiles; c.grid_tiles = max_tiles;
    c.rows = 0; c.max_rows = kDecodeTileRows;
    c.y = h; c.y_dtype = kF16; c.ldy = d.d_ff;
    if (d.gate_bias) {
        c.ebias[0] = d.gate_bias - lo * d.d_ff;
        c.ebias[1] = d.up_bias - lo * d.d_ff;
    }
    c.limit = d.act == IQ_ACT_SWIGLU_OAI ? d.act_limit : 0.f;
    c.act = d.act;
    return launch_qmv_imma_grouped(l->ctx, cs, c);
}

// Likewise the down projection of every tile: yd[row, :] = h[row, :] W_down^T + b_d.
int32_t run_down(iq_moe* l, cudaStream_t cs, const __half* h, const Tile* tiles, const uint32_t* ntiles, int max_tiles, void* yd,
                 int32_t yd_dtype) {
    const iq_moe_desc& d = l->d;
    const int64_t lo = d.expert_lo;
    GqmvCall c;
    c.mode = kModeDown;
    c.fmt = l->fmt;
    c.w_estride = (int64_t)d.d_model * (d.d_ff / 8);
    c.s_estride = (int64_t)d.d_model * (d.d_ff / d.down.group);
    const size_t sb = l->fmt == kFmtMxfp4 ? 1 : 2;
    c.w[0] = static_cast<const uint32_t*>(d.down.w) - lo * c.w_estride;
    c.s[0] = static_cast<const char*>(d.down.scales) - lo * c.s_estride * (int64_t)sb;
    if (d.down.biases) c.b[0] = static_cast<const char*>(d.down.biases) - lo * c.s_estride * 2;
    c.expert_lo = d.expert_lo; c.expert_count = d.expert_count;
    c.N = d.d_model; c.K = d.d_ff;
    c.x = h; c.x_dtype = kF16; c.ldx = d.d_ff;
    c.tiles = tiles; c.ntiles = ntiles; c.grid_tiles = max_tiles;
    c.rows = 0; c.max_rows = kDecodeTileRows;
    c.y = yd; c.y_dtype = yd_dtype; c.ldy = d.d_model;
    if (d.down_bias) c.ebias[0] = d.down_bias - lo * d.d_model;
    return launch_qmv_imma_grouped(l->ctx, cs, c);
}

bool use_int8_path(const iq_moe* l, int64_t rows) {
    return l->fmt == kFmtAffine4 && rows <= (int64_t)l->d.expert_count * (two_digit_inputs(l) ? kInt8RowsPerExpert : kWideRowsPerExpert);
}
// The limit of the expert-parallel pieces, whose rows come as halves, on csrc/qmv_imma_grouped.cuh (128 experts of 2048 x 768, gate/up and down together: four
// rows each 124 us against 139 on the grouped GEMM, eight 168 against 145)
constexpr int kEpInt8RowsPerExpert = 6;
// Token rows per tile of the grouped GEMM, by the average rows per expert. Up to 64 rows two CTAs share an SM (and 32 hold two
// stages of activations more than 64); from 96 rows on every weight tile is dequantised less often at 192.
int tensor_tile_rows(int64_t rows, int64_t expert_slots) {
    return rows <= expert_slots * 8 ? 32 : rows <= expert_slots * 48 ? 64 : rows < expert_slots * 96 ? 128 : 192;
}

// rows16: fp16 rows [n_rows, d_model] in tile order
int32_t run_gateup_tc(iq_moe* l, cudaStream_t cs, const __half* rows16, int64_t n_rows, const Tile* tiles,
                      const uint32_t* ntiles, __half* h, int bn, bool early = false, const QmmSplit& split = QmmSplit()) {
    const iq_moe_desc& d = l->d;
    QmmCall c;
    c.fmt = l->fmt; c.epi = 1; c.bn = bn;
    c.x16 = rows16; c.ldx = d.d_model; c.x_rows = n_rows;
    c.w[0] = d.gate.w; c.w[1] = d.up.w;
    c.s[0] = d.gate.scales; c.s[1] = d.up.scales;
    c.b[0] = d.gate.biases; c.b[1] = d.up.biases;
    c.experts = d.expert_count; c.expert_lo = d.expert_lo;
    c.N = d.d_ff; c.K = d.d_model; c.M = (int32_t)n_rows;
    c.tiles = tiles; c.ntiles = ntiles;
    c.y = h; c.y_dtype = kF16; c.ldy = d.d_ff;
    c.ebias[0] = d.gate_bias; c.ebias[1] = d.up_bias;
    c.early = early;
    c.split = split;
    c.limit = d.act == IQ_ACT_SWIGLU_OAI ? d.act_limit : 0.f;
    c.act = d.act;
    return launch_qmm(l->ctx, cs, c);
}

int32_t run_down_tc(iq_moe* l, cudaStream_t cs, const __half* h, int64_t n_rows, const Tile* tiles, const uint32_t* ntiles,
                    void* yd, int32_t yd_dtype, int bn, bool early = false, const QmmSplit& split = QmmSplit()) {
    const iq_moe_desc& d = l->d;
    QmmCall c;
    c.fmt = l->fmt; c.epi = 0; c.bn = bn;
    c.x16 = h; c.ldx = d.d_ff; c.x_rows = n_rows;
    c.w[0] = d.down.w; c.s[0] = d.down.scales; c.b[0] = d.down.biases;
    c.experts = d.expert_count; c.expert_lo = d.expert_lo;
    c.N = d.d_model; c.K = d.d_ff; c.M = (int32_t)n_rows;
    c.tiles = tiles; c.ntiles = ntiles;
    c.y = yd; c.y_dtype = yd_dtype; c.ldy = d.d_model;
    c.ebias[0] = d.down_bias;
    c.early = early;
    c.split = split;
    return launch_qmm(l->ctx, cs, c);
}

// The same on tiles of up to eight rows, from block fixed point (csrc/qmv_tile.cuh). Of two digits, the sums go over the grouped kernel's K slices: a
// layer has the bits that iq_moe_experts gives for the same rows
int32_t run_gateup_tile(iq_moe* l, cudaStream_t cs, const MoeWs& w, bool wide, int max_tiles) {
    const iq_moe_desc& d = l->d;
    QmmCall c;
    c.fmt = l->fmt; c.epi = 1; c.bn = kDecodeTileRows;
    c.w[0] = d.gate.w; c.w[1] = d.up.w;
    c.s[0] = d.gate.scales; c.s[1] = d.up.scales;
    c.b[0] = d.gate.biases; c.b[1] = d.up.biases;
    c.experts = d.expert_count; c.expert_lo = d.expert_lo;
    c.N = d.d_ff; c.K = d.d_model;
    c.tiles = w.tiles_a; c.ntiles = w.ntiles;
    c.y = w.h; c.y_dtype = kF16; c.ldy = d.d_ff;
    c.ebias[0] = d.gate_bias; c.ebias[1] = d.up_bias;
    c.limit = d.act == IQ_ACT_SWIGLU_OAI ? d.act_limit : 0.f;
    c.act = d.act;
    return launch_qmv_tile(l->ctx, cs, c, w.fx, wide, w.row_map, d.top_k, 1, max_tiles);
}
int32_t run_down_tile(iq_moe* l, cudaStream_t cs, const MoeWs& w, bool wide, int max_tiles) {
    const iq_moe_desc& d = l->d;
    const int slice = wide ? 1 : d.d_ff / 256 / qmv_grouped_slices(d.d_ff, 1);  // (two digits: the widths that the grouped kernel takes)
    QmmCall c;
    c.fmt = l->fmt; c.epi = 0; c.bn = kDecodeTileRows;
    c.w[0] = d.down.w; c.s[0] = d.down.scales; c.b[0] = d.down.biases;
    c.experts = d.expert_count; c.expert_lo = d.expert_lo;
    c.N = d.d_model; c.K = d.d_ff;
    c.tiles = w.tiles_a; c.ntiles = w.ntiles;
    c.y = w.yd; c.y_dtype = yd_dtype_of(l); c.ldy = d.d_model;
    c.ebias[0] = d.down_bias;
    c.early = true;
    return launch_qmv_tile(l->ctx, cs, c, w.fh, wide, nullptr, 1, slice, max_tiles);
}

// ---- few tokens (csrc/moe_small.cuh) ----
int router_tokens(int tokens) { return tokens <= 1 ? 1 : tokens <= 2 ? 2 : tokens <= 4 ? 4 : 8; }
typedef void (*RouterKernel)(const RouterIn, float*, int, int, int, int);
template <int WFMT>
RouterKernel router_kernel_of(int tt) {
    return tt == 1 ? router_logits_kernel<WFMT, 1> : tt == 2 ? router_logits_kernel<WFMT, 2> : tt == 4 ? router_logits_kernel<WFMT, 4> : router_logits_kernel<WFMT, 8>;
}
RouterKernel router_kernel_pick(bool q8, int tt) { return q8 ? router_kernel_of<1>(tt) : router_kernel_of<0>(tt); }
typedef void (*RouteSmallKernel)(const RouteSmallParams);
template <int WFMT, int TT>
RouteSmallKernel route_small_vpl(int experts) {
    return experts <= 128 ? moe_route_small_kernel<WFMT, TT, 4> : moe_route_small_kernel<WFMT, TT, 16>;
}
template <int WFMT>
RouteSmallKernel route_small_of(int tt, int experts) {
    return tt == 1 ? route_small_vpl<WFMT, 1>(experts) : tt == 2 ? route_small_vpl<WFMT, 2>(experts) : route_small_vpl<WFMT, 4>(experts);
}
RouteSmallKernel route_small_pick(bool q8, int tt, int experts) { return q8 ? route_small_of<1>(tt, experts) : route_small_of<0>(tt, experts); }
constexpr size_t kRouteSmallSmemMax = 200 * 1024;

// Router, top-k and permutation in one cluster: while the float64 products of a block (a cluster has eight) stay at a few
// microseconds and the tokens fit its shared memory.
bool use_route_small(const iq_moe* l, int tokens) {
    const iq_moe_desc& d = l->d;
    const int tt = router_tokens(tokens);
    return tokens <= kSmallTokens && l->ext_inds == nullptr && d.expert_lo == 0 && d.expert_count == d.experts &&
           (int64_t)d.experts * d.d_model * tt <= (1 << 21) && route_small_smem(tt, d.d_model, d.experts) <= kRouteSmallSmemMax;
}
// The experts' kernels for few tokens: affine 4-bit weights, 16-byte aligned; one token, or two and three of small experts. Beyond 24 million
// weights (of one matrix, of every token's experts) the decode tiles take two and three, with three digits; below, the tiles leave the GPU
// half empty. MoE block, us, here / tiles: 64 experts of 1536 x 512 at two and three tokens (12.6 and 18.9 million) 27.0 / 28.7, 30.5 / 32.1, 32 of 1024 x
// 1792 (14.7, 22.0) 26.6 / 29.0, 36.9 / 34.8, 64 of 2880 x 704 (16.2, 24.3) 35.5 / 35.9, 44.1 / 40.0, 128 of 2048 x 768 at two (25.2) 40.9 / 39.9, 64 of
// 2048 x 1408 (34.6) 44.8 / 43.8, 128 of 2880 x 768 (35.4) 61.9 / 50.3
bool use_experts_small(const iq_moe* l, int tokens) {
    const iq_moe_desc& d = l->d;
    if (tokens > 1 && (int64_t)tokens * d.top_k * d.d_model * d.d_ff > 24000000) return false;
    uintptr_t a = 0;
    for (const iq_qlinear* m : {&d.gate, &d.up, &d.down})
        a |= reinterpret_cast<uintptr_t>(m->w) | (reinterpret_cast<uintptr_t>(m->scales) << 2) | (reinterpret_cast<uintptr_t>(m->biases) << 2);
    return l->fmt == kFmtAffine4 && (a & 15) == 0;
}

int32_t run_route_small(iq_moe* l, cudaStream_t cs, const void* x, int32_t x_dtype, int64_t ldx, int tokens, const MoeWs& w, bool fixed, bool wide) {
    const iq_moe_desc& d = l->d;
    RouteSmallParams p;
    p.r = route_params(l, w.logits, l->ld, tokens, w.inds, w.wts);
    p.in = RouterIn{x, x_dtype, ldx, d.router_w, d.router_scales, d.router_biases, d.d_model};
    p.counts = w.counts; p.offsets = w.offsets; p.row_map = w.row_map; p.pos = w.pos; p.ntiles = w.ntiles;
    p.tiles_a = w.tiles_a; p.tiles_b = w.tiles_b;
    p.fx = fixed ? w.fx : FixedRows{nullptr, nullptr};
    p.wide = wide ? 1 : 0;
    const int tt = router_tokens(tokens);
    return check_cuda(l->ctx, launch_dependent(route_small_pick(d.router_kind != IQ_ROUTER_BF16, tt, d.experts), dim3(kSmallCluster), kSmallThreads,
                                               route_small_smem(tt, d.d_model, d.experts), cs, p), "moe_route_small launch");
}

int32_t run_experts_small(iq_moe* l, cudaStream_t cs, int tokens, const MoeWs& w, void* out, int32_t out_dtype, int64_t ldo, int accumulate) {
    const iq_moe_desc& d = l->d;
    iq_ctx* ctx = l->ctx;
    GateUpSmallParams g;
    const iq_qlinear* m[2] = {&d.gate, &d.up};
    for (int i = 0; i < 2; i++) {
        g.w[i] = static_cast<const unsigned char*>(m[i]->w);
        g.s[i] = static_cast<const unsigned char*>(m[i]->scales);
        g.b[i] = static_cast<const unsigned char*>(m[i]->biases);
        g.ebias[i] = i ? d.up_bias : d.gate_bias;
    }
    g.D = d.d_model; g.I = d.d_ff; g.topk = d.top_k;
    g.x = w.fx; g.row_map = w.row_map; g.tiles = w.tiles_a; g.ntiles = w.ntiles;
    g.act = d.act; g.limit = d.act == IQ_ACT_SWIGLU_OAI ? d.act_limit : 0.f;
    g.h = w.h; g.fh = w.fh;
    const int64_t items = (int64_t)tokens * d.top_k * (d.d_ff / 64);
    int32_t st = check_cuda(ctx, launch_dependent(moe_gateup_small_kernel, dim3((unsigned)(items < ctx->sms ? items : ctx->sms)), kSmallThreads, 0, cs, g),
                            "moe_gateup_small launch");
    if (st != kOk) return st;
    DownSmallParams p;
    p.w = static_cast<const unsigned char*>(d.down.w);
    p.s = static_cast<const unsigned char*>(d.down.scales);
    p.b = static_cast<const unsigned char*>(d.down.biases);
    p.D = d.d_model; p.I = d.d_ff; p.topk = d.top_k; p.T = tokens;
    p.fh = w.fh; p.inds = w.inds; p.pos = w.pos; p.wts = w.wts;
    p.ebias = d.down_bias;
    p.yd = static_cast<__half*>(w.yd);
    p.out = out; p.out_dtype = out_dtype; p.ldo = ldo; p.accumulate = accumulate;
    p.slices = 1;
    while (p.slices * 2 * d.top_k <= 16) p.slices *= 2;
    const int ditems = tokens * (d.d_model / 16);
    return check_cuda(ctx, launch_dependent(moe_down_small_kernel, dim3(ditems < ctx->sms ? ditems : ctx->sms), kSmallThreads, 0, cs, p),
                      "moe_down_small launch");
}

// The shared expert (MoE.swift:140-154; the reference runs it as expert id E of the same kernels): one more FFN over all
// tokens, rows in place, through the same tile kernels with a copy of the layer whose expert tensors are the shared
// expert's; out += w_s * y_s with w_s = sigmoid(x . shared_gate) or 1.
int32_t run_shared_expert(iq_moe* l, cudaStream_t cs, const void* x, int32_t x_dtype, int64_t ldx, int tokens, const MoeWs& w,
                          void* out, int32_t out_dtype, int64_t ldo) {
    const iq_moe_desc& d = l->d;
    iq_ctx* ctx = l->ctx;
    iq_moe tmp = *l;
    tmp.d.gate = d.shared_gate_proj; tmp.d.up = d.shared_up; tmp.d.down = d.shared_down;
    tmp.d.d_ff = d.shared_up.n;
    tmp.d.expert_lo = 0; tmp.d.expert_count = 1;
    tmp.d.gate_bias = nullptr; tmp.d.up_bias = nullptr; tmp.d.down_bias = nullptr;
    const bool gated = d.shared == IQ_SHARED_GATED;
    shared_gate_kernel<<<(tokens + 3) / 4, 128, 0, cs>>>(
        x, x_dtype, ldx, gated ? static_cast<const uint32_t*>(d.shared_gate.w) : nullptr,
        static_cast<const uint16_t*>(d.shared_gate.scales), static_cast<const uint16_t*>(d.shared_gate.biases), w.s_w, tokens,
        d.d_model);
    int32_t st = check_cuda(ctx, cudaGetLastError(), "shared_gate launch");
    if (st != kOk) return st;
    const int32_t ydt = yd_dtype_of(l);
    if (tokens <= 16) {  // a dense FFN on the decode kernels
        GqmvCall c;
        c.mode = kModeGateUp;
        c.fmt = kFmtAffine4;
        const iq_qlinear* m[2] = {&d.shared_gate_proj, &d.shared_up};
        for (int i = 0; i < 2; i++) {
            c.w[i] = static_cast<const uint32_t*>(m[i]->w);
            c.s[i] = m[i]->scales;
            c.b[i] = m[i]->biases;
        }
        c.N = d.shared_up.n; c.K = d.d_model;
        c.x = x; c.x_dtype = x_dtype; c.ldx = ldx;
        c.rows = tokens; c.max_rows = tokens;
        c.y = w.s_h; c.y_dtype = kF16; c.ldy = d.shared_up.n;
        c.limit = d.act == IQ_ACT_SWIGLU_OAI ? d.act_limit : 0.f;
        c.act = d.act;
        st = launch_gqmv(ctx, cs, c);
        if (st != kOk) return st;
        GqmvCall q;
        q.mode = kModePlain;
        q.fmt = kFmtAffine4;
        q.w[0] = static_cast<const uint32_t*>(d.shared_down.w);
        q.s[0] = d.shared_down.scales;
        q.b[0] = d.shared_down.biases;
        q.N = q.n_full = d.d_model; q.K = d.shared_up.n;
        q.x = w.s_h; q.x_dtype = kF16; q.ldx = d.shared_up.n;
        q.rows = tokens; q.max_rows = tokens;
        q.y = w.s_yd; q.y_dtype = ydt; q.ldy = d.d_model;
        st = launch_gqmv(ctx, cs, q);
    } else {  // ... or on the GEMM
        const QmmSplit gu = qmm_split(ctx, kFmtAffine4, 1, tokens, d.shared_up.n, d.d_model, w.split.part, w.split.bytes);
        const QmmSplit dn = qmm_split(ctx, kFmtAffine4, 0, tokens, d.d_model, d.shared_up.n, w.split.part, w.split.bytes);
        st = launch_convert_x(ctx, cs, x, x_dtype, ldx, w.s_x16, tokens, d.d_model);
        if (st == kOk) st = run_gateup_tc(&tmp, cs, w.s_x16, tokens, nullptr, nullptr, w.s_h, 0, false, gu);
        if (st == kOk) st = run_down_tc(&tmp, cs, w.s_h, tokens, nullptr, nullptr, w.s_yd, ydt, 0, false, dn);
    }
    if (st != kOk) return st;
    shared_add_kernel<<<tokens, 256, 0, cs>>>(w.s_yd, ydt, w.s_w, out, out_dtype, ldo, tokens, d.d_model);
    return check_cuda(ctx, cudaGetLastError(), "shared_add launch");
}

// The experts' kernels wrote yd; the rows then go where the caller's table points (peer memory included).
int32_t scatter_rows(iq_ctx* ctx, cudaStream_t cs, const void* yd, void* const* yd_rows, int max_rows, int d_model,
                     int32_t yd_dtype) {
    const int row_bytes = d_model * (yd_dtype == kF32 ? 4 : 2);
    const int want = (max_rows + 3) / 4, cap = ctx->sms * 8;
    moe_scatter_rows_kernel<<<want < cap ? want : cap, 256, 0, cs>>>(yd, reinterpret_cast<const uint64_t*>(yd_rows), max_rows, row_bytes);
    return check_cuda(ctx, cudaGetLastError(), "moe_scatter_rows launch");
}

}  // namespace

int32_t moe_init(iq_ctx* ctx) {
    cudaFuncSetAttribute(reinterpret_cast<const void*>(router_logits_tiled_kernel<0, 64>),
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)router_tiled_smem(64));
    cudaFuncSetAttribute(reinterpret_cast<const void*>(router_logits_tiled_kernel<1, 64>),
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)router_tiled_smem(64));
    cudaError_t e = cudaSuccess;
    for (int v = 0; v < 8 && e == cudaSuccess; v++)
        e = cudaFuncSetAttribute(reinterpret_cast<const void*>(router_kernel_pick(v & 1, 1 << (v >> 1))),
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, kRouterSmemMax);
    for (int v = 0; v < 16 && e == cudaSuccess; v++)
        e = cudaFuncSetAttribute(reinterpret_cast<const void*>(route_small_pick(v & 1, 1 << (v >> 1 & 3), v >> 3 ? 256 : 32)),
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRouteSmallSmemMax);
    return check_cuda(ctx, e, "cudaFuncSetAttribute(router)");
}

// ---------------------------------------------------------------------------------------------------------------------
// Elementwise gated activation of the dense FFN GEMM path: h[r, i] = half(act(gu[r, i], gu[r, d_ff + i]))
// (dswiglu_hh of the reference, Shaders/yy_model.metal:187-227).
__global__ void dswiglu_kernel(const float* __restrict__ gu, __half* __restrict__ h, int rows, int d_ff, int act,
                               float limit) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)rows * d_ff) return;
    const size_t r = i / d_ff, c = i % d_ff;
    const float g = gu[r * 2 * d_ff + c], u = gu[r * 2 * d_ff + d_ff + c];
    h[i] = __float2half_rn(glu_rt(act, g, u, limit));
}

}  // namespace iq

using namespace iq;

// ---------------------------------------------------------------------------------------------------------------------
// dense FFN

namespace {
// Scratch of the GEMM path: h fp16 | converted x | (ternary: gate|up fp32) | partial sums of the GEMMs' K splits
struct FfnWs {
    size_t convert, need;  // offset of the converted x; of the partial sums (the scratch without them)
    bool fused;            // gate/up with the activation in its epilogue
};
FfnWs ffn_ws(const iq_qlinear* gate_up, const iq_qlinear* down, int rows, int32_t x_dtype) {
    FfnWs w;
    const int32_t fmt = format_of(gate_up);
    const size_t d_ff = down->k;
    w.convert = round_up_sz((size_t)rows * d_ff * 2, 256);
    w.need = w.convert + round_up_sz(qmm_convert_bytes(rows, gate_up->k, x_dtype), 256);
    w.fused = fmt != kFmtTernary && fmt != kFmtAffine6;
    if (!w.fused) w.need += round_up_sz((size_t)rows * 2 * d_ff * 4, 256);
    return w;
}
// ... of the GEMV path (up to 16 rows): h fp16 | x, then h, as block fixed point
size_t ffn_small_ws(const iq_qlinear* gate_up, const iq_qlinear* down, int rows) {
    const size_t d_ff = down->k;
    return round_up_sz((size_t)rows * d_ff * 2, 256) + round_up_sz((size_t)rows * std::max(d_ff, (size_t)gate_up->k) / 2 * 7, 256);
}
int32_t ffn_chain_check(iq_ctx* ctx, const iq_qlinear* gate_up, const iq_qlinear* down) {
    if (ctx == nullptr || gate_up == nullptr || down == nullptr) return kErrInvalidArg;
    if (gate_up->n % 2 != 0 || gate_up->n / 2 != down->k || gate_up->k != down->n)
        return fail(ctx, kErrInvalidArg, "dense_ffn: gate|up [%d, %d] and down [%d, %d] do not chain", gate_up->n,
                    gate_up->k, down->n, down->k);
    return kOk;
}
}  // namespace

extern "C" int32_t iq_dense_ffn_workspace_bytes(iq_ctx* ctx, const iq_qlinear* gate_up, const iq_qlinear* down,
                                                int32_t rows, int32_t x_dtype, size_t* bytes) {
    const int32_t st = bytes == nullptr ? kErrInvalidArg : ffn_chain_check(ctx, gate_up, down);
    if (st != kOk) return st;
    // never less than a smaller call takes
    *bytes = ffn_small_ws(gate_up, down, std::min(rows, 16));
    if (rows > 16) {
        const FfnWs w = ffn_ws(gate_up, down, rows, x_dtype);
        *bytes = std::max(*bytes, w.need + std::max(qmm_split_bound(ctx, format_of(gate_up), w.fused, rows, w.fused ? down->k : gate_up->n, gate_up->k),
                                                    qmm_split_bound(ctx, format_of(down), 0, rows, down->n, down->k)));
    }
    return kOk;
}

extern "C" int32_t iq_dense_ffn(iq_ctx* ctx, void* stream, const void* x, int32_t x_dtype, int64_t ldx,
                                const iq_qlinear* gate_up, const iq_qlinear* down, int32_t act, float act_limit, void* out,
                                int32_t out_dtype, int64_t ldo, int32_t rows, uint32_t flags, void* workspace,
                                size_t workspace_bytes) {
    int32_t st = ffn_chain_check(ctx, gate_up, down);
    if (st != kOk) return st;
    const FfnWs ws = ffn_ws(gate_up, down, rows, x_dtype);
    // (a workspace without room for the K splits is good as well: every tile is one item then)
    const size_t need = rows <= 16 ? ffn_small_ws(gate_up, down, rows) : ws.need;
    if (workspace == nullptr || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 15) != 0)
        return fail(ctx, kErrWorkspace, "dense_ffn: workspace %zu < %zu (16-byte aligned)", workspace_bytes, need);
    if (act < IQ_ACT_SILU || act > IQ_ACT_RELU2) return fail(ctx, kErrUnsupported, "dense_ffn: activation %d", act);
    const int32_t fmt = format_of(gate_up);
    if (fmt < 0 || format_of(down) < 0) return fail(ctx, kErrUnsupported, "dense_ffn: weight format");
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(stream);
    const int d_ff = down->k;
    __half* h = static_cast<__half*>(workspace);
    if (rows <= 16) {
        if (rows < 1) return fail(ctx, kErrInvalidArg, "dense_ffn: rows = %d", rows);
        if (d_ff % 16 != 0 || gate_up->k % 64 != 0 || ldx % 8 != 0)
            return fail(ctx, kErrInvalidArg, "dense_ffn: shapes (d_ff %% 16, d %% 64, ldx %% 8)");
        // gate and up rows of the concatenated matrix feed one fused gate+up+activation launch
        const size_t row_words = (size_t)gate_up->k / 32 * gate_up->bits;
        const size_t row_groups = (size_t)gate_up->k / gate_up->group;
        const size_t sbytes = fmt == kFmtMxfp4 ? 1 : 2;
        GqmvCall c;
        c.mode = kModeGateUp;
        c.fmt = fmt;
        c.w[0] = static_cast<const uint32_t*>(gate_up->w);
        c.w[1] = c.w[0] + (size_t)d_ff * row_words;
        c.s[0] = gate_up->scales;
        c.s[1] = static_cast<const char*>(gate_up->scales) + (size_t)d_ff * row_groups * sbytes;
        c.b[0] = gate_up->biases;
        c.b[1] = gate_up->biases ? static_cast<const char*>(gate_up->biases) + (size_t)d_ff * row_groups * 2 : nullptr;
        c.N = d_ff; c.K = gate_up->k;
        c.x = x; c.x_dtype = x_dtype; c.ldx = ldx;
        c.rows = rows; c.max_rows = rows;
        c.y = h; c.y_dtype = kF16; c.ldy = d_ff;
        c.limit = act == IQ_ACT_SWIGLU_OAI ? act_limit : 0.f;
        c.act = act;
        c.scratch = static_cast<char*>(workspace) + round_up_sz((size_t)rows * d_ff * 2, 256);
        st = launch_gqmv(ctx, cs, c);
        if (st != kOk) return st;
        return qmv_with_scratch(ctx, stream, h, IQ_F16, d_ff, down, out, out_dtype, ldo, rows, flags, 0, c.scratch);
    }
    if (fmt != kFmtTernary && fmt != kFmtAffine6) {
        // GEMM path, fused: the gate and the up rows of the concatenated matrix are the two weight tiles of one stage of
        // the tcgen05 kernel, whose epilogue applies the activation and writes h = half(act(gate x, up x)) directly
        // (dswiglu_hh of the reference, Shaders/yy_model.metal:187-227, without the fp32 gate|up round trip: at
        // rows = 2048, d_ff = 14336 that is 235 MB not written and read back); then the down GEMM.
        if (rows % 64 != 0 || d_ff % 64 != 0 || gate_up->k % 64 != 0)
            return fail(ctx, kErrInvalidArg, "dense_ffn: rows = %d, d_ff = %d, d = %d must be multiples of 64", rows, d_ff, gate_up->k);
        st = qmm_check(ctx, h, IQ_F16, d_ff, down, out, out_dtype, ldo, rows);
        if (st != kOk) return st;
        char* base = static_cast<char*>(workspace);
        const void* x16 = x;
        int64_t ld16 = ldx;
        const QmmSplit gu = qmm_split(ctx, fmt, 1, rows, d_ff, gate_up->k, base + ws.need, workspace_bytes - ws.need);
        const QmmSplit dn = qmm_split(ctx, format_of(down), 0, rows, down->n, down->k, base + ws.need, workspace_bytes - ws.need);
        if (x_dtype != IQ_F16) {
            if (ldx < gate_up->k || ldx % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0)
                return fail(ctx, kErrInvalidArg, "dense_ffn: x must be 16-byte aligned with ldx >= d and ldx %% 8 == 0");
            st = launch_convert_x(ctx, cs, x, x_dtype, ldx, base + ws.convert, rows, gate_up->k);
            if (st != kOk) return st;
            x16 = base + ws.convert;
            ld16 = gate_up->k;
        }
        const size_t row_words = (size_t)gate_up->k / 32 * gate_up->bits;
        const size_t row_groups = (size_t)gate_up->k / gate_up->group;
        const size_t sbytes = fmt == kFmtMxfp4 ? 1 : 2;
        QmmCall c;
        c.fmt = fmt; c.epi = 1;
        c.x16 = x16; c.ldx = ld16; c.x_rows = rows;
        c.w[0] = gate_up->w;
        c.w[1] = static_cast<const uint32_t*>(gate_up->w) + (size_t)d_ff * row_words;
        c.s[0] = gate_up->scales;
        c.s[1] = static_cast<const char*>(gate_up->scales) + (size_t)d_ff * row_groups * sbytes;
        c.b[0] = gate_up->biases;
        c.b[1] = gate_up->biases ? static_cast<const char*>(gate_up->biases) + (size_t)d_ff * row_groups * 2 : nullptr;
        c.experts = 1;
        c.N = d_ff; c.K = gate_up->k; c.M = rows;
        c.y = h; c.y_dtype = kF16; c.ldy = d_ff;
        c.limit = act == IQ_ACT_SWIGLU_OAI ? act_limit : 0.f;
        c.act = act;
        c.split = gu;
        st = launch_qmm(ctx, cs, c);
        if (st != kOk) return st;
        return qmm_f16(ctx, cs, h, d_ff, down, out, out_dtype, ldo, rows, flags, dn);
    }
    // ternary gate/up rows: gate|up GEMM -> activation -> down GEMM
    char* p = static_cast<char*>(workspace) + round_up_sz((size_t)rows * d_ff * 2, 256);
    float* gu = reinterpret_cast<float*>(p);
    p += round_up_sz((size_t)rows * 2 * d_ff * 4, 256);
    const size_t qbytes = workspace_bytes - (p - static_cast<char*>(workspace));
    st = iq_qmm(ctx, stream, x, x_dtype, ldx, gate_up, gu, IQ_F32, 2 * d_ff, rows, 0, p, qbytes);
    if (st != kOk) return st;
    const size_t total = (size_t)rows * d_ff;
    dswiglu_kernel<<<(unsigned)((total + 255) / 256), 256, 0, cs>>>(gu, h, rows, d_ff, act, act_limit);
    st = check_cuda(ctx, cudaGetLastError(), "dswiglu launch");
    if (st != kOk) return st;
    return iq_qmm(ctx, stream, h, IQ_F16, d_ff, down, out, out_dtype, ldo, rows, flags, p, qbytes);
}

// ---------------------------------------------------------------------------------------------------------------------
// MoE

extern "C" int32_t iq_moe_create(iq_ctx* ctx, const iq_moe_desc* d, iq_moe** out) {
    if (ctx == nullptr || d == nullptr || out == nullptr) return kErrInvalidArg;
    *out = nullptr;
    // the reference's load guards (Layers/MoE.swift:186-219, Layers/MoEPrefill.swift:129-142)
    if (d->experts <= 0 || d->experts % 32 != 0 || d->experts > 512)
        return fail(ctx, kErrUnsupported, "moe: experts = %d (a multiple of 32, at most 512)", d->experts);
    if (d->top_k < 1 || d->top_k > 16 || d->top_k > d->experts)
        return fail(ctx, kErrUnsupported, "moe: top_k = %d (1..16)", d->top_k);
    if (d->d_ff <= 0 || d->d_ff % 64 != 0) return fail(ctx, kErrUnsupported, "moe: d_ff = %d (a multiple of 64)", d->d_ff);
    if (d->d_model < 128 || d->d_model % 64 != 0)
        return fail(ctx, kErrUnsupported, "moe: d_model = %d (a multiple of 64, at least 128)", d->d_model);
    if (d->act < IQ_ACT_SILU || d->act > IQ_ACT_RELU2) return fail(ctx, kErrUnsupported, "moe: activation %d", d->act);
    if (d->router_score != IQ_SCORE_SOFTMAX && d->router_score != IQ_SCORE_SIGMOID)
        return fail(ctx, kErrUnsupported, "moe: router score %d", d->router_score);
    if (d->router_kind != IQ_ROUTER_BF16 && d->router_kind != IQ_ROUTER_Q8)
        return fail(ctx, kErrUnsupported, "moe: router kind %d (bf16 or 8-bit g64; a 4-bit router is not supported)",
                    d->router_kind);
    if (d->router_w == nullptr || (d->router_kind == IQ_ROUTER_Q8 && (!d->router_scales || !d->router_biases)))
        return fail(ctx, kErrInvalidArg, "moe: router tensors missing");
    const int32_t fg = format_of(&d->gate), fu = format_of(&d->up), fd = format_of(&d->down);
    if (fg != fu || fg != fd || (fg != kFmtAffine4 && fg != kFmtMxfp4))
        return fail(ctx, kErrUnsupported, "moe: experts must be all affine 4-bit g64 or all mxfp4");
    if (d->gate.n != d->d_ff || d->gate.k != d->d_model || d->up.n != d->d_ff || d->up.k != d->d_model ||
        d->down.n != d->d_model || d->down.k != d->d_ff)
        return fail(ctx, kErrInvalidArg, "moe: expert tensor shapes do not match d_model/d_ff");
    if (d->expert_lo < 0 || d->expert_count < 1 || d->expert_lo + d->expert_count > d->experts ||
        d->gate.experts != d->expert_count || d->up.experts != d->expert_count || d->down.experts != d->expert_count)
        return fail(ctx, kErrInvalidArg, "moe: expert range [%d, %d) vs %d stacked experts", d->expert_lo,
                    d->expert_lo + d->expert_count, d->gate.experts);
    if (!d->gate.w || !d->up.w || !d->down.w || !d->gate.scales || !d->up.scales || !d->down.scales)
        return fail(ctx, kErrInvalidArg, "moe: expert tensors missing");
    if (fg != kFmtMxfp4 && (!d->gate.biases || !d->up.biases || !d->down.biases))
        return fail(ctx, kErrInvalidArg, "moe: affine experts without biases");
    if ((d->gate_bias != nullptr) != (d->up_bias != nullptr))
        return fail(ctx, kErrInvalidArg, "moe: gate and up expert biases go together");
    if (d->shared != IQ_SHARED_NONE) {
        // the reference's load guards (MoE.swift:186-219, MoEPrefill.swift:129-141): 4-bit affine shared expert, 8-bit
        // gate, width a multiple of 64, no shared expert beside MXFP4 experts
        if (d->shared != IQ_SHARED_GATED && d->shared != IQ_SHARED_UNGATED)
            return fail(ctx, kErrUnsupported, "moe: shared expert kind %d", d->shared);
        if (fg == kFmtMxfp4) return fail(ctx, kErrUnsupported, "moe: MXFP4 experts have no shared expert");
        if (format_of(&d->shared_gate_proj) != kFmtAffine4 || format_of(&d->shared_up) != kFmtAffine4 ||
            format_of(&d->shared_down) != kFmtAffine4)
            return fail(ctx, kErrUnsupported, "moe: the shared expert must be 4-bit affine g64 (got %d/%d/%d bits)",
                        d->shared_gate_proj.bits, d->shared_up.bits, d->shared_down.bits);
        const int si = d->shared_up.n;
        if (si < 64 || si % 64 != 0 || d->shared_gate_proj.n != si || d->shared_up.k != d->d_model ||
            d->shared_gate_proj.k != d->d_model || d->shared_down.n != d->d_model || d->shared_down.k != si ||
            d->shared_up.experts != 1 || d->shared_gate_proj.experts != 1 || d->shared_down.experts != 1)
            return fail(ctx, kErrInvalidArg, "moe: shared expert shapes (width %d)", si);
        if (!d->shared_gate_proj.w || !d->shared_up.w || !d->shared_down.w || !d->shared_gate_proj.biases ||
            !d->shared_up.biases || !d->shared_down.biases)
            return fail(ctx, kErrInvalidArg, "moe: shared expert tensors missing");
        if (d->shared == IQ_SHARED_GATED &&
            (format_of(&d->shared_gate) != kFmtAffine8 || d->shared_gate.n != 1 || d->shared_gate.k != d->d_model ||
             !d->shared_gate.w || !d->shared_gate.scales || !d->shared_gate.biases))
            return fail(ctx, kErrUnsupported, "moe: the shared expert's gate must be 8-bit affine g64 [1, d_model]");
    }
    iq_moe* l = new (std::nothrow) iq_moe();
    if (l == nullptr) return kErrCuda;
    l->ctx = ctx;
    l->d = *d;
    l->fmt = fg;
    l->ld = round_up(d->experts, 64);
    if (d->router_kind == IQ_ROUTER_BF16 && d->router_score == IQ_SCORE_SOFTMAX) {
        // set-up time (this call takes no stream): the largest row norm of the router, for the error bound of the
        // tensor-core logits. The router tensor must be complete on the device when the layer is created.
        uint32_t* dmax = nullptr;
        cudaError_t e = cudaMalloc(&dmax, 4);
        if (e == cudaSuccess) e = cudaMemset(dmax, 0, 4);
        if (e == cudaSuccess) {
            router_wnorm_max_kernel<<<d->experts, 256>>>(static_cast<const uint16_t*>(d->router_w), d->d_model, dmax);
            e = cudaGetLastError();
        }
        uint32_t bits = 0;
        if (e == cudaSuccess) e = cudaMemcpy(&bits, dmax, 4, cudaMemcpyDeviceToHost);
        if (dmax) cudaFree(dmax);
        if (e != cudaSuccess) {
            delete l;
            return check_cuda(ctx, e, "moe: router norm");
        }
        float f;
        memcpy(&f, &bits, 4);
        if (f > 0.f && f < 3.0e38f) l->router_wnorm_max = f;  // otherwise (zero or non-finite router): the float64 path
    }
    *out = l;
    return kOk;
}

extern "C" void iq_moe_destroy(iq_moe* l) { delete l; }

extern "C" int32_t iq_moe_workspace_bytes(const iq_moe* l, int32_t max_tokens, size_t* bytes) {
    if (l == nullptr || bytes == nullptr || max_tokens < 1) return kErrInvalidArg;
    *bytes = carve(l, nullptr, max_tokens).bytes + (l->d.shared != IQ_SHARED_NONE && max_tokens > 16 ? qmm_split_max_bytes(l->ctx) : 0);
    return kOk;
}

extern "C" int32_t iq_moe_get_views(const iq_moe* l, void* workspace, int32_t tokens, iq_moe_views* v) {
    if (l == nullptr || workspace == nullptr || v == nullptr || tokens < 1) return kErrInvalidArg;
    MoeWs w = carve(l, workspace, tokens);
    v->logits = w.logits; v->ld = l->ld;
    v->inds = l->ext_inds ? const_cast<uint32_t*>(l->ext_inds) : w.inds;
    v->wts = l->ext_wts ? const_cast<float*>(l->ext_wts) : w.wts;
    v->offsets = w.offsets; v->row_map = w.row_map; v->pos = w.pos;
    v->h = w.h; v->yd = w.yd; v->yd_dtype = yd_dtype_of(l);
    return kOk;
}

extern "C" int32_t iq_moe_set_external_routing(iq_moe* l, const uint32_t* inds, const float* wts) {
    if (l == nullptr || ((inds == nullptr) != (wts == nullptr))) return kErrInvalidArg;
    l->ext_inds = inds;
    l->ext_wts = wts;
    return kOk;
}

extern "C" int32_t iq_moe_route(iq_moe* l, void* stream, const float* logits, int32_t ld, int32_t tokens, uint32_t* inds,
                                float* wts) {
    if (l == nullptr) return kErrInvalidArg;
    if (logits == nullptr || inds == nullptr || wts == nullptr || tokens < 1 || ld < l->d.experts)
        return fail(l->ctx, kErrInvalidArg, "moe_route: arguments");
    return launch_route(l, reinterpret_cast<cudaStream_t>(stream), logits, ld, tokens, inds, wts);
}

extern "C" int32_t iq_moe_forward(iq_moe* l, void* stream, const void* x, int32_t x_dtype, int64_t ldx, void* out,
                                  int32_t out_dtype, int64_t ldo, int32_t tokens, uint32_t flags, uint32_t pieces,
                                  void* workspace, size_t workspace_bytes) {
    if (l == nullptr) return kErrInvalidArg;
    iq_ctx* ctx = l->ctx;
    const iq_moe_desc& d = l->d;
    if (tokens < 1) return fail(ctx, kErrInvalidArg, "moe: tokens = %d", tokens);
    if (x_dtype < 0 || x_dtype > 2 || out_dtype < 0 || out_dtype > 2) return fail(ctx, kErrInvalidArg, "moe: dtype");
    if ((pieces & (IQ_PIECE_ROUTER | IQ_PIECE_ROUTE | IQ_PIECE_GATEUP)) && (x != nullptr || (pieces & (IQ_PIECE_ROUTER | IQ_PIECE_GATEUP))) &&
        (x == nullptr || ldx < d.d_model || ldx % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0))
        return fail(ctx, kErrInvalidArg, "moe: x must be 16-byte aligned with ldx >= d_model and ldx %% 8 == 0");
    if ((pieces & IQ_PIECE_COMBINE) && (out == nullptr || ldo < d.d_model || ldo % 4 != 0))
        return fail(ctx, kErrInvalidArg, "moe: out / ldo");
    MoeWs w = carve(l, workspace, tokens);
    if (workspace == nullptr || workspace_bytes < w.bytes)
        return fail(ctx, kErrWorkspace, "moe: workspace %zu < %zu", workspace_bytes, w.bytes);
    w.split.part = reinterpret_cast<float*>(static_cast<char*>(workspace) + w.bytes);
    w.split.bytes = workspace_bytes - w.bytes;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(stream);
    const int P = tokens * d.top_k;
    const uint32_t* inds = l->ext_inds ? l->ext_inds : w.inds;
    const float* wts = l->ext_wts ? l->ext_wts : w.wts;
    int32_t st;

    const bool small = pieces == IQ_PIECE_ALL && use_route_small(l, tokens), small_experts = small && use_experts_small(l, tokens);
    const bool int8 = use_int8_path(l, P);
    const bool few_on_tiles = small && !small_experts;  // (the kernels for few tokens take three digits of both)
    const bool wide = few_on_tiles || !two_digit_inputs(l), wide_h = few_on_tiles || !two_digit_h(l);
    if (small) {
        st = run_route_small(l, cs, x, x_dtype, ldx, tokens, w, small_experts || int8, small_experts || wide);
        if (st == kOk && small_experts)
            st = run_experts_small(l, cs, tokens, w, out, out_dtype, ldo, (flags & IQ_FLAG_ACCUMULATE) ? 1 : 0);
        if (st != kOk) return st;
        if (small_experts)
            return d.shared != IQ_SHARED_NONE ? run_shared_expert(l, cs, x, x_dtype, ldx, tokens, w, out, out_dtype, ldo) : kOk;
        pieces &= ~(uint32_t)(IQ_PIECE_ROUTER | IQ_PIECE_ROUTE | IQ_PIECE_GROUP);
    }
    const bool fast_router = tensor_router(l, tokens, x_dtype);
    if ((pieces & IQ_PIECE_ROUTER) && fast_router) {
        QmmCall c;
        c.fmt = kFmtBf16Plain; c.epi = 0; c.bn = 128;
        // one CTA per (token tile, 128 experts): narrower token tiles until the grid covers the GPU (4096 tokens and 128
        // experts: 32 CTAs of 128 tokens took 21 us, the K loop's latency; 128 CTAs of 32 tokens run it side by side)
        while (c.bn > 32 && ((tokens + c.bn - 1) / c.bn) * ((d.experts + 127) / 128) < ctx->sms) c.bn /= 2;
        c.x16 = x; c.ldx = ldx; c.x_rows = tokens;
        c.w[0] = d.router_w;
        c.experts = 1;
        c.N = l->ld; c.w_rows = d.experts; c.K = d.d_model; c.M = tokens;  // (the columns past the experts become zeros)
        c.y = w.logits; c.y_dtype = kF32; c.ldy = l->ld;
        st = launch_qmm(ctx, cs, c);
        if (st != kOk) return st;
    } else if ((pieces & IQ_PIECE_ROUTER) && l->ext_inds == nullptr) {
        // eight experts per block (fewer where that leaves the GPU empty) and as many tokens as fit shared memory
        int tt = router_tokens(tokens);
        while (tt > 1 && router_block_smem(tt, d.d_model, 8) > (size_t)kRouterSmemMax) tt /= 2;
        const bool fits = router_block_smem(tt, d.d_model, 8) <= (size_t)kRouterSmemMax;
        if (tokens > 64 && (router_work(l, tokens) > kRouterTiledWork || !fits)) {
            // register-tiled float64 GEMM; the K range is split over a cluster until the grid fills the GPU several
            // times over (the blocks of one SM share its float64 pipe, so balance comes from many small blocks)
            const int bm = tokens >= 1024 ? 64 : 32;
            const int tiles = ((tokens + bm - 1) / bm) * ((d.experts + kRtBN - 1) / kRtBN);
            const int nchunks = d.d_model / kRtBK;
            int S = 1;
            while (tiles * S < 4 * ctx->sms && S < 8 && nchunks / (2 * S) >= 2) S *= 2;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((tokens + bm - 1) / bm, (d.experts + kRtBN - 1) / kRtBN, S);
            cfg.blockDim = dim3(128);
            cfg.dynamicSmemBytes = router_tiled_smem(bm);
            cfg.stream = cs;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = S;
            cfg.attrs = at; cfg.numAttrs = 1;
            const int cps = (nchunks + S - 1) / S;
            const bool q8 = d.router_kind != IQ_ROUTER_BF16;
            const void* rw = d.router_w;
            const void* rs = q8 ? d.router_scales : nullptr;
            const void* rb = q8 ? d.router_biases : nullptr;
            auto kern = bm == 64 ? (q8 ? router_logits_tiled_kernel<1, 64> : router_logits_tiled_kernel<0, 64>)
                                 : (q8 ? router_logits_tiled_kernel<1, 32> : router_logits_tiled_kernel<0, 32>);
            st = check_cuda(ctx, cudaLaunchKernelEx(&cfg, kern, x, x_dtype, ldx, rw, rs, rb, w.logits, tokens, d.experts,
                                                    d.d_model, l->ld, cps),
                            "router_logits_tiled launch");
            if (st != kOk) return st;
        } else {
        const int groups = (tokens + tt - 1) / tt;
        const int epc = d.experts / 8 * groups * 2 <= ctx->sms ? 4 : 8;
        const size_t smem = router_block_smem(tt, d.d_model, epc);
        if (!fits) return fail(ctx, kErrUnsupported, "moe: d_model = %d is too wide for the router kernel", d.d_model);
        const RouterIn in = {x, x_dtype, ldx, d.router_w, d.router_scales, d.router_biases, d.d_model};
        st = check_cuda(ctx, launch_dependent(router_kernel_pick(d.router_kind != IQ_ROUTER_BF16, tt), dim3(groups, d.experts / epc), kRouterThreads, smem, cs,
                                              in, w.logits, tokens, d.experts, l->ld, epc), "router_logits launch");
        if (st != kOk) return st;
        }
        st = check_cuda(ctx, cudaGetLastError(), "router_logits launch");
        if (st != kOk) return st;
    }
    if ((pieces & IQ_PIECE_ROUTE) && l->ext_inds == nullptr) {
        if (fast_router && x == nullptr) return fail(ctx, kErrInvalidArg, "moe: the route piece needs x (it recomputes logits)");
        st = launch_route(l, cs, w.logits, l->ld, tokens, w.inds, w.wts, fast_router ? x : nullptr, ldx);
        if (st != kOk) return st;
    }
    const int bn = tensor_tile_rows(P, d.expert_count);
    // whole calls on the decode tiles: the grouping kernel leaves the activations as fixed point
    const bool fixed = int8 && (pieces & IQ_PIECE_GATEUP) && (small || ((pieces & IQ_PIECE_GROUP) && tokens <= kFixedTokens && P < kGroupChunkedMinPairs));
    if (pieces & IQ_PIECE_GROUP) {
        GroupParams gp;
        gp.inds = inds; gp.counts = w.counts; gp.offsets = w.offsets; gp.row_map = w.row_map; gp.pos = w.pos;
        gp.tiles_a = w.tiles_a; gp.tiles_b = w.tiles_b; gp.ntiles = w.ntiles;
        gp.P = P; gp.E = d.experts; gp.bm_b = bn;
        // the tiles of eight rows are the int8 kernels'; elsewhere one entry per expert (a prefill of 4096 tokens spent 2.5 us on 32)
        gp.bm_a = int8 ? kDecodeTileRows : 1 << 20;
        gp.e_lo = d.expert_lo; gp.e_hi = d.expert_lo + d.expert_count;
        gp.chunk_hist = w.chunk_hist;
        gp.chunks = (P + kGroupChunk - 1) / kGroupChunk;
        gp.fx = FixedRows{nullptr, nullptr};
        st = kOk;
        if (P >= kGroupChunkedMinPairs && d.experts * 8 * 4 <= 48 * 1024) {
            // many pairs: a chunked counting sort touches each pair once per kernel instead of once per expert
            st = check_cuda(ctx, launch_dependent(moe_hist_kernel, dim3(gp.chunks), 256, d.experts * 4, cs, gp), "moe_hist launch");
            if (st == kOk) st = check_cuda(ctx, launch_dependent(moe_scan_kernel, dim3(1), 256, 0, cs, gp), "moe_scan launch");
            if (st == kOk) st = check_cuda(ctx, launch_dependent(moe_place_kernel, dim3(gp.chunks), 256, d.experts * 8 * 4, cs, gp), "moe_place launch");
        } else {
            if (fixed) { gp.fx = w.fx; gp.fx_wide = wide ? 1 : 0; gp.x = x; gp.x_dtype = x_dtype; gp.ldx = ldx; gp.T = tokens; gp.D = d.d_model; }
            st = check_cuda(ctx, launch_dependent(moe_group_kernel, dim3(d.experts), 256, 0, cs, gp), "moe_group launch");
        }
        if (st == kOk) st = check_cuda(ctx, cudaGetLastError(), "moe_group launch");
        if (st != kOk) return st;
    }
    const int max_tiles = (int)std::min<int64_t>((int64_t)d.expert_count + P / kDecodeTileRows, P);
    bool after_gemm = false;  // h by the GEMM of this call: a down projection on it may start on the tile list and its weights before h is there
    if (pieces & IQ_PIECE_GATEUP) {
        if (int8) {
            st = fixed ? kOk : launch_fixed_rows(ctx, cs, x, x_dtype, ldx, tokens, d.d_model, w.fx, wide);
            if (st == kOk) st = run_gateup_tile(l, cs, w, wide, max_tiles);
        } else {
            after_gemm = true;
            st = check_cuda(ctx, launch_dependent(moe_pack_tokens_kernel, dim3(tokens), 256, 0, cs, x, x_dtype, ldx, w.pos, w.xs, d.d_model, d.top_k),
                            "moe_pack_tokens launch");
            if (st == kOk) st = run_gateup_tc(l, cs, w.xs, P, w.tiles_b, w.ntiles + 1, w.h, bn, true);
        }
        if (st != kOk) return st;
    }
    if (pieces & IQ_PIECE_DOWN) {
        // h's digits come from the halves that lie in the workspace, whichever call or caller left them there: the kernels for few tokens leave digits of
        // another form in fh. The tiles may start before the digits are there: the kernel that makes them lets them, after its own wait.
        if (int8 && (!wide_h || P <= (int64_t)d.expert_count * (d.d_ff < 1024 ? 2 : kWideRowsPerExpert))) {
            st = launch_fixed_rows(ctx, cs, w.h, kF16, d.d_ff, P, d.d_ff, w.fh, wide_h);
            if (st == kOk) st = run_down_tile(l, cs, w, wide_h, max_tiles);
        } else {
            st = run_down_tc(l, cs, w.h, P, w.tiles_b, w.ntiles + 1, w.yd, yd_dtype_of(l), bn, after_gemm);
        }
        if (st != kOk) return st;
    }
    if (pieces & IQ_PIECE_COMBINE) {
        CombineParams cp;
        cp.yd = w.yd; cp.yd_dtype = yd_dtype_of(l); cp.pos = w.pos; cp.wts = wts;
        cp.out = out; cp.out_dtype = out_dtype; cp.ldo = ldo;
        cp.T = tokens; cp.D = d.d_model; cp.topk = d.top_k;
        cp.accumulate = (flags & IQ_FLAG_ACCUMULATE) ? 1 : 0;
        st = check_cuda(ctx, launch_dependent(moe_combine_kernel, dim3(tokens), 256, 0, cs, cp), "moe_combine launch");
        if (st != kOk) return st;
        if (d.shared != IQ_SHARED_NONE) {
            st = run_shared_expert(l, cs, x, x_dtype, ldx, tokens, w, out, out_dtype, ldo);
            if (st != kOk) return st;
        }
    }
    return kOk;
}

// ---------------------------------------------------------------------------------------------------------------------
// Expert-parallel pieces and the stack helper

extern "C" int32_t iq_moe_pack_rows(iq_moe* l, void* stream, const void* x, int32_t x_dtype, int64_t ldx, int32_t tokens,
                                    void* workspace, size_t workspace_bytes, void* rows_f16) {
    if (l == nullptr) return kErrInvalidArg;
    iq_ctx* ctx = l->ctx;
    const iq_moe_desc& d = l->d;
    if (tokens < 1 || x == nullptr || rows_f16 == nullptr || x_dtype < 0 || x_dtype > 2 || ldx < d.d_model || ldx % 8 != 0 ||
        (reinterpret_cast<uintptr_t>(x) & 15) != 0 || (reinterpret_cast<uintptr_t>(rows_f16) & 15) != 0)
        return fail(ctx, kErrInvalidArg, "moe_pack_rows: arguments");
    MoeWs w = carve(l, workspace, tokens);
    if (workspace == nullptr || workspace_bytes < w.bytes)
        return fail(ctx, kErrWorkspace, "moe_pack_rows: workspace %zu < %zu", workspace_bytes, w.bytes);
    const int P = tokens * d.top_k;
    moe_pack_rows_kernel<<<P, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(x, x_dtype, ldx, w.pos,
                                                                                static_cast<__half*>(rows_f16), P,
                                                                                d.d_model, d.top_k);
    return check_cuda(ctx, cudaGetLastError(), "moe_pack_rows launch");
}

namespace {
struct ExpertsWs {
    Tile* tiles;
    uint32_t* ntiles;
    __half* h;
    __half* xs;  // rows fetched through an index, in tile order (tensor-core path)
    size_t bytes;
};
ExpertsWs carve_experts(const iq_moe* l, void* base, int max_rows, int sources) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        void* p = base ? static_cast<char*>(base) + off : nullptr;
        off += round_up_sz(bytes, 256);
        return p;
    };
    ExpertsWs w;
    w.tiles = static_cast<Tile*>(take(((size_t)max_rows / 8 + (size_t)sources * l->d.expert_count + 1) * sizeof(Tile)));
    w.ntiles = static_cast<uint32_t*>(take(16));
    w.h = static_cast<__half*>(take((size_t)max_rows * l->d.d_ff * 2));
    w.xs = static_cast<__half*>(take((size_t)max_rows * l->d.d_model * 2));
    w.bytes = off;
    return w;
}
}  // namespace

extern "C" int32_t iq_moe_experts_workspace_bytes(const iq_moe* l, int32_t max_rows, int32_t sources, size_t* bytes) {
    if (l == nullptr || bytes == nullptr || max_rows < 1 || sources < 1 || sources > kMaxEpSources) return kErrInvalidArg;
    *bytes = carve_experts(l, nullptr, max_rows, sources).bytes;
    return kOk;
}

namespace {
int32_t moe_experts_impl(iq_moe* l, void* stream, const void* rows_f16, const uint32_t* row_index, int32_t total_rows,
                         int32_t max_rows, const uint32_t* counts, int32_t sources, int32_t region_rows, void* yd, int32_t yd_dtype,
                         void* const* yd_rows, void* workspace, size_t workspace_bytes);
}

extern "C" int32_t iq_moe_experts(iq_moe* l, void* stream, const void* rows_f16, int32_t total_rows, int32_t max_rows,
                                  const uint32_t* counts, int32_t sources, int32_t region_rows, void* yd, int32_t yd_dtype,
                                  void* const* yd_rows, void* workspace, size_t workspace_bytes) {
    return moe_experts_impl(l, stream, rows_f16, nullptr, total_rows, max_rows, counts, sources, region_rows, yd, yd_dtype, yd_rows,
                            workspace, workspace_bytes);
}

extern "C" int32_t iq_moe_experts_indexed(iq_moe* l, void* stream, const void* rows_f16, const uint32_t* row_index,
                                          int32_t total_rows, int32_t max_rows, const uint32_t* counts, void* yd, int32_t yd_dtype,
                                          void* const* yd_rows, void* workspace, size_t workspace_bytes) {
    if (l != nullptr && row_index == nullptr) return fail(l->ctx, kErrInvalidArg, "moe_experts_indexed: row_index");
    return moe_experts_impl(l, stream, rows_f16, row_index, total_rows, max_rows, counts, 1, 0, yd, yd_dtype, yd_rows, workspace,
                            workspace_bytes);
}

namespace {
int32_t moe_experts_impl(iq_moe* l, void* stream, const void* rows_f16, const uint32_t* row_index, int32_t total_rows,
                         int32_t max_rows, const uint32_t* counts, int32_t sources, int32_t region_rows, void* yd, int32_t yd_dtype,
                         void* const* yd_rows, void* workspace, size_t workspace_bytes) {
    if (l == nullptr) return kErrInvalidArg;
    iq_ctx* ctx = l->ctx;
    const iq_moe_desc& d = l->d;
    if (rows_f16 == nullptr || counts == nullptr || yd == nullptr || sources < 1 || sources > kMaxEpSources ||
        sources * d.expert_count > 4096 ||
        total_rows < 0 || total_rows > max_rows || (yd_dtype != kF32 && yd_dtype != kF16) || region_rows < 0 ||
        (int64_t)region_rows * sources > max_rows ||
        (reinterpret_cast<uintptr_t>(rows_f16) & 15) != 0)
        return fail(ctx, kErrInvalidArg, "moe_experts: arguments");
    if (total_rows == 0) return kOk;
    ExpertsWs w = carve_experts(l, workspace, max_rows, sources);
    if (workspace == nullptr || workspace_bytes < w.bytes)
        return fail(ctx, kErrWorkspace, "moe_experts: workspace %zu < %zu", workspace_bytes, w.bytes);
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(stream);
    const int64_t slots = (int64_t)sources * d.expert_count;
    // the row count is only known on the device: bounds come from the capacity, total_rows picks the kernels
    const bool int8 = l->fmt == kFmtAffine4 && total_rows <= slots * kEpInt8RowsPerExpert;
    const int bn = int8 ? 16 : tensor_tile_rows(total_rows, slots);  // (where a shape does not fit the int8 kernels the GEMM takes their tiles)
    ep_tiles_kernel<<<1, 512, 0, cs>>>(counts, sources, d.experts, d.expert_lo, d.expert_count, int8 ? kDecodeTileRows : bn,
                                       (uint32_t)region_rows, w.tiles, w.ntiles);
    int32_t st = check_cuda(ctx, cudaGetLastError(), "ep_tiles launch");
    if (st != kOk) return st;
    const int max_tiles = (int)std::min<int64_t>(max_rows / kDecodeTileRows + slots, max_rows);
    st = int8 ? run_gateup(l, cs, rows_f16, kF16, d.d_model, row_index, w.tiles, w.ntiles, max_tiles, w.h) : 1;
    if (st == 1) {
        const __half* rows = static_cast<const __half*>(rows_f16);
        if (row_index != nullptr) {
            moe_gather_rows_kernel<<<ctx->sms * 8, 256, 0, cs>>>(rows, row_index, w.tiles, w.ntiles, bn, w.xs, d.d_model);
            st = check_cuda(ctx, cudaGetLastError(), "moe_gather_rows launch");
            if (st != kOk) return st;
            rows = w.xs;
        }
        st = run_gateup_tc(l, cs, rows, max_rows, w.tiles, w.ntiles, w.h, bn);
    }
    if (st != kOk) return st;
    st = int8 ? run_down(l, cs, w.h, w.tiles, w.ntiles, max_tiles, yd, yd_dtype) : 1;
    if (st == 1) st = run_down_tc(l, cs, w.h, max_rows, w.tiles, w.ntiles, yd, yd_dtype, bn);
    if (st != kOk || yd_rows == nullptr) return st;
    return scatter_rows(ctx, cs, yd, yd_rows, max_rows, d.d_model, yd_dtype);
}
}  // namespace

extern "C" int32_t iq_moe_combine_rows(iq_moe* l, void* stream, const void* yd_rows, int32_t yd_dtype, int32_t tokens,
                                       void* out, int32_t out_dtype, int64_t ldo, uint32_t flags, void* workspace,
                                       size_t workspace_bytes) {
    if (l == nullptr) return kErrInvalidArg;
    iq_ctx* ctx = l->ctx;
    const iq_moe_desc& d = l->d;
    if (yd_rows == nullptr || out == nullptr || tokens < 1 || (yd_dtype != kF32 && yd_dtype != kF16) || out_dtype < 0 ||
        out_dtype > 2 || ldo < d.d_model || ldo % 4 != 0)
        return fail(ctx, kErrInvalidArg, "moe_combine_rows: arguments");
    MoeWs w = carve(l, workspace, tokens);
    if (workspace == nullptr || workspace_bytes < w.bytes)
        return fail(ctx, kErrWorkspace, "moe_combine_rows: workspace %zu < %zu", workspace_bytes, w.bytes);
    CombineParams cp;
    cp.yd = yd_rows; cp.yd_dtype = yd_dtype; cp.pos = w.pos; cp.wts = l->ext_wts ? l->ext_wts : w.wts;
    cp.out = out; cp.out_dtype = out_dtype; cp.ldo = ldo;
    cp.T = tokens; cp.D = d.d_model; cp.topk = d.top_k;
    cp.accumulate = (flags & IQ_FLAG_ACCUMULATE) ? 1 : 0;
    moe_combine_kernel<<<tokens, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(cp);
    return check_cuda(ctx, cudaGetLastError(), "moe_combine launch");
}

extern "C" int32_t iq_rmsnorm(iq_ctx* ctx, void* stream, const float* x, int64_t ldx, void* out, int32_t out_dtype,
                              int64_t ldo, int32_t rows, int32_t d, float eps) {
    if (ctx == nullptr) return kErrInvalidArg;
    if (x == nullptr || out == nullptr || rows < 1 || d < 4 || d % 4 != 0 || ldx < d || ldo < d || ldx % 4 != 0 ||
        ldo % 4 != 0 || out_dtype < 0 || out_dtype > 2)
        return fail(ctx, kErrInvalidArg, "rmsnorm: arguments");
    return check_cuda(ctx, launch_dependent(rmsnorm_kernel, dim3(rows), 256, 0, reinterpret_cast<cudaStream_t>(stream), x, ldx, out, out_dtype, ldo, d, eps),
                      "rmsnorm launch");
}
