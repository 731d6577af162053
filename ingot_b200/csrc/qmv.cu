// Launchers of the GEMV family and the iq_qmv entry point.
#include <stdarg.h>
#include <stdio.h>

#include <stdlib.h>
#include <string.h>

#include <algorithm>

#include "gqmv.cuh"
#include "internal.h"
#include "qmv_imma.cuh"
#include "qmv_imma_grouped.cuh"
#include "qmv_ring.cuh"
#include "qmv_stream.cuh"

namespace iq {

namespace {

typedef void (*GqmvKernel)(const GqmvParams);

// (RG, WK) pairs: RG row groups of 16 rows and WK K-slices per CTA, always 8 warps.
template <int FMT, int MH, int MODE, int RG, int WK>
constexpr GqmvKernel kernel_of() {
    return gqmv_kernel<FMT, MH, (MODE == kModeGateUp ? 2 : 1), MODE, RG, WK>;
}

template <int FMT, int MH, int MODE>
GqmvKernel pick_cfg(int wk) {
    switch (wk) {
        case 8: return kernel_of<FMT, MH, MODE, 1, 8>();
        case 4: return kernel_of<FMT, MH, MODE, 2, 4>();
        default: return kernel_of<FMT, MH, MODE, 4, 2>();
    }
}

template <int FMT, int MH>
GqmvKernel pick_mode(int mode, int wk) {
    switch (mode) {
        case kModeGateUp: return pick_cfg<FMT, MH, kModeGateUp>(wk);
        default: return pick_cfg<FMT, MH, kModePlain>(wk);
    }
}

template <int FMT>
GqmvKernel pick_mh(int mh, int mode, int wk) {
    return mh == 2 ? pick_mode<FMT, 2>(mode, wk) : pick_mode<FMT, 1>(mode, wk);
}

GqmvKernel pick(int32_t fmt, int mh, int mode, int wk) {
    switch (fmt) {
        case kFmtAffine4: return pick_mh<kFmtAffine4>(mh, mode, wk);
        case kFmtAffine8: return pick_mh<kFmtAffine8>(mh, mode, wk);
        case kFmtMxfp4: return pick_mh<kFmtMxfp4>(mh, mode, wk);
        case kFmtAffine4G32: return pick_mh<kFmtAffine4G32>(mh, mode, wk);
        default: return nullptr;
    }
}

constexpr int kSmemBudget = 200 * 1024;

// ---- streaming (TMA ring) path --------------------------------------------------------------------------------------
typedef void (*QsKernel)(const QsParams);

QsKernel qs_pick(int mh, int mode) {
    if (mode == kModeGateUp) return mh == 2 ? qmv_stream_kernel<2, kModeGateUp> : qmv_stream_kernel<1, kModeGateUp>;
    return mh == 2 ? qmv_stream_kernel<2, kModePlain> : qmv_stream_kernel<1, kModePlain>;
}
constexpr int kQsSmemMax = 226 * 1024;

constexpr int kQiCtasPerSm = 2;  // two CTAs per SM where they fit (one row, one CTA with a deeper ring 10.7 against 10.0 us)

// Returns kOk after a launch, 1 when the shape does not fit this path (the caller falls back), or an error.
int32_t launch_qmv_stream(iq_ctx* ctx, cudaStream_t st, const GqmvCall& c) {
    if (c.fmt != kFmtMxfp4) return 1;
    const int nw = c.mode == kModeGateUp ? 2 : 1;
    const int mh = c.max_rows > 8 ? 2 : 1;
    const int row_bytes = c.K / 2, srow_bytes = c.K / 32, per_row = row_bytes + srow_bytes;
    for (int i = 0; i < nw; i++)
        if ((reinterpret_cast<uintptr_t>(c.w[i]) & 15) || (reinterpret_cast<uintptr_t>(c.s[i]) & 15)) return 1;
    int rgs = 1;
    while (rgs < 8 && 16 * rgs * per_row * nw < 24 * 1024 && 16 * rgs * 2 <= c.N) rgs *= 2;
    const int R = 16 * rgs;
    const int mat_bytes = round_up(R * per_row, 128);
    const int stage_bytes = nw * mat_bytes;
    const int nsteps = (row_bytes / 16 + 3) / 4;
    const int xs_bytes = round_up(nsteps * 4 * c.max_rows * 4 * 16, 128);
    const int red_bytes = 2 * 8 * nw * mh * 4 * 32 * 4;
    const int fixed = xs_bytes + red_bytes + 256;  // + barriers, abort flag, zero block
    if (stage_bytes > 80 * 1024) return 1;
    // two CTAs per SM when the activations are small: twice the warps to hide dependency and barrier stalls
    int ctas_per_sm = 1;
    int nstages = (kQsSmemMax - fixed) / stage_bytes;
    if (mh == 1 && nw == 1 && (kQsSmemMax / 2 - 1024 - fixed) / stage_bytes >= 2) {
        ctas_per_sm = 2;
        nstages = (kQsSmemMax / 2 - 1024 - fixed) / stage_bytes;
    }
    if (nstages < 2 && c.rows > 1) {
        // the rows' activations leave no room for two stages: two launches of half the rows, so that a row stays on this kernel
        // (and keeps its bits) whatever the rows of the call
        GqmvCall half = c;
        half.rows = half.max_rows = c.rows / 2;
        const int32_t r = launch_qmv_stream(ctx, st, half);
        if (r != kOk) return r;
        half.x = static_cast<const char*>(c.x) + (size_t)half.rows * c.ldx * dtype_size(c.x_dtype);
        half.y = static_cast<char*>(c.y) + (size_t)half.rows * c.ldy * dtype_size(c.y_dtype);
        half.rows = half.max_rows = c.rows - half.rows;
        return launch_qmv_stream(ctx, st, half);
    }
    if (nstages < 2) return 1;
    if (nstages > 8) nstages = 8;

    QsParams p;
    memset(&p, 0, sizeof(p));
    for (int i = 0; i < 2; i++) {
        p.w[i] = reinterpret_cast<const unsigned char*>(c.w[i] ? c.w[i] : c.w[0]);
        p.s[i] = reinterpret_cast<const unsigned char*>(c.s[i] ? c.s[i] : c.s[0]);
    }
    p.N = c.N; p.K = c.K;
    p.x = c.x; p.x_dtype = c.x_dtype; p.ldx = c.ldx;
    p.M = c.rows;
    p.y = c.y; p.y_dtype = c.y_dtype; p.ldy = c.ldy; p.accumulate = c.accumulate;
    p.limit = c.limit;
    p.act = c.act;
    p.R = R; p.NB = (c.N + R - 1) / R; p.rgs = rgs; p.wk = 8 / rgs;
    p.row_bytes = row_bytes; p.srow_bytes = srow_bytes; p.mat_bytes = mat_bytes; p.stage_bytes = stage_bytes;
    p.nstages = nstages;
    p.xs_bytes = xs_bytes; p.red_bytes = red_bytes;
    p.status = ctx->d_status;

    const int slots = ctx->sms * ctas_per_sm;
    return check_cuda(ctx, launch_dependent(qs_pick(mh, c.mode), dim3(p.NB < slots ? p.NB : slots), kQsThreads,
                                            (size_t)(fixed + nstages * stage_bytes), st, p), "qmv_stream launch");
}

// The tail split's scratch slot of a stream: launches of one stream run in series (a dependent launch waits for its
// predecessor before it touches the scratch), so a stream keeps one slot for good; streams may overlap, so each gets its
// own, and a context serves at most kQmvTailSlots of them. -1 when they are used up.
int tail_slot_of(iq_ctx* ctx, cudaStream_t st) {
    std::lock_guard<std::mutex> hold(ctx->qmv_tail_lock);
    for (int i = 0; i < ctx->qmv_tail_stream_count; i++)
        if (ctx->qmv_tail_streams[i] == static_cast<void*>(st)) return i;
    if (ctx->qmv_tail_stream_count >= kQmvTailSlots) return -1;
    ctx->qmv_tail_streams[ctx->qmv_tail_stream_count] = static_cast<void*>(st);
    return ctx->qmv_tail_stream_count++;
}

// ---- int8 tensor-core path with a ring of weights per warp: the plain GEMVs the staged kernel refuses, and the dense FFN's
// gate + up ---------------------------------------------------------------------------------------------------------
typedef void (*QrKernel)(const QrMaps, const QrParams);
template <int FMT, int NW, int MS, int LAY>
QrKernel qr_pick_v(bool vec) { return vec ? qmv_ring_kernel<FMT, MS, NW, true, LAY> : qmv_ring_kernel<FMT, MS, NW, false, LAY>; }
template <int FMT, int NW>
QrKernel qr_pick_16(int ms, bool vec) { return ms == 4 ? qr_pick_v<FMT, NW, 4, kQr16>(vec) : ms == 2 ? qr_pick_v<FMT, NW, 2, kQr16>(vec) : qr_pick_v<FMT, NW, 1, kQr16>(vec); }
template <int FMT, int NW>
QrKernel qr_pick_23(int lay, int ms, bool vec) {
    if (lay == kQr23Tall) return ms == 2 ? qr_pick_v<FMT, NW, 2, kQr23Tall>(vec) : qr_pick_v<FMT, NW, 1, kQr23Tall>(vec);
    return ms == 2 ? qr_pick_v<FMT, NW, 2, kQr23>(vec) : qr_pick_v<FMT, NW, 1, kQr23>(vec);
}
QrKernel qr_pick(int32_t fmt, int nw, int lay, int ms, bool vec) {
    if (fmt == kFmtAffine8) return nw == 2 ? qr_pick_16<kFmtAffine8, 2>(ms, vec) : qr_pick_16<kFmtAffine8, 1>(ms, vec);
    if (fmt == kFmtAffine4G32) return nw == 2 ? qr_pick_23<kFmtAffine4G32, 2>(lay, ms, vec) : qr_pick_23<kFmtAffine4G32, 1>(lay, ms, vec);
    if (lay == kQr16) return qr_pick_16<kFmtAffine4, 1>(ms, vec);
    return nw == 2 ? qr_pick_23<kFmtAffine4, 2>(lay, ms, vec) : qr_pick_23<kFmtAffine4, 1>(lay, ms, vec);
}
constexpr int kQrPreUnits = 1000;
// Shapes of a launch, by the rows it takes
struct QrShape { int lay, ms; };
constexpr QrShape kQrShapes16[3] = {{kQr16, 1}, {kQr16, 2}, {kQr16, 4}};
constexpr QrShape kQrShapes23[4] = {{kQr23, 1}, {kQr23, 2}, {kQr23Tall, 1}, {kQr23Tall, 2}};
int qr_shape_rows(QrShape h) { return h.ms * qr_rows(h.lay); }
// How a matrix is split, whatever the rows of the call (a row's bits must not depend on them).
struct QrPlan {
    int max_rows;  // rows a launch can take
    int warps, wk;
};
// wk8: eight slices of equal length, the sums of the staged kernel. wide: 23-bit digits.
QrPlan qr_plan(int32_t fmt, int N, int K, int nw, bool vec, int sms, bool wk8, bool wide) {
    QrPlan best = {0, 0, 0};
    auto fits = [&](QrShape h, int warps) { return qr_smem(fmt, K, nw, h.lay, h.ms, vec, warps, 2) <= (size_t)kQsSmemMax; };
    if (wide) {
        // as many warps as fit beside two rows; a launch with more rows takes fewer where it has to
        for (int w = kQrMaxWarps; w >= 4 && best.warps == 0; w -= 4)
            if (fits(kQrShapes23[0], w)) best.warps = w;
    } else {
        // as many row sets as fit beside at least two slots per warp, then as many warps
        for (int v = 2; v >= 0 && best.warps == 0; v--)
            for (int w = kQrMaxWarps; w >= (v > 0 ? 8 : 4); w -= wk8 ? 8 : 4)
                if (fits(kQrShapes16[v], w)) { best.max_rows = qr_shape_rows(kQrShapes16[v]); best.warps = w; break; }
    }
    if (best.warps == 0) return best;
    // K slices: the least (rounds of a CTA) x (columns of a warp in a round + the round's own cost, about one column's)
    const int gpc = qr_groups(fmt), G = K / (fmt == kFmtAffine4G32 ? 32 : 64), ncol = (G + gpc - 1) / gpc, nblk = N / 16;
    long long cost = -1;
    for (int wk = best.warps; wk >= 1; wk--) {
        if (best.warps % wk != 0 || wk > ncol || (wk8 && wk != 8)) continue;
        const long long per = (long long)(best.warps / wk) * sms, rounds = (nblk + per - 1) / per, c = rounds * ((ncol + wk - 1) / wk + 1);
        if (cost < 0 || c < cost) { cost = c; best.wk = wk; }
    }
    if (wide && best.wk > 0)
        for (int v = 0; v < 4; v++)
            for (int w = best.warps; w >= 8 || w == best.warps; w -= best.wk)
                if (fits(kQrShapes23[v], w)) { best.max_rows = qr_shape_rows(kQrShapes23[v]); break; }
    return best;
}
// Where csrc/qmv_rows.cuh takes a plain call over, one launch for any rows: by the rows that a launch here holds (max_rows: of 4-bit weights two above
// some 11000 inputs, four above 7300, eight above 4100; of 8-bit ones four above 11000, eight above 5000), and by whether the launches here share one
// conversion of the activations (pre, the dense FFN's down projection). us here / there, matrices of 300 MB in rotation:
// 4 bits, two rows a launch, 5 / 8 / 9 / 16 rows: 4096 x 14336 38.2 / 24.2, 53.7 / 27.3, 64.6 / 51.1, 106 / 62.3; 5120 x 13824 48.3 / 46.1, 67.2 / 50.5, 81.7 /
//   53.8, 134 / 65.1. Four: 4096 x 11008 30.3 / 20.3, 41.9 / 23.0, 51.0 / 24.2, 83.2 / 30.9; 2048 x 7680 15.1 / 12.8, 19.1 / 14.3, 24.4 / 16.3, 37.6 / 20.7.
//   Eight: 4096 x 5504 14.4 / 11.8, 18.1 / 13.2, 24.6 / 15.1, 36.1 / 18.8; 9216 x 5120 14.7 / 18.3, 17.2 / 20.7, 25.8 / 22.2, 33.3 / 28.8; 2048 x 5120 at 8 / 9
//   11.3 / 14.2, 16.0 / 16.2.
// 8 bits, four rows a launch, 5 / 8 / 16 rows: 4096 x 14336 36.5 / 26.9, 43.0 / 28.9, 85.5 / 35.8. Eight: 4096 x 11008 at 6 / 8 / 16 29.8 / 18.1, 34.3 / 19.4,
//   66.5 / 31.8, 4096 x 8768 at 8 / 9 22.2 / 25.6, 33.1 / 27.4, 2048 x 5504 11.6 / 12.5, 17.1 / 14.7.
// Groups of 32, two rows a launch, 6 / 8 / 9 / 16 rows: 5120 x 13824 53.9 / 56.2, 71.9 / 60.2, 87.8 / 67.7, 144 / 80.8. Four: 2048 x 7680 at 6 / 8 / 12 16.6 / 16.3,
//   19.2 / 17.6, 28.4 / 23.2, 4096 x 11008 at 8 / 9 / 12 42.7 / 28.3, 52.7 / 54.8, 63.8 / 60.6. Eight: 9216 x 5120 at 5 / 12 / 16 19.7 / 23.2, 37.4 / 33.4, 46.4 /
//   36.3, 7168 x 5376 at 12 38.8 / 40.3.
// Many features are more than a wave of clusters: 12288 x 7680 at 5 / 8 rows 36.1 / 44.4, 43.4 / 49.2 (groups of 32 at 8 / 12 45.5 / 60.5, 68.2 / 75.7), 14336 x
//   5504 at 9 / 12 43.0 / 45.5, 47.9 / 50.0. FFN with the down projection here / there: 4096 / 11008 at 9 / 16 rows 68.5 / 61.2, 88.1 / 72.4, 2048 / 7680 at 8 / 9 /
//   16 27.1 / 28.2, 36.9 / 35.9, 45.7 / 41.6. Over 350 calls the rule takes none that is slower there; it leaves some that would be faster (groups of 32 at
//   five rows of 4096 x 14336 41.8 / 29.8 or nine of 8192 x 8768 69.2 / 63.6, 4 bits at five rows of 16384 x 10240 65.5 / 55.2).
bool rows_kernel_pays(const GqmvCall& c, int nw, int max_rows, bool pre) {
    if (nw != 1 || c.rows < 5) return false;
    if (c.fmt == kFmtAffine8) {
        if (max_rows <= 4) return c.N <= 16384 || c.rows > 12;  // (30000 x 12288 at 7 / 12 / 14 rows 153.8 / 157.2, 229.9 / 234.2, 302.9 / 249.3)
        return !pre && max_rows == 8 && c.N <= 4096 && (c.rows > 8 || (c.rows > 5 && c.K >= 9200));
    }
    if (c.fmt == kFmtAffine4G32) {
        if (max_rows <= 2) return c.N <= 8192 && c.rows > 6 && (!pre || c.rows <= 8 || c.rows > 13);
        if (pre || max_rows > 8) return false;
        return max_rows <= 4 ? c.N <= 8192 && (c.rows > 11 || ((c.rows == 7 || c.rows == 8) && c.K >= 7500)) : c.N >= 4096 && c.N <= 9216 && c.rows > 12;
    }
    if (max_rows <= 2) return !pre || c.rows <= 8 || c.rows > 12;
    if (max_rows <= 4) {
        if (pre) return c.N <= 4096 && (c.rows > 12 || (c.rows > 8 && c.K >= 9200));
        return c.N <= 8192 || c.rows > 12;
    }
    return !pre && max_rows <= 8 && ((c.rows > 8 && c.N >= 4096 && c.N <= 9216) || (c.K >= 5500 && c.N <= 4096));
}
// Returns kOk after a launch, 1 when the shape does not fit this path (the caller falls back), or an error.
int32_t launch_qmv_ring(iq_ctx* ctx, cudaStream_t st, const GqmvCall& c, bool wk8 = false) {
    if (c.rows < 1 || c.rows > 16 || c.N % 16 != 0 || c.K % 64 != 0 || ctx->encode_tiled == nullptr) return 1;
    if (c.fmt != kFmtAffine4 && c.fmt != kFmtAffine4G32 && c.fmt != kFmtAffine8) return 1;
    const int nw = c.mode == kModeGateUp ? 2 : 1, gpc = qr_groups(c.fmt), G = c.K / (c.fmt == kFmtAffine4G32 ? 32 : 64);
    const bool wide = c.fmt != kFmtAffine8 && !wk8;
    bool vec = G % gpc == 0;
    QrParams p;
    memset(&p, 0, sizeof(p));
    for (int i = 0; i < nw; i++) {
        p.s[i] = static_cast<const unsigned char*>(c.s[i]);
        p.b[i] = static_cast<const unsigned char*>(c.b[i]);
        const uintptr_t sb = reinterpret_cast<uintptr_t>(p.s[i]) | reinterpret_cast<uintptr_t>(p.b[i]);
        if ((reinterpret_cast<uintptr_t>(c.w[i]) & 15) || (sb & 3)) return 1;
        if (sb & (uintptr_t)(2 * gpc - 1)) vec = false;
    }
    const QrPlan plan = qr_plan(c.fmt, c.n_full > 0 ? c.n_full : c.N, c.K, nw, vec, ctx->sms, wk8, wide);
    if (plan.max_rows == 0 || plan.wk == 0) return 1;
    // The activations: every CTA converts them, or one more kernel does it for all where that is shorter (a CTA takes about
    // 1 us per 2000 units of eight inputs, the kernel 1.5 us)
    const int units = c.rows * (c.K / 8);
    const bool pre = c.scratch != nullptr && units > kQrPreUnits;
    if (!wk8 && rows_kernel_pays(c, nw, plan.max_rows, pre)) {
        const int32_t r = launch_qmv_rows(ctx, st, c, plan.wk);
        if (r != 1) return r;
    }
    const int row_bytes = c.fmt == kFmtAffine8 ? c.K : c.K / 2;
    QrMaps maps = {};
    for (int i = 0; i < nw; i++) {
        const int32_t r = cached_rows_map(ctx, c.w[i], c.N, row_bytes, 16, &maps.w[i]);
        if (r != kOk) return r;
    }
    p.N = c.N; p.K = c.K;
    p.x_dtype = c.x_dtype; p.ldx = c.ldx;
    p.y_dtype = c.y_dtype; p.ldy = c.ldy; p.accumulate = c.accumulate;
    p.act = c.act; p.limit = c.limit;
    p.wk = plan.wk;
    p.runs = wk8 ? 1 : 0;
    p.status = ctx->d_status;
    const size_t xes = c.x_dtype == kF32 ? 4 : 2, yes = c.y_dtype == kF32 ? 4 : 2;
    const size_t rec = (size_t)G * qr_record(c.fmt == kFmtAffine4G32, wide ? kQr23 : kQr16);  // bytes of a row's digits
    if (pre) {
        unsigned char* digits = static_cast<unsigned char*>(c.scratch);
        float2* scale = reinterpret_cast<float2*>(digits + c.rows * rec);
        auto k = c.fmt == kFmtAffine8 ? qr_convert_kernel<true, false, false> : c.fmt == kFmtAffine4G32 ? qr_convert_kernel<false, true, true>
               : wide ? qr_convert_kernel<false, false, true> : qr_convert_kernel<false, false, false>;
        const int32_t r = check_cuda(ctx, launch_dependent(k, dim3((units + 255) / 256), 256, 0, st, c.x, c.x_dtype, c.ldx, c.K, c.rows, wk8 ? 7 : 8, digits, scale), "qr_convert launch");
        if (r != kOk) return r;
        p.xd = digits;
        p.xs = scale;
    }
    for (int m0 = 0; m0 < c.rows;) {
        const QrShape* h = wide ? kQrShapes23 : kQrShapes16;
        while (qr_shape_rows(*h) < plan.max_rows && qr_shape_rows(*h) < c.rows - m0) h++;
        auto smem = [&](int warps, int depth) { return qr_smem(c.fmt, c.K, nw, h->lay, h->ms, vec, warps, depth); };
        int warps = plan.warps;
        while (smem(warps, 2) > (size_t)kQsSmemMax) warps -= plan.wk;  // (23 bits: a multiple of the slices that fits, the plan saw to it)
        p.M = std::min(c.rows - m0, qr_shape_rows(*h));
        p.x = static_cast<const char*>(c.x) + (size_t)m0 * c.ldx * xes;
        p.y = static_cast<char*>(c.y) + (size_t)m0 * c.ldy * yes;
        p.depth = 2;
        while (p.depth < 6 && smem(warps, p.depth + 1) <= (size_t)kQsSmemMax) p.depth++;
        const int nsup = (c.N / 16 + warps / plan.wk - 1) / (warps / plan.wk);
        const int32_t r = check_cuda(ctx, launch_dependent(qr_pick(c.fmt, nw, h->lay, h->ms, vec), dim3(std::min(nsup, ctx->sms)), warps * 32,
                                                           smem(warps, p.depth), st, maps, p), "qmv_ring launch");
        if (r != kOk) return r;
        if (pre) { p.xd += p.M * rec; p.xs += (size_t)p.M * G * (wide ? 2 : 1); }
        m0 += p.M;
    }
    return kOk;
}

// ---- int8 tensor-core path (decode, up to four rows, affine codes) -----------------------------------------------
// How it cuts K inputs of 4-, 6- or 8-bit codes; `fits`: two stages beside what eight rows need, whatever the row count of the call: a row must
// see the same arithmetic alone and among sixteen.
struct QiCut {
    bool tm, pair, fits;
    int row_bytes, row_pitch, stage_bytes;
};
constexpr int kQiConsumers = 8;  // warps (16 measured slower: 11.3 against 10.0 us on the 14336 x 4096 layer)
// (+ 1024: the stages of the tensor copies start on a 1024-byte boundary)
int qi_fixed_bytes(int K, bool tm, int ms) { return K / 64 * 544 * ms + 512 * ms * kQiConsumers + 256 + (tm ? 1024 : 0); }
QiCut qi_cut(int32_t fmt, int K, bool tensor_copies) {
    const bool w8 = fmt == kFmtAffine8, w6 = fmt == kFmtAffine6;
    QiCut c;
    c.row_bytes = w8 ? K : (w6 ? K / 4 * 3 : K / 2);
    // 4-bit codes with rows of 1 KB (K = 2048): one swizzled tensor copy per block of 16 rows, no padding (the swizzle
    // spreads the rows over the banks). Otherwise one bulk copy per row (4-bit) or per pair of rows (6- and 8-bit), padded apart by a quad's piece.
    c.tm = fmt == kFmtAffine4 && c.row_bytes <= 1024 && tensor_copies;
    c.pair = w8 || w6;  // two rows per bulk copy
    c.row_pitch = c.tm ? c.row_bytes : (c.pair ? 2 : 1) * c.row_bytes + (w8 ? 64 : (w6 ? 48 : 32));
    c.stage_bytes = (c.tm ? kQiRows * c.row_bytes : (c.pair ? kQiRows / 2 : kQiRows) * c.row_pitch) + 2 * kQiRows * (K / 64 * 2);
    c.fits = K % 2048 == 0 && (kQsSmemMax - qi_fixed_bytes(K, c.tm, 2)) / c.stage_bytes >= 2;
    return c;
}
// Returns kOk after a launch, 1 when the shape does not fit this path (the caller falls back), or an error.
int32_t launch_qmv_imma(iq_ctx* ctx, cudaStream_t st, const GqmvCall& c) {
    if (c.mode != kModePlain || c.rows > 16 || c.rows < 1) return 1;
    if (c.fmt != kFmtAffine4 && c.fmt != kFmtAffine8 && c.fmt != kFmtAffine6) return 1;
    const QiCut cut = qi_cut(c.fmt, c.K, ctx->encode_tiled != nullptr);
    if (!cut.fits || c.N < kQiRows) return 1;
    if ((reinterpret_cast<uintptr_t>(c.w[0]) & 15) || (reinterpret_cast<uintptr_t>(c.s[0]) & 15) ||
        (reinterpret_cast<uintptr_t>(c.b[0]) & 15))
        return 1;
    const bool w8 = c.fmt == kFmtAffine8, w6 = c.fmt == kFmtAffine6, tm = cut.tm;
    const int G = c.K / 64;
    QiParams p;
    memset(&p, 0, sizeof(p));
    p.row_bytes = cut.row_bytes;
    p.pair = cut.pair ? 1 : 0;
    p.row_pitch = cut.row_pitch;
    p.srow_bytes = G * 2;
    p.srow_pitch = p.srow_bytes;
    p.stage_bytes = cut.stage_bytes;
    constexpr int ncw = kQiConsumers;
    auto fixed_bytes = [&](int ms) { return qi_fixed_bytes(c.K, tm, ms); };
    p.w = reinterpret_cast<const unsigned char*>(c.w[0]);
    p.s = reinterpret_cast<const unsigned char*>(c.s[0]);
    p.b = reinterpret_cast<const unsigned char*>(c.b[0]);
    p.N = c.N; p.K = c.K;
    p.x_dtype = c.x_dtype; p.ldx = c.ldx;
    p.y_dtype = c.y_dtype; p.ldy = c.ldy; p.accumulate = c.accumulate;
    p.status = ctx->d_status;
    CUtensorMap wmap = {};
    const CUtensorMap* map = &wmap;
    if (tm) {
        // the matrix as the kernel sees it: all rows of W, whatever prefix of them this call computes (one cached map
        // per matrix, not one per prefix)
        const int32_t r = cached_rowblock_map(ctx, p.w, c.n_full > c.N ? c.n_full : c.N, p.row_bytes, kQiRows, &wmap);
        if (r != kOk) return r;
    }
    const int blocks = c.N / kQiRows;
    // Tail split, decided from the output features this call computes and the GPU alone (not from the activation row
    // count, so an activation row sees the same arithmetic alone and among sixteen; a call with n_prefix may split
    // differently from a call over the whole matrix): when the blocks do not divide over two CTAs per SM and few are
    // left over, the left-over blocks are cut into K slices and dealt out one piece per CTA.
    const int slots = 2 * ctx->sms;
    const int per2 = blocks / slots, tail = blocks - per2 * slots;
    int tail_slices = 0;
    if (c.N % kQiRows == 0 && per2 >= 1 && tail > 0 && tail * 8 <= slots && tail <= kQmvTailBlocks) {
        tail_slices = 1;
        while (tail_slices * 2 * tail <= slots && tail_slices * 2 <= 32 && G % (tail_slices * 2) == 0) tail_slices *= 2;
        if (tail_slices < 8 || tail * tail_slices > kQmvTailPieces) tail_slices = 0;
    }
    // Nine to sixteen rows: the ring kernel reads the weights once, with the same K slices and order of sums (14336 x 4096 at 4
    // bits and 16 rows 50.1 -> 33.5 us, 8 bits 56.0 -> 40.7); up to eight this kernel's deeper staging is level or ahead (one
    // row 9.2 against 13.2). Left-over blocks are summed by pieces, so a matrix that has them stays here.
    if (c.rows > 8 && tail_slices == 0 && !w6) {
        const int32_t r = launch_qmv_ring(ctx, st, c, true);
        if (r != 1) return r;
    }
    const size_t xes = c.x_dtype == kF32 ? 4 : 2, yes = c.y_dtype == kF32 ? 4 : 2;
    for (int m0 = 0; m0 < c.rows; m0 += 8) {  // nine to sixteen rows: two launches of up to eight
        const int m = c.rows - m0 < 8 ? c.rows - m0 : 8;
        const int ms = m > 4 ? 2 : 1;
        p.M = m;
        p.x = static_cast<const char*>(c.x) + (size_t)m0 * c.ldx * xes;
        p.y = static_cast<char*>(c.y) + (size_t)m0 * c.ldy * yes;
        p.xq_bytes = G * 512 * ms;
        p.xsc_bytes = G * 32 * ms;
        p.red_bytes = 512 * ms * ncw;
        p.ncw = ncw;
        // Two CTAs per SM when each still gets two stages: with the ten warps of one, a scheduler issued in 42 of 100 cycles (eight rows of a
        // 128,000 x 2048 6-bit head with arg-max 70.2 -> 62.9 us, of a 151,936 x 2048 4-bit one with candidates 88.1 -> 78.4)
        int ctas = 1;
        if (kQiCtasPerSm == 2 && (kQsSmemMax / 2 - 1024 - fixed_bytes(ms)) / p.stage_bytes >= 2) ctas = 2;
        int nstages = ((ctas == 2 ? kQsSmemMax / 2 - 1024 : kQsSmemMax) - fixed_bytes(ms)) / p.stage_bytes;
        if (nstages > 8) nstages = 8;
        p.nstages = nstages;
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3(blocks < ctx->sms * ctas ? blocks : ctx->sms * ctas, 1, 1);
        p.tail_blocks = 0;
        if (tail_slices > 0) {
            const int slot = tail_slot_of(ctx, st);
            if (slot < 0)
                return fail(ctx, kErrInvalidArg, "qmv: more than %d streams launch GEMVs with a tail split on this context",
                            kQmvTailSlots);
            p.tail_blocks = tail;
            p.tail_slices = tail_slices;
            p.blocks_per_cta = per2 * (2 / ctas);
            p.tail_scratch = ctx->qmv_tail_scratch + (size_t)slot * kQmvTailPieces * 2 * 64;
            p.tail_counters = ctx->qmv_tail_counters + (size_t)slot * kQmvTailBlocks;
            cfg.gridDim = dim3(ctx->sms * ctas, 1, 1);
        }
        cfg.blockDim = dim3(32 * (ncw + 2), 1, 1);
        cfg.dynamicSmemBytes = fixed_bytes(ms) + nstages * p.stage_bytes;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        // up to four rows and eight or four groups per warp (K = 4096, 2048): the activation fragments stay in registers
        const int gwh = ms == 1 ? G / ncw : 0;
        cudaError_t e;
#define IQ_QI_LAUNCH(F)                                                                             \
    (ms == 2 ? cudaLaunchKernelEx(&cfg, qmv_imma_kernel<F, 2, 0>, *map, p)                          \
             : gwh == 8 ? cudaLaunchKernelEx(&cfg, qmv_imma_kernel<F, 1, 8>, *map, p)               \
                        : gwh == 4 ? cudaLaunchKernelEx(&cfg, qmv_imma_kernel<F, 1, 4>, *map, p)    \
                                   : cudaLaunchKernelEx(&cfg, qmv_imma_kernel<F, 1, 0>, *map, p))
        if (tm) e = ms == 2 ? cudaLaunchKernelEx(&cfg, qmv_imma_kernel<kFmtAffine4, 2, 0, true>, *map, p)
                            : cudaLaunchKernelEx(&cfg, qmv_imma_kernel<kFmtAffine4, 1, 4, true>, *map, p);
        else if (w6) e = IQ_QI_LAUNCH(kFmtAffine6);
        else if (w8) e = IQ_QI_LAUNCH(kFmtAffine8);
        else e = IQ_QI_LAUNCH(kFmtAffine4);
#undef IQ_QI_LAUNCH
        const int32_t r = check_cuda(ctx, e, "qmv_imma launch");
        if (r != kOk) return r;
    }
    return kOk;
}

// ---- int8 tensor-core path of the expert-parallel pieces (gate/up + activation, down; affine 4-bit experts) ---------------
typedef void (*QgKernel)(const CUtensorMap, const CUtensorMap, const QgParams);
// gw4: each consumer warp's K slice is four groups, its activation fragments stay in registers
// (the two-wide fp32 form costs registers: it pays in the down projections)
QgKernel qg_pick(int mode, bool gw4) {
    if (mode == kModeGateUp) return gw4 ? qmv_imma_grouped_kernel<kModeGateUp, 4, false> : qmv_imma_grouped_kernel<kModeGateUp, 0, false>;
    return gw4 ? qmv_imma_grouped_kernel<kModeDown, 4, true> : qmv_imma_grouped_kernel<kModeDown, 0, true>;
}

// How a call is cut. K slices per block of rows: one slice of four groups per warp when K allows it (the activation
// fragments then live in registers: 69 against 83 us on the 64-token layer); else four slices (32-row blocks: half as
// many hand-overs per byte) when two stages of that size fit, else eight.
struct QgCut {
    int wk, nstages;  // (fewer than two stages: the shape does not fit)
    int srow_bytes, xq_bytes, xsc_bytes, red_bytes, fixed, mat_bytes;
};
QgCut qg_cut(int K, int nw) {
    constexpr int ms = 2;  // sets of four activation rows per tile
    const int G = K / 64, row_bytes = K / 2;
    QgCut c = {};
    if (K % 256 != 0 || K > 65536) return c;  // (tensor copies: whole columns of 128 bytes, up to 256 of them)
    c.srow_bytes = G * 2;
    c.xq_bytes = G * ms * 512;
    c.xsc_bytes = G * ms * 32;
    c.red_bytes = 2 * kQgWarps * nw * ms * 64 * 4;
    c.fixed = c.xq_bytes + c.xsc_bytes + c.red_bytes + 256 + 1024;
    const bool gw4 = G == 4 * kQgWarps;
    const int cand[4] = {gw4 ? kQgWarps : kQgWarps / 2, kQgWarps, kQgWarps / 4, kQgWarps / 8};
    for (int ci = 0; ci < 4 && c.nstages < 2; ci++) {
        const int wk = cand[ci];
        if (G % wk != 0 || (G / wk) % 4 != 0) continue;  // a warp's K slice: runs of four groups
        const int R = 16 * (kQgWarps / wk);
        if ((R * c.srow_bytes) % 16 != 0) continue;
        c.wk = wk;
        c.mat_bytes = round_up(R * row_bytes + 2 * R * c.srow_bytes, 1024);
        c.nstages = (kQsSmemMax - c.fixed) / (nw * c.mat_bytes);
    }
    return c;
}
}  // namespace

int qmv_grouped_slices(int K, int nw) {
    const QgCut c = qg_cut(K, nw);
    return c.nstages >= 2 ? c.wk : 0;
}

// Returns kOk after a launch, 1 when the shape does not fit this path (the caller falls back), or an error.
int32_t launch_qmv_imma_grouped(iq_ctx* ctx, cudaStream_t st, const GqmvCall& c) {
    if ((c.mode != kModeGateUp && c.mode != kModeDown) || c.tiles == nullptr || c.fmt != kFmtAffine4) return 1;
    if (c.N % 16 != 0 || c.max_rows > 8 || c.accumulate || ctx->encode_tiled == nullptr) return 1;
    const int nw = c.mode == kModeGateUp ? 2 : 1;
    for (int i = 0; i < nw; i++)
        if ((reinterpret_cast<uintptr_t>(c.w[i]) & 15) || (reinterpret_cast<uintptr_t>(c.s[i]) & 15) ||
            (reinterpret_cast<uintptr_t>(c.b[i]) & 15))
            return 1;
    const int G = c.K / 64;
    QgParams p;
    memset(&p, 0, sizeof(p));
    p.row_bytes = c.K / 2;
    const QgCut cut = qg_cut(c.K, nw);
    if (cut.nstages < 2) return 1;
    const int nstages = cut.nstages < 8 ? cut.nstages : 8, R = 16 * (kQgWarps / cut.wk), fixed = cut.fixed;
    p.srow_bytes = cut.srow_bytes;
    p.xq_bytes = cut.xq_bytes; p.xsc_bytes = cut.xsc_bytes; p.red_bytes = cut.red_bytes;
    p.wk = cut.wk; p.rgs = kQgWarps / cut.wk;
    p.NB = (c.N + R - 1) / R;
    p.mat_bytes = cut.mat_bytes; p.stage_bytes = nw * cut.mat_bytes;
    p.nstages = nstages;
    for (int i = 0; i < 2; i++) {
        p.s[i] = reinterpret_cast<const unsigned char*>(c.s[i] ? c.s[i] : c.s[0]);
        p.b[i] = reinterpret_cast<const unsigned char*>(c.b[i] ? c.b[i] : c.b[0]);
        p.ebias[i] = c.ebias[i];
    }
    p.s_ebytes = c.s_estride * 2;
    p.expert_lo = c.expert_lo;
    CUtensorMap wmaps[2] = {};
    for (int i = 0; i < nw; i++) {
        const int32_t r = cached_rowblock_map(ctx, c.w[i] + (int64_t)c.expert_lo * c.w_estride, (int64_t)c.expert_count * c.N, p.row_bytes, 16 * p.rgs, &wmaps[i]);
        if (r != kOk) return r;
    }
    p.N = c.N; p.K = c.K;
    p.x = c.x; p.x_dtype = c.x_dtype; p.ldx = c.ldx;
    p.row_map = c.row_map;
    p.tiles = c.tiles; p.ntiles = c.ntiles;
    p.y = c.y; p.y_dtype = c.y_dtype; p.ldy = c.ldy;
    p.limit = c.limit;
    p.act = c.act;
    p.status = ctx->d_status;
    const int64_t items = (int64_t)p.NB * c.grid_tiles;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)(items < ctx->sms ? items : ctx->sms), 1, 1);
    cfg.blockDim = dim3(kQgThreads, 1, 1);
    cfg.dynamicSmemBytes = fixed + nstages * p.stage_bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return check_cuda(ctx, cudaLaunchKernelEx(&cfg, qg_pick(c.mode, G == 4 * kQgWarps && p.wk == kQgWarps), wmaps[0], wmaps[1], p), "qmv_imma_grouped launch");
}

int32_t gqmv_init(iq_ctx* ctx) {
#define IQ_QI_ALL(F)                                                                                           \
    reinterpret_cast<const void*>(qmv_imma_kernel<F, 1, 0>), reinterpret_cast<const void*>(qmv_imma_kernel<F, 1, 4>), \
        reinterpret_cast<const void*>(qmv_imma_kernel<F, 1, 8>), reinterpret_cast<const void*>(qmv_imma_kernel<F, 2, 0>)
    const void* qi[14] = {IQ_QI_ALL(kFmtAffine4), IQ_QI_ALL(kFmtAffine8), IQ_QI_ALL(kFmtAffine6),
                          reinterpret_cast<const void*>(qmv_imma_kernel<kFmtAffine4, 1, 4, true>),
                          reinterpret_cast<const void*>(qmv_imma_kernel<kFmtAffine4, 2, 0, true>)};
#undef IQ_QI_ALL
    for (int i = 0; i < 14; i++) {
        cudaError_t e = cudaFuncSetAttribute(qi[i], cudaFuncAttributeMaxDynamicSharedMemorySize, kQsSmemMax);
        if (e != cudaSuccess) return check_cuda(ctx, e, "cudaFuncSetAttribute(qmv_imma)");
    }
    for (int mode = kModeGateUp; mode <= kModeDown; mode++)
        for (int v = 0; v < 2; v++) {  // activations in registers or not
            cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(qg_pick(mode, v == 1)),
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, kQsSmemMax);
            if (e != cudaSuccess) return check_cuda(ctx, e, "cudaFuncSetAttribute(qmv_imma_grouped)");
        }
    for (int v = 0; v < 44; v++) {  // formats and shapes, one and two matrices, scales in one piece or not
        const int i = v >> 2;
        const int32_t fmt = i < 3 ? kFmtAffine8 : i < 7 ? kFmtAffine4G32 : kFmtAffine4;
        const QrShape h = i < 3 ? kQrShapes16[i] : kQrShapes23[(i - 3) % 4];
        cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(qr_pick(fmt, 1 + (v & 1), h.lay, h.ms, (v & 2) != 0)),
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, kQsSmemMax);
        if (e == cudaSuccess && i < 3)  // 4 bits in the staged kernel's place
            e = cudaFuncSetAttribute(reinterpret_cast<const void*>(qr_pick(kFmtAffine4, 1, h.lay, h.ms, (v & 2) != 0)),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, kQsSmemMax);
        if (e != cudaSuccess) return check_cuda(ctx, e, "cudaFuncSetAttribute(qmv_ring)");
    }
    for (int fmt = 0; fmt < 4; fmt++)
        for (int mh = 1; mh <= 2; mh++)
            for (int mode = kModePlain; mode <= kModeGateUp; mode++)
                for (int wk = 2; wk <= 8; wk *= 2) {
                    GqmvKernel k = pick(fmt, mh, mode, wk);
                    cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(k),
                                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget + 20480);
                    if (e != cudaSuccess) return check_cuda(ctx, e, "cudaFuncSetAttribute(gqmv)");
                }
    for (int mh = 1; mh <= 2; mh++)
        for (int mode = kModePlain; mode <= kModeGateUp; mode++) {
            cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(qs_pick(mh, mode)),
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, kQsSmemMax);
            if (e != cudaSuccess) return check_cuda(ctx, e, "cudaFuncSetAttribute(qmv_stream)");
        }
    return kOk;
}

int32_t launch_gqmv(iq_ctx* ctx, cudaStream_t st, const GqmvCall& c) {
    // One kernel per (format, shape), chosen from the matrix alone: for affine codes the int8 tensor-core kernels (staged
    // where K fits the staging, else with a ring per warp), the streaming fp16 kernel for MXFP4, the register-staged
    // fp16 kernel where K is too wide for either.
    int32_t r = launch_qmv_imma(ctx, st, c);
    if (r != 1) return r;
    r = launch_qmv_ring(ctx, st, c);
    if (r != 1) return r;
    r = launch_qmv_stream(ctx, st, c);
    if (r != 1) return r;
    if (c.fmt == kFmtAffine6)
        return fail(ctx, kErrUnsupported, "qmv: 6-bit weights run on the int8 kernel only (a plain GEMV, k a multiple of 2048, n >= 16)");
    const int ck = c.fmt == kFmtAffine8 ? 16 : 32;  // inputs per 16-byte chunk
    const int mh = c.max_rows > 8 ? 2 : 1;
    const int nw = c.mode == kModeGateUp ? 2 : 1;
    // K tile: everything at once when the staged activations of sixteen rows fit, else the largest multiple of 1024 that does
    // (whatever the rows of this call: the tiles, and the slices inside them, set the order of a row's sums)
    int kt = c.K;
    auto smem_for = [&](int ktile, int rows, int* xs_bytes) {
        const int nsteps = (ktile / ck + 3) / 4;
        const int qu = ck == 32 ? 4 : 2;
        *xs_bytes = nsteps * qu * rows * 4 * 16;
        const int red_bytes = 8 * nw * (rows > 8 ? 2 : 1) * 4 * 32 * 4;
        return *xs_bytes + red_bytes;
    };
    int xs_bytes;
    while (smem_for(kt, 16, &xs_bytes) > kSmemBudget) {
        kt = kt > 1024 ? (kt - 1) / 1024 * 1024 : 0;
        if (kt == 0) return fail(ctx, kErrInvalidArg, "qmv: activations do not fit shared memory");
    }
    const int smem = smem_for(kt, c.max_rows, &xs_bytes);

    // K slices per CTA: the fewest that still fill the GPU, keeping at least two steps per warp
    const int nsteps = (kt / ck + 3) / 4;
    const int64_t row_groups = c.N / 16;
    const int64_t target = (int64_t)ctx->sms * 24;
    int wk = 2;
    while (wk < 8 && row_groups * wk < target && nsteps / (wk * 2) >= 2) wk *= 2;
    const int rg = 8 / wk;

    GqmvKernel k = pick(c.fmt, mh, c.mode, wk);
    if (k == nullptr) return fail(ctx, kErrNoKernel, "qmv: no kernel for format %d", c.fmt);

    GqmvParams p;
    for (int i = 0; i < 2; i++) {
        p.w[i] = c.w[i] ? c.w[i] : c.w[0];
        p.s[i] = c.s[i] ? c.s[i] : c.s[0];
        p.b[i] = c.b[i] ? c.b[i] : c.b[0];
    }
    p.N = c.N; p.K = c.K;
    p.x = c.x; p.x_dtype = c.x_dtype; p.ldx = c.ldx;
    p.M = c.rows;
    p.y = c.y; p.y_dtype = c.y_dtype; p.ldy = c.ldy; p.accumulate = c.accumulate;
    p.limit = c.limit;
    p.act = c.act;
    p.kt = kt; p.xs_bytes = xs_bytes;

    dim3 grid((c.N / 16 + rg - 1) / rg);
    k<<<grid, 256, smem, st>>>(p);
    return check_cuda(ctx, cudaGetLastError(), "gqmv launch");
}

int32_t format_of(const iq_qlinear* m) {
    if (m->mode == IQ_MODE_MXFP4) return (m->bits == 4 && m->group == 32) ? kFmtMxfp4 : -1;
    if (m->mode != IQ_MODE_AFFINE) return -1;
    if (m->group == 32) return m->bits == 4 ? kFmtAffine4G32 : -1;
    if (m->group == 128) return m->bits == 2 ? kFmtTernary : -1;
    if (m->group != 64) return -1;
    if (m->bits == 6) return kFmtAffine6;
    if (m->bits == 4) return kFmtAffine4;
    if (m->bits == 8) return kFmtAffine8;
    return -1;
}

}  // namespace iq

using namespace iq;

int32_t iq::qmv_with_scratch(iq_ctx* ctx, void* stream, const void* x, int32_t x_dtype, int64_t ldx, const iq_qlinear* m, void* y,
                             int32_t y_dtype, int64_t ldy, int32_t rows, uint32_t flags, int32_t n_prefix, void* scratch) {
    if (ctx == nullptr) return kErrInvalidArg;
    if (x == nullptr || y == nullptr || m == nullptr || m->w == nullptr || m->scales == nullptr)
        return fail(ctx, kErrInvalidArg, "qmv: null pointer");
    const int32_t fmt = format_of(m);
    if (fmt < 0)
        return fail(ctx, kErrUnsupported, "qmv: %d-bit group %d mode %d has no kernel (affine 4/6/8-bit g64, 4-bit g32, ternary 2-bit g128, mxfp4 g32)",
                    m->bits, m->group, m->mode);
    if (fmt != kFmtMxfp4 && fmt != kFmtTernary && m->biases == nullptr)
        return fail(ctx, kErrInvalidArg, "qmv: affine layer without biases");
    if (rows < 1 || rows > 16) return fail(ctx, kErrInvalidArg, "qmv: rows = %d (1..16)", rows);
    if (m->n % 16 != 0 || m->k % 64 != 0 || m->n <= 0 || m->k <= 0)
        return fail(ctx, kErrInvalidArg, "qmv: n = %d must be a multiple of 16 and k = %d of 64", m->n, m->k);
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return fail(ctx, kErrInvalidArg, "qmv: dtype");
    if (ldx < m->k || ldx % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0)
        return fail(ctx, kErrInvalidArg, "qmv: x must be 16-byte aligned with ldx >= k and ldx %% 8 == 0");
    int32_t n = m->n;
    if (n_prefix > 0) {
        if (n_prefix % 16 != 0 || n_prefix > m->n) return fail(ctx, kErrInvalidArg, "qmv: n_prefix = %d", n_prefix);
        n = n_prefix;
    }
    if (ldy < n) return fail(ctx, kErrInvalidArg, "qmv: ldy = %lld < n", (long long)ldy);
    if (fmt == kFmtTernary)  // the rotated ternary format has kernels of its own (csrc/tern.cu)
        return launch_tern_qmv(ctx, reinterpret_cast<cudaStream_t>(stream), x, x_dtype, ldx, m, y, y_dtype, ldy, rows, n,
                               (flags & IQ_FLAG_ACCUMULATE) ? 1 : 0);
    GqmvCall c;
    c.mode = kModePlain;
    c.fmt = fmt;
    c.w[0] = reinterpret_cast<const uint32_t*>(m->w);
    c.s[0] = m->scales;
    c.b[0] = m->biases;
    c.N = n;
    c.n_full = m->n;
    c.K = m->k;
    c.x = x; c.x_dtype = x_dtype; c.ldx = ldx;
    c.rows = rows; c.max_rows = rows; c.grid_tiles = 1;
    c.y = y; c.y_dtype = y_dtype; c.ldy = ldy;
    c.accumulate = (flags & IQ_FLAG_ACCUMULATE) ? 1 : 0;
    c.scratch = scratch;
    return launch_gqmv(ctx, reinterpret_cast<cudaStream_t>(stream), c);
}

extern "C" int32_t iq_qmv_plan(const iq_qlinear* m, int32_t rows, int32_t sms, const int32_t clusters_at_once[3], iq_qmv_tiling* out) {
    if (m == nullptr || out == nullptr || clusters_at_once == nullptr || rows < 1 || rows > 16 || sms < 1 || m->n < 16 || m->n % 16 != 0 || m->k < 64 || m->k % 64 != 0)
        return kErrInvalidArg;
    const int at_once[3] = {clusters_at_once[0], clusters_at_once[1], clusters_at_once[2]};
    for (int n : at_once)
        if (n < 1) return kErrInvalidArg;
    memset(out, 0, sizeof(*out));
    GqmvCall c;
    c.fmt = format_of(m); c.rows = rows; c.N = m->n; c.K = m->k;
    if (c.fmt < 0) return kErrUnsupported;
    if (c.fmt != kFmtAffine4 && c.fmt != kFmtAffine4G32 && c.fmt != kFmtAffine8) return kOk;
    if (c.fmt != kFmtAffine4G32 && qi_cut(c.fmt, c.K, true).fits) return kOk;
    const bool vec = c.K / (c.fmt == kFmtAffine4G32 ? 32 : 64) % qr_groups(c.fmt) == 0;
    const QrPlan plan = qr_plan(c.fmt, c.N, c.K, 1, vec, sms, false, c.fmt != kFmtAffine8);
    if (plan.max_rows == 0 || plan.wk == 0 || !rows_kernel_pays(c, 1, plan.max_rows, false)) return kOk;
    out->cluster = qmv_rows_cluster(at_once, c.fmt, rows, c.N, c.K, plan.wk);
    if (out->cluster > 0) { out->tiles = (c.N + 127) / 128; out->slices = plan.wk; }
    return kOk;
}

extern "C" int32_t iq_qmv(iq_ctx* ctx, void* stream, const void* x, int32_t x_dtype, int64_t ldx, const iq_qlinear* m,
                          void* y, int32_t y_dtype, int64_t ldy, int32_t rows, uint32_t flags, int32_t n_prefix) {
    return qmv_with_scratch(ctx, stream, x, x_dtype, ldx, m, y, y_dtype, ldy, rows, flags, n_prefix, nullptr);
}
