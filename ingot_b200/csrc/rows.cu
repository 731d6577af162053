// Launcher of the decode linears of several rows and wide inputs on tcgen05 integers (csrc/qmv_rows.cuh).
#include <string.h>

#include <algorithm>

#include "gqmv.cuh"
#include "internal.h"
#include "qmv_rows.cuh"

namespace iq {

namespace {
typedef void (*QwKernel)(const CUtensorMap, const QwParams);
QwKernel qw_pick(int32_t fmt, int t) {
    if (fmt == kFmtAffine8) return t == 8 ? qmv_rows_kernel<kFmtAffine8, 8> : qmv_rows_kernel<kFmtAffine8, 16>;
    if (fmt == kFmtAffine4G32) return t == 8 ? qmv_rows_kernel<kFmtAffine4G32, 8> : qmv_rows_kernel<kFmtAffine4G32, 16>;
    return t == 8 ? qmv_rows_kernel<kFmtAffine4, 8> : qmv_rows_kernel<kFmtAffine4, 16>;
}

// How a call is cut: CTAs per tile (0: it does not fit), stages, columns of a CTA. at_once: clusters of two, four and eight CTAs that run at once
struct QwPlan {
    int cluster, stages, xcols;
    size_t smem;
};
QwPlan qw_plan(const int (&at_once)[3], int32_t fmt, int t, int N, int K, int wk) {
    const int ci = fmt == kFmtAffine8 ? 128 : 256, gpc = fmt == kFmtAffine8 ? 2 : fmt == kFmtAffine4G32 ? 8 : 4, nd = fmt == kFmtAffine8 ? 2 : 3;
    const int ncol = (K + ci - 1) / ci, tiles = (N + 127) / 128, stage = kQtCodes + 2 * 128 * 2 * gpc;
    QwPlan best = {0, 0, 0, 0};
    double cost = 0;
    for (int s = 2; s <= 8 && s <= wk; s *= 2) {
        const int js = (wk + s - 1) / s, xcols = std::min(ncol, js * ((ncol + wk - 1) / wk));
        const size_t most = 227 * 1024, fixed = kQwFixed + xcols * qw_x_bytes(ci, gpc, t, nd) + (size_t)js * t * 512;
        if (xcols >= kQwThreads || fixed + 3 * stage > most) continue;
        // cycles: a CTA's start, its digits and its columns, some 1100 per 256 inputs (16 rows: 1500); clusters at once: as the driver says (of
        // eight CTAs the GPU holds fewer than 148 / 8, since a cluster stays in one group of SMs: 2048 x 5120 as 16 clusters of eight took two waves)
        const int slots = at_once[s == 8 ? 2 : s == 4], waves = (tiles + slots - 1) / slots;
        const double col = (t == 8 ? 1100.0 : 1500.0) * ci / 256, dig = (double)xcols * ci / 256 * 18 * t;
        const double c = waves * (8000 + dig + xcols * col);
        if (best.cluster == 0 || c < cost) {
            cost = c;
            best.cluster = s; best.stages = (int)std::min<size_t>(kQwMaxStages, (most - fixed) / stage); best.xcols = xcols;
            best.smem = fixed + (size_t)best.stages * stage;
        }
    }
    return best;
}
}  // namespace

int qmv_rows_cluster(const int (&at_once)[3], int32_t fmt, int rows, int N, int K, int wk) { return qw_plan(at_once, fmt, rows <= 8 ? 8 : 16, N, K, wk).cluster; }

int32_t launch_qmv_rows(iq_ctx* ctx, cudaStream_t st, const GqmvCall& c, int wk) {
    if (c.rows < 1 || c.rows > 16 || ctx->encode_tiled == nullptr || c.mode != kModePlain) return 1;
    if (c.fmt != kFmtAffine4 && c.fmt != kFmtAffine4G32 && c.fmt != kFmtAffine8) return 1;
    const int t = c.rows <= 8 ? 8 : 16, row_bytes = c.fmt == kFmtAffine8 ? c.K : c.K / 2;
    const QwPlan plan = qw_plan(ctx->rows_clusters, c.fmt, t, c.N, c.K, wk);
    const uintptr_t align = reinterpret_cast<uintptr_t>(c.s[0]) | reinterpret_cast<uintptr_t>(c.b[0]);
    if (plan.cluster == 0 || (reinterpret_cast<uintptr_t>(c.w[0]) & 15) || (align & 1)) return 1;
    CUtensorMap map = {};
    const int32_t r = cached_rows_map(ctx, c.w[0], c.n_full > c.N ? c.n_full : c.N, row_bytes, 128, &map);
    if (r != kOk) return r;
    const int spb = c.fmt == kFmtAffine8 ? 4 : c.fmt == kFmtAffine4G32 ? 16 : 8;  // scale bytes of a row and column
    const int srow = c.K / (c.fmt == kFmtAffine4G32 ? 32 : 64) * 2;
    QwParams p;
    memset(&p, 0, sizeof(p));
    p.s = c.s[0]; p.b = c.b[0];
    p.vec = srow % spb == 0 && (align & (uintptr_t)(spb - 1)) == 0;
    p.N = c.N; p.K = c.K; p.M = c.rows;
    p.x = c.x; p.x_dtype = c.x_dtype; p.ldx = c.ldx;
    p.y = c.y; p.y_dtype = c.y_dtype; p.ldy = c.ldy; p.accumulate = c.accumulate;
    p.wk = wk;
    p.cluster = plan.cluster; p.xcols = plan.xcols; p.stages = plan.stages;
    p.status = ctx->d_status;
    const int tiles = (c.N + 127) / 128;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(tiles * plan.cluster, 1, 1);
    cfg.blockDim = dim3(kQwThreads, 1, 1);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = plan.cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return check_cuda(ctx, cudaLaunchKernelEx(&cfg, qw_pick(c.fmt, t), map, p), "qmv_rows launch");
}

int32_t rows_init(iq_ctx* ctx) {
    for (int v = 0; v < 6; v++) {
        const int32_t fmt = v < 2 ? kFmtAffine8 : v < 4 ? kFmtAffine4G32 : kFmtAffine4;
        cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(qw_pick(fmt, v & 1 ? 16 : 8)), cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return check_cuda(ctx, e, "cudaFuncSetAttribute(qmv_rows)");
    }
    for (int i = 1; i < 4; i++) {
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3(ctx->sms / (1 << i) << i, 1, 1);
        cfg.blockDim = dim3(kQwThreads, 1, 1);
        cfg.dynamicSmemBytes = 227 * 1024;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 1 << i; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        cudaError_t e = cudaOccupancyMaxActiveClusters(&n, qw_pick(kFmtAffine4, 16), &cfg);
        if (e != cudaSuccess) {  // (a guess does, the plans only have to be good)
            cudaGetLastError();
            n = ctx->sms * 7 / 8 >> i;
        }
        ctx->rows_clusters[i - 1] = std::max(n, 1);
    }
    return kOk;
}

}  // namespace iq
