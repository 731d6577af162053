// Launchers of the MoE decode tiles on tcgen05 integers (csrc/qmv_tile.cuh).
#include <string.h>

#include <algorithm>

#include "internal.h"
#include "qmv_tile.cuh"

namespace iq {

int32_t launch_fixed_rows(iq_ctx* ctx, cudaStream_t st, const void* x, int32_t x_dtype, int64_t ldx, int rows, int D, const FixedRows& fx, bool wide) {
    return check_cuda(ctx, launch_dependent(wide ? fixed_rows_kernel<true> : fixed_rows_kernel<false>, dim3(std::min(rows, 8 * ctx->sms)), 256, 0, st, x, x_dtype, ldx,
                                            rows, D, fx), "fixed_rows launch");
}

typedef void (*QtKernel)(const QtMaps, const QtParams);
static QtKernel qt_pick(int epi, bool wide) {
    if (epi) return wide ? qmv_tile_kernel<1, 3> : qmv_tile_kernel<1, 2>;
    return wide ? qmv_tile_kernel<0, 3> : qmv_tile_kernel<0, 2>;
}

int32_t launch_qmv_tile(iq_ctx* ctx, cudaStream_t st, const QmmCall& c, const FixedRows& x, bool wide, const uint32_t* row_map, int32_t topk, int32_t slice, int32_t max_tiles) {
    if (c.fmt != kFmtAffine4 || c.tiles == nullptr || c.K % (wide ? 64 : 256) != 0 || c.bn != kQtRows || c.accumulate || c.y_dtype != kF16 || slice < 1)
        return fail(ctx, kErrNoKernel, "moe: no decode tiles for format %d, %d inputs", c.fmt, c.K);
    QtParams p;
    memset(&p, 0, sizeof(p));
    QtMaps maps = {};
    uintptr_t align = 0;
    for (int i = 0; i <= c.epi; i++) {
        align |= reinterpret_cast<uintptr_t>(c.s[i]) | reinterpret_cast<uintptr_t>(c.b[i]);
        p.s[i] = c.s[i]; p.b[i] = c.b[i]; p.ebias[i] = c.ebias[i];
        const int32_t r = cached_rows_map(ctx, c.w[i], (int64_t)c.experts * c.N, c.K / 2, c.epi ? 64 : 128, &maps.w[i]);
        if (r != kOk) return r;
    }
    if (align & 1) return fail(ctx, kErrInvalidArg, "moe: scales and biases must be 2-byte aligned");
    p.vec = c.K % 256 == 0 && (align & 7) == 0;
    p.expert_lo = c.expert_lo;
    p.N = c.N; p.K = c.K;
    p.x = x; p.row_map = row_map; p.topk = topk; p.slice = slice;
    p.tiles = c.tiles; p.ntiles = c.ntiles;
    p.y = static_cast<__half*>(c.y); p.ldy = c.ldy;
    p.limit = c.limit; p.act = c.act;
    p.early = c.early ? 1 : 0;
    p.status = ctx->d_status;
    const int nrows = c.epi ? 64 : 128;
    const int64_t items = (int64_t)max_tiles * ((c.N + nrows - 1) / nrows);
    return check_cuda(ctx, launch_dependent(qt_pick(c.epi, wide),
                                            dim3((unsigned)std::min<int64_t>(items, 2 * ctx->sms)), qt_threads(wide ? 3 : 2), qt_smem(wide ? 3 : 2), st, maps, p),
                      "qmv_tile launch");
}

int32_t tile_init(iq_ctx* ctx) {
    for (int v = 0; v < 4; v++) {
        cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(qt_pick(v & 1, v >= 2)), cudaFuncAttributeMaxDynamicSharedMemorySize, qt_smem(v >= 2 ? 3 : 2));
        if (e != cudaSuccess) return check_cuda(ctx, e, "cudaFuncSetAttribute(qmv_tile)");
    }
    return kOk;
}

}  // namespace iq
