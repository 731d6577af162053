// Host side of the tcgen05 GEMM: tensor maps, kernel selection, the iq_qmm entry point.
#include <string.h>

#include <algorithm>

#include "internal.h"
#include "qmm_ta.cuh"
#include "qmm_tc.cuh"

namespace iq {

namespace {

typedef void (*QmmKernel)(const CUtensorMap, const CUtensorMap, const QmmParams);

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

struct KernelEntry {
    int32_t fmt;
    int bn;
    QmmKernel fn;
    int smem;
};

template <int FMT, int BN>
KernelEntry entry() {
    return KernelEntry{FMT, BN, qmm_tc_kernel<FMT, BN>, QmmSmem<FMT, BN>::TOTAL};
}

const KernelEntry* table(int* n) {
    static const KernelEntry t[] = {
        // bf16 x bf16 (the router's approximate logits); the small token tiles spread few experts over many CTAs
        entry<kFmtBf16Plain, 128>(), entry<kFmtBf16Plain, 64>(), entry<kFmtBf16Plain, 32>(),
        entry<kFmtInt8Plain, 256>(), entry<kFmtInt8Plain, 128>(),  // rotated W8A8
    };
    *n = (int)(sizeof(t) / sizeof(t[0]));
    return t;
}

const KernelEntry* find(int32_t fmt, int bn) {
    int n;
    const KernelEntry* t = table(&n);
    for (int i = 0; i < n; i++)
        if (t[i].fmt == fmt && t[i].bn == bn) return &t[i];
    return nullptr;
}

int ta_step_bytes(int32_t fmt) { return fmt == kFmtAffine8 ? 64 : (fmt == kFmtTernary ? 16 : 32); }  // code bytes of a row per K step

typedef void (*TaKernel)(const TaMaps, const TaParams);

// gate/up: the formats of experts and of dense FFNs
template <int GROUPS, bool PAIR>
TaKernel ta_pick(int32_t fmt, int epi) {
    switch (fmt) {
        case kFmtAffine4: return epi ? qmm_ta_kernel<kFmtAffine4, 1, GROUPS, PAIR> : qmm_ta_kernel<kFmtAffine4, 0, GROUPS, PAIR>;
        case kFmtMxfp4: return epi ? qmm_ta_kernel<kFmtMxfp4, 1, GROUPS, PAIR> : qmm_ta_kernel<kFmtMxfp4, 0, GROUPS, PAIR>;
        case kFmtAffine8: return epi ? qmm_ta_kernel<kFmtAffine8, 1, GROUPS, PAIR> : qmm_ta_kernel<kFmtAffine8, 0, GROUPS, PAIR>;
        case kFmtAffine4G32: return epi ? qmm_ta_kernel<kFmtAffine4G32, 1, GROUPS, PAIR> : qmm_ta_kernel<kFmtAffine4G32, 0, GROUPS, PAIR>;
        case kFmtTernary: return epi ? nullptr : qmm_ta_kernel<kFmtTernary, 0, GROUPS, PAIR>;
        default: return nullptr;
    }
}

// Tiling of a dense GEMM: token rows per tile (a multiple of 16, at most 192), one CTA or a pair per tile, K split of the tiles beyond
// the whole rounds.
struct TaPlan {
    int rows, n_tiles, ustep, grid;
    TaSplit split;
    bool low;   // two CTAs per SM
    bool pair;  // clusters of two CTAs on tiles of twice the features
};
int ta_xk(bool low, int rows) { return low ? (rows <= 32 ? 4 : 2) : (rows <= 128 ? 4 : 2); }  // K steps per copy of X
int ta_ustep(int32_t fmt, int xk) { return std::max(128 / ta_step_bytes(fmt), xk); }  // whole stages of codes and of X

// The height with the least time: whole rounds over the SMs, or with the split the share of the split tiles and what the split costs.
TaPlan ta_plan(int32_t fmt, int epi, int M, int N, int K, int sms, bool may_split) {
    TaPlan best = {};
    double best_cost = -1;
    const int features = epi ? 64 : 128, ksteps = K / 64;
    for (int tiles = (M + kTaMaxRows - 1) / kTaMaxRows; tiles <= (M + 15) / 16; tiles++) {
        const int rows = round_up((M + tiles - 1) / tiles, 16);
        for (int pair = 0; pair < (sms % 2 == 0 ? 2 : 1); pair++) {
            TaPlan p;
            p.rows = rows;
            p.pair = pair != 0;
            p.n_tiles = (N + (features << pair) - 1) / (features << pair);
            const int total = (M + rows - 1) / rows * p.n_tiles;
            // Two CTAs per SM for low tiles; with a tile per SM or less the one with four dequantiser groups (MXFP4 24576 x 2048 at 64
            // rows 21.0 -> 18.5 us)
            p.low = !pair && rows <= kTaLowRows && total > sms;
            const int ctas = pair ? sms / 2 : p.low ? 2 * sms : sms;
            p.ustep = ta_ustep(fmt, ta_xk(p.low, rows));
            // (two CTAs per SM: never divided. Of 14,000 shapes asked none was, and the low kernel is faster without the code)
            p.split = may_split && !p.low ? ta_split(total, ctas, ksteps, p.ustep, rows, p.pair) : TaSplit{0, 0, 0};
            const double step = ta_step_cycles(rows, p.low, p.pair);
            double cost = (double)((total - p.split.tiles + ctas - 1) / ctas) * ksteps * step + (pair ? 1500 : 0);  // (a pair's start)
            if (p.split.tiles)
                cost += (p.split.tiles * p.split.units + p.split.ctas - 1) / p.split.ctas * p.ustep * step + (double)ta_split_cycles(p.split, rows, p.pair);
            p.grid = (total < ctas && p.split.tiles == 0 ? total : ctas) << pair;
            if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = p; }
        }
        if (rows <= 64) break;
    }
    return best;
}

// What the split of any call of up to M rows takes at most. The split of one call is no measure of a shorter one's (4096 x 14336:
// 39 MiB of FFN scratch at 512 rows, 28 at 640), and a buffer sized for the most rows has to serve them all. Per height, more tiles mean more
// slots until the split no longer pays, so the largest number of tiles for which it does is searched by halving.
size_t ta_split_bound(int32_t fmt, int epi, int M, int N, int K, int sms) {
    const int features = epi ? 64 : 128, ksteps = K / 64;
    size_t most = 0;
    for (int rows = 16; rows <= std::min(kTaMaxRows, round_up(M, 16)); rows += 16)
        for (int pair = 0; pair < (sms % 2 == 0 ? 2 : 1); pair++) {
            const int ctas = pair ? sms / 2 : sms, ustep = ta_ustep(fmt, ta_xk(false, rows));
            const int64_t total = (int64_t)((M + rows - 1) / rows) * ((N + (features << pair) - 1) / (features << pair));
            int lo = 0, hi = (int)std::min<int64_t>(total, ctas - 1);  // tiles of the last round: the split pays for lo of them
            while (lo < hi) {
                const int mid = (lo + hi + 1) / 2;
                if (ta_split(mid, ctas, ksteps, ustep, rows, pair).tiles != 0) lo = mid;
                else hi = mid - 1;
            }
            if (lo != 0) most = std::max(most, ta_split_bytes(ta_split(lo, ctas, ksteps, ustep, rows, pair), rows, pair));
        }
    return round_up_sz(most, 256);
}

}  // namespace

int32_t qmm_init(iq_ctx* ctx) {
    for (int fmt = 0; fmt <= kFmtTernary; fmt++)
        for (int epi = 0; epi < 2; epi++) {
            const TaKernel k = ta_pick<kTaGroups, false>(fmt, epi), pair = ta_pick<kTaGroups, true>(fmt, epi), low = ta_pick<kTaGroupsLow, false>(fmt, epi);
            if (k == nullptr) continue;
            cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(k), cudaFuncAttributeMaxDynamicSharedMemorySize, kTaSmemMax);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(reinterpret_cast<const void*>(pair), cudaFuncAttributeMaxDynamicSharedMemorySize, kTaSmemMax);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(reinterpret_cast<const void*>(low), cudaFuncAttributeMaxDynamicSharedMemorySize, kTaSmemLow);
            if (e != cudaSuccess) return check_cuda(ctx, e, "cudaFuncSetAttribute(qmm_ta)");
        }
    int n;
    const KernelEntry* t = table(&n);
    for (int i = 0; i < n; i++) {
        cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(t[i].fn),
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, t[i].smem);
        if (e != cudaSuccess) return check_cuda(ctx, e, "cudaFuncSetAttribute(qmm)");
    }
    return kOk;
}

// 2-D tensor map over a row-major matrix: `inner` elements per row, `rows` rows, `row_bytes` between rows.
// elem: 0 = bytes, 1 = fp16, 2 = bf16 elements
int32_t make_map_2d(iq_ctx* ctx, CUtensorMap* map, const void* base, int elem, uint64_t inner, uint64_t rows,
                    uint64_t row_bytes, uint32_t box_inner, uint32_t box_rows, bool swizzle128) {
    if (ctx->encode_tiled == nullptr) return fail(ctx, kErrCuda, "cuTensorMapEncodeTiled is not available");
    if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || row_bytes % 16 != 0)
        return fail(ctx, kErrInvalidArg, "qmm: TMA needs a 16-byte aligned base and row pitch");
    const cuuint64_t dims[2] = {inner, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_inner, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = reinterpret_cast<EncodeTiledFn>(ctx->encode_tiled)(
        map, elem == 1 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : (elem == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8),
        2, const_cast<void*>(base), dims,
        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
        swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(ctx, kErrCuda, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return kOk;
}

// X as the TMA of qmm_ta.cuh sees it: [K / 64][rows][64 fp16], box = xk K steps of box_rows rows, 128-byte swizzle.
static int32_t make_map_ksteps(iq_ctx* ctx, CUtensorMap* map, const void* base, uint64_t rows, uint64_t ksteps, uint64_t row_bytes,
                               uint32_t box_rows, uint32_t xk) {
    if (ctx->encode_tiled == nullptr) return fail(ctx, kErrCuda, "cuTensorMapEncodeTiled is not available");
    if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || row_bytes % 16 != 0)
        return fail(ctx, kErrInvalidArg, "qmm: TMA needs a 16-byte aligned base and row pitch");
    const cuuint64_t dims[3] = {64, rows, ksteps};
    const cuuint64_t strides[2] = {row_bytes, 128};
    const cuuint32_t box[3] = {64, box_rows, xk};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = reinterpret_cast<EncodeTiledFn>(ctx->encode_tiled)(
        map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(ctx, kErrCuda, "cuTensorMapEncodeTiled (K steps) failed (%d)", (int)r);
    return kOk;
}

int32_t make_map_rowblock(iq_ctx* ctx, CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes,
                          uint32_t box_rows) {
    if (ctx->encode_tiled == nullptr) return fail(ctx, kErrCuda, "cuTensorMapEncodeTiled is not available");
    if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || row_bytes % 128 != 0 || row_bytes / 128 > 256 || rows < 1 || box_rows < 8 ||
        box_rows > 256 || box_rows % 8 != 0)
        return fail(ctx, kErrInvalidArg, "qmv: TMA needs a 16-byte aligned base and rows of 128..32768 bytes in 128-byte steps");
    const cuuint64_t dims[3] = {128, rows, row_bytes / 128};
    const cuuint64_t strides[2] = {row_bytes, 128};
    const cuuint32_t box[3] = {128, box_rows, (cuuint32_t)(row_bytes / 128)};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = reinterpret_cast<EncodeTiledFn>(ctx->encode_tiled)(
        map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(ctx, kErrCuda, "cuTensorMapEncodeTiled (row block) failed (%d)", (int)r);
    return kOk;
}

int32_t cached_rowblock_map(iq_ctx* ctx, const void* base, int64_t rows, int32_t row_bytes, int32_t box_rows, CUtensorMap* out) {
    std::lock_guard<std::mutex> hold(ctx->qmv_maps_lock);
    if (ctx->qmv_maps == nullptr) ctx->qmv_maps = new iq_ctx::QmvMap[iq_ctx::kQmvMaps];
    const uintptr_t key = reinterpret_cast<uintptr_t>(base);
    iq_ctx::QmvMap& e = ctx->qmv_maps[((key >> 8) ^ (key >> 20) ^ (uintptr_t)rows ^ (uintptr_t)box_rows) % iq_ctx::kQmvMaps];
    if (e.base != base || e.rows != rows || e.row_bytes != row_bytes || e.box_rows != box_rows) {
        e.base = nullptr;
        const int32_t r = make_map_rowblock(ctx, &e.map, base, (uint64_t)rows, (uint64_t)row_bytes, (uint32_t)box_rows);
        if (r != kOk) return r;
        e.base = base; e.rows = (int32_t)rows; e.row_bytes = row_bytes; e.box_rows = box_rows;
    }
    *out = e.map;
    return kOk;
}

// Blocks of box_rows rows x 128 bytes with the 128-byte swizzle, of a matrix with any row pitch that is a multiple of 16 bytes.
int32_t cached_rows_map(iq_ctx* ctx, const void* base, int64_t rows, int32_t row_bytes, int32_t box_rows, CUtensorMap* out) {
    std::lock_guard<std::mutex> hold(ctx->qmv_maps_lock);
    if (ctx->qmv_maps == nullptr) ctx->qmv_maps = new iq_ctx::QmvMap[iq_ctx::kQmvMaps];
    const uintptr_t key = reinterpret_cast<uintptr_t>(base);
    iq_ctx::QmvMap& e = ctx->qmv_maps[((key >> 8) ^ (key >> 20) ^ (uintptr_t)rows ^ (uintptr_t)(box_rows - 16)) % iq_ctx::kQmvMaps];
    if (e.base != base || e.rows != rows || e.row_bytes != row_bytes || e.box_rows != -box_rows) {  // (negative: this kind of map)
        e.base = nullptr;
        const int32_t r = make_map_2d(ctx, &e.map, base, 0, (uint64_t)row_bytes, (uint64_t)rows, (uint64_t)row_bytes, 128, (uint32_t)box_rows, true);
        if (r != kOk) return r;
        e.base = base; e.rows = (int32_t)rows; e.row_bytes = row_bytes; e.box_rows = -box_rows;
    }
    *out = e.map;
    return kOk;
}

// The quantized formats: weights through tensor memory (csrc/qmm_ta.cuh). c.bn: the largest tile of the list (grouped).
static int32_t launch_qmm_ta(iq_ctx* ctx, cudaStream_t st, const QmmCall& c) {
    if (ta_pick<kTaGroups, false>(c.fmt, c.epi) == nullptr) return fail(ctx, kErrNoKernel, "qmm: no kernel for format %d, epilogue %d", c.fmt, c.epi);
    TaParams p;
    memset(&p, 0, sizeof(p));
    TaPlan plan = {};
    if (c.tiles == nullptr) {
        plan = ta_plan(c.fmt, c.epi, c.M, c.N, c.K, ctx->sms, c.split.part != nullptr);
    } else {
        plan.rows = c.bn;
        plan.low = plan.rows <= kTaLowRows;
        plan.pair = plan.rows == kTaMaxRows && ctx->sms % 2 == 0;  // (tiles of 128: 1024 tokens of 128 experts 198 us alone, 200 in pairs)
        plan.grid = plan.low ? 2 * ctx->sms : ctx->sms;
        plan.ustep = ta_ustep(c.fmt, ta_xk(plan.low, plan.rows));
    }
    const int rows = plan.rows;
    const bool low = plan.low;
    const int ctas = plan.pair ? 2 : 1;
    const TaKernel k = low ? ta_pick<kTaGroupsLow, false>(c.fmt, c.epi) : plan.pair ? ta_pick<kTaGroups, true>(c.fmt, c.epi) : ta_pick<kTaGroups, false>(c.fmt, c.epi);
    p.pair = plan.pair;
    p.ustep = plan.ustep;
    p.split = plan.split;
    p.part = c.split.part;
    p.tile_rows = rows;
    // Boxes of X: dense tiles have one height; tiles of a list have up to `rows`, a box of the nearest quarter of that. Two K
    // steps per copy, four where that is still small.
    p.xbox = c.tiles == nullptr || rows <= 16 ? rows : round_up(rows / 4, 16);
    p.nbox = rows / p.xbox;
    p.xk = ta_xk(low, rows);
    p.x_stage = rows / ctas * 128 * p.xk;
    p.dcols = low ? kTaLowRows : (rows <= 128 ? 128 : kTaMaxRows);
    // stages: at least three of codes, then up to eight of X, then as many of codes as fit
    const int room = (low ? kTaSmemLow : kTaSmemMax) - kTaSmemFixed;
    const int c_stage = ta_code_stage(c.fmt);
    p.nx = (room - 3 * c_stage) / p.x_stage;
    if (p.nx > 8) p.nx = 8;
    p.nc = (room - p.nx * p.x_stage) / c_stage;
    if (p.nc > kTaMaxStages) p.nc = kTaMaxStages;
    const int smem = kTaSmemFixed + p.nx * p.x_stage + p.nc * c_stage;

    const uint64_t row_bytes = (uint64_t)c.K / 64 * ta_step_bytes(c.fmt);
    TaMaps maps;
    int32_t r = kOk;
    for (int i = 0; i < p.nbox && r == kOk; i++)
        r = make_map_ksteps(ctx, &maps.x[i], c.x16, (uint64_t)c.x_rows, (uint64_t)c.K / 64, (uint64_t)c.ldx * 2, p.xbox * (i + 1) / ctas, p.xk);
    const uint32_t wbox = c.epi ? 64 : 128;
    for (int i = 0; i <= c.epi && r == kOk; i++)
        r = make_map_2d(ctx, &maps.w[i], c.w[i], 0, row_bytes, (uint64_t)c.experts * c.N, row_bytes, 128, wbox, true);
    if (r != kOk) return r;
    uintptr_t align = 0;
    for (int i = 0; i < 2; i++) {
        p.s[i] = c.s[i] ? c.s[i] : c.s[0];
        p.b[i] = c.b[i] ? c.b[i] : c.b[0];
        p.ebias[i] = c.ebias[i];
        align |= reinterpret_cast<uintptr_t>(p.s[i]) | reinterpret_cast<uintptr_t>(p.b[i]);
    }
    // scale bytes of a weight row, and of it per stage of codes: asynchronous copies of that size need the row pitch and the
    // base to be multiples of it
    const int srow = c.fmt == kFmtMxfp4 ? c.K / 32 : (c.fmt == kFmtTernary ? c.K / 64 : (c.fmt == kFmtAffine4G32 ? c.K / 16 : c.K / 32));
    const int spb = c.fmt == kFmtAffine8 ? 4 : (c.fmt == kFmtAffine4G32 ? 16 : 8);
    p.vec = srow % spb == 0 && (align & (uintptr_t)(spb - 1)) == 0 ? 1 : (align & 1) ? -1 : 0;
    if (p.vec < 0 && c.fmt != kFmtMxfp4) return fail(ctx, kErrInvalidArg, "qmm: scales and biases must be 2-byte aligned");
    p.expert_lo = c.expert_lo;
    p.early = c.early ? 1 : 0;
    p.N = c.N; p.K = c.K; p.M = c.M;
    p.tiles = c.tiles; p.ntiles = c.ntiles;
    p.y = c.y; p.y_dtype = c.y_dtype; p.ldy = c.ldy; p.accumulate = c.accumulate;
    p.limit = c.limit;
    p.act = c.act;
    p.status = ctx->d_status;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(plan.grid, 1, 1);
    cfg.blockDim = dim3(ta_threads(low ? kTaGroupsLow : kTaGroups), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = plan.pair ? 2 : 1;
    r = check_cuda(ctx, cudaLaunchKernelEx(&cfg, k, maps, p), "qmm launch");
    if (r != kOk || p.split.tiles == 0) return r;
    const int warps = plan.split.tiles * ((rows + 3) / 4) * 4 * ctas, blocks = (warps + 7) / 8;
    return check_cuda(ctx, launch_dependent(c.epi ? ta_sum_kernel<1> : ta_sum_kernel<0>, dim3(std::min(blocks, 8 * ctx->sms)), 256, 0, st, p),
                      "qmm sums launch");
}

int32_t launch_qmm(iq_ctx* ctx, cudaStream_t st, const QmmCall& c) {
    if (c.fmt != kFmtBf16Plain && c.fmt != kFmtInt8Plain) return launch_qmm_ta(ctx, st, c);
    // bf16 activations and weights, or int8 rows on both sides, copied as they are
    const KernelEntry* ke = find(c.fmt, c.bn);
    if (ke == nullptr || c.epi != 0 || c.tiles != nullptr)
        return fail(ctx, kErrNoKernel, "qmm: no kernel for format %d, tile %d, epilogue %d", c.fmt, c.bn, c.epi);
    const bool i8 = c.fmt == kFmtInt8Plain;
    const int elem = i8 ? 0 : 2, es = i8 ? 1 : 2, bke = i8 ? 128 : 64;
    CUtensorMap mx, mw;
    int32_t r = make_map_2d(ctx, &mx, c.x16, elem, (uint64_t)c.K, (uint64_t)c.x_rows, (uint64_t)c.ldx * es, bke, c.bn, true);
    if (r == kOk) r = make_map_2d(ctx, &mw, c.w[0], elem, (uint64_t)c.K, (uint64_t)(c.w_rows ? c.w_rows : c.N), (uint64_t)c.K * es, bke, kWRows, true);
    if (r != kOk) return r;
    QmmParams p = {};
    p.s = c.s[0]; p.b = c.b[0];
    p.N = c.N; p.K = c.K; p.M = c.M;
    p.y = c.y; p.y_dtype = c.y_dtype; p.ldy = c.ldy; p.accumulate = c.accumulate;
    p.limit = c.limit;
    p.status = ctx->d_status;
    const int work = ((c.M + c.bn - 1) / c.bn) * ((c.N + kWRows - 1) / kWRows);
    ke->fn<<<work < ctx->sms ? work : ctx->sms, kQmmThreads, ke->smem, st>>>(mx, mw, p);
    return check_cuda(ctx, cudaGetLastError(), "qmm launch");
}

}  // namespace iq

using namespace iq;

namespace iq {
QmmSplit qmm_split(iq_ctx* ctx, int32_t fmt, int epi, int M, int N, int K, void* scratch, size_t bytes) {
    QmmSplit r;
    if (fmt < 0 || fmt == kFmtAffine6 || fmt > kFmtTernary) return r;
    const TaPlan p = ta_plan(fmt, epi, M, N, K, ctx->sms, true);
    r.bytes = round_up_sz(ta_split_bytes(p.split, p.rows, p.pair), 256);
    if (r.bytes != 0 && bytes >= r.bytes && (reinterpret_cast<uintptr_t>(scratch) & 15) == 0) r.part = static_cast<float*>(scratch);
    return r;
}
size_t qmm_split_bound(iq_ctx* ctx, int32_t fmt, int epi, int M, int N, int K) {
    return fmt < 0 || fmt == kFmtAffine6 || fmt > kFmtTernary ? 0 : ta_split_bound(fmt, epi, M, N, K, ctx->sms);
}
size_t qmm_split_max_bytes(iq_ctx* ctx) { return (size_t)2 * ctx->sms * ta_slot(kTaMaxRows) * 4; }
size_t qmm_convert_bytes(int rows, int k, int32_t x_dtype) { return x_dtype == IQ_F16 ? 0 : round_up_sz((size_t)rows * k * 2, 256); }

}  // namespace iq

extern "C" int32_t iq_qmm_workspace_bytes(iq_ctx* ctx, const iq_qlinear* m, int32_t rows, int32_t x_dtype, size_t* bytes) {
    if (ctx == nullptr || m == nullptr || bytes == nullptr || rows < 1) return kErrInvalidArg;
    // The MMA takes fp16 weights with fp16 activations only (a bf16 B operand beside an fp16 A operand is an illegal
    // instruction on sm_100a: kind::f16 wants both operands of one type), so bf16 and fp32 activations are converted
    *bytes = qmm_convert_bytes(rows, m->k, x_dtype) + qmm_split_bound(ctx, format_of(m), 0, rows, m->n, m->k);
    return kOk;
}

extern "C" int32_t iq_qmm_plan(const iq_qlinear* m, int32_t gate_up, int32_t rows, int32_t sms, iq_qmm_tiling* out) {
    if (m == nullptr || out == nullptr || rows < 1 || sms < 1 || m->n < 1 || m->k < 64 || (gate_up && m->n % 2 != 0)) return kErrInvalidArg;
    const int32_t fmt = format_of(m);
    if (fmt < 0 || fmt == kFmtAffine6 || (gate_up && fmt == kFmtTernary)) return kErrUnsupported;
    const int n = gate_up ? m->n / 2 : m->n;
    const TaPlan p = ta_plan(fmt, gate_up != 0, rows, n, m->k, sms, true);
    out->tile_rows = p.rows; out->tiles = (rows + p.rows - 1) / p.rows * p.n_tiles;
    out->pair = p.pair; out->two_per_sm = p.low;
    out->split_tiles = p.split.tiles; out->split_ctas = p.split.ctas;
    out->split_bytes = round_up_sz(ta_split_bytes(p.split, p.rows, p.pair), 256);
    out->bytes_up_to_rows = ta_split_bound(fmt, gate_up != 0, rows, n, m->k, sms);
    return kOk;
}

namespace iq {
int32_t qmm_check(iq_ctx* ctx, const void* x, int32_t x_dtype, int64_t ldx, const iq_qlinear* m, const void* y, int32_t y_dtype, int64_t ldy,
                  int32_t rows) {
    if (x == nullptr || y == nullptr || m == nullptr || m->w == nullptr || m->scales == nullptr)
        return fail(ctx, kErrInvalidArg, "qmm: null pointer");
    const int32_t fmt = format_of(m);
    if (fmt < 0 || fmt == kFmtAffine6)
        return fail(ctx, kErrUnsupported,
                    "qmm: %d-bit group %d mode %d has no kernel (affine 4/8-bit g64, 4-bit g32, ternary 2-bit g128, mxfp4 g32)",
                    m->bits, m->group, m->mode);
    if (fmt != kFmtMxfp4 && fmt != kFmtTernary && m->biases == nullptr)
        return fail(ctx, kErrInvalidArg, "qmm: affine layer without biases");
    if (fmt == kFmtTernary && m->k % 128 != 0) return fail(ctx, kErrInvalidArg, "qmm: ternary k = %d must be a multiple of 128", m->k);
    // the reference's preconditions (Layers/Linear.swift:695)
    if (rows < 64 || rows % 64 != 0) return fail(ctx, kErrInvalidArg, "qmm: rows = %d must be a multiple of 64", rows);
    if (m->n % 64 != 0 || m->k % 64 != 0 || m->n <= 0 || m->k <= 0)
        return fail(ctx, kErrInvalidArg, "qmm: n = %d and k = %d must be multiples of 64", m->n, m->k);
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return fail(ctx, kErrInvalidArg, "qmm: dtype");
    if (ldx < m->k || ldx % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0 || ldy < m->n)
        return fail(ctx, kErrInvalidArg, "qmm: x must be 16-byte aligned with ldx >= k, ldx %% 8 == 0; ldy >= n");
    return kOk;
}

int32_t launch_convert_x(iq_ctx* ctx, cudaStream_t st, const void* x, int32_t x_dtype, int64_t ldx, void* out, int rows, int k) {
    const size_t units = (size_t)rows * k / 8;
    return check_cuda(ctx, launch_dependent(convert_x_f16_kernel, dim3((unsigned)((units + 255) / 256)), 256, 0, st, x, x_dtype, ldx,
                                            static_cast<__half*>(out), rows, k), "convert_x launch");
}

int32_t qmm_f16(iq_ctx* ctx, cudaStream_t st, const void* x, int64_t ldx, const iq_qlinear* m, void* y, int32_t y_dtype, int64_t ldy, int32_t rows,
                uint32_t flags, const QmmSplit& split) {
    QmmCall c;
    c.fmt = format_of(m);
    c.epi = 0;
    c.x16 = x; c.ldx = ldx; c.x_rows = rows;
    c.w[0] = m->w; c.s[0] = m->scales; c.b[0] = m->biases;
    c.experts = 1;
    c.N = m->n; c.K = m->k; c.M = rows;
    c.y = y; c.y_dtype = y_dtype; c.ldy = ldy;
    c.accumulate = (flags & IQ_FLAG_ACCUMULATE) ? 1 : 0;
    c.split = split;
    return launch_qmm(ctx, st, c);
}
}  // namespace iq

extern "C" int32_t iq_qmm(iq_ctx* ctx, void* stream, const void* x, int32_t x_dtype, int64_t ldx, const iq_qlinear* m,
                          void* y, int32_t y_dtype, int64_t ldy, int32_t rows, uint32_t flags, void* workspace,
                          size_t workspace_bytes) {
    if (ctx == nullptr) return kErrInvalidArg;
    int32_t st = qmm_check(ctx, x, x_dtype, ldx, m, y, y_dtype, ldy, rows);
    if (st != kOk) return st;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(stream);
    const size_t need = qmm_convert_bytes(rows, m->k, x_dtype);
    QmmSplit split;  // (a workspace that holds the converted activations only is good as well: every tile is one item then)
    if (workspace != nullptr && workspace_bytes > need)
        split = qmm_split(ctx, format_of(m), 0, rows, m->n, m->k, static_cast<char*>(workspace) + need, workspace_bytes - need);
    if (x_dtype == IQ_F16) return qmm_f16(ctx, cs, x, ldx, m, y, y_dtype, ldy, rows, flags, split);
    if (workspace == nullptr || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255) != 0)
        return fail(ctx, kErrWorkspace, "qmm: workspace %zu < %zu (256-byte aligned)", workspace_bytes, need);
    st = launch_convert_x(ctx, cs, x, x_dtype, ldx, workspace, rows, m->k);
    return st != kOk ? st : qmm_f16(ctx, cs, workspace, m->k, m, y, y_dtype, ldy, rows, flags, split);
}

// ---------------------------------------------------------------------------------------------------------------------
// Prefill GEMM for callers that cannot allocate device memory.
//
// Some hosts of this library may not call cudaMalloc at all: a plugin loaded into an engine whose memory pool owns
// every device byte and forbids side allocations, a call site that runs after the pool has been sealed, or code under
// a "no allocation after start-up" rule (real-time serving paths, sandboxes that filter the allocator entry points).
// iq_qmm needs a scratch buffer when the activations are bf16 or fp32 (they are converted to fp16 first) and expects the
// caller to bring it. This variant brings its own: a fixed array that is part of the library image, so it exists on
// every GPU that loads the library, from load until the process exits, and costs that GPU kNoAllocBytes + kNoAllocSplit of memory.
constexpr size_t kNoAllocBytes = 8u << 20;   // 8 MiB: rows * k <= 4,194,304 activations (e.g. 1024 x 4096)
constexpr size_t kNoAllocSplit = 28u << 20;  // partial sums of the K split: the most that any call on 148 SMs takes
static_assert(kNoAllocSplit >= (size_t)2 * 148 * ta_slot(kTaMaxRows) * 4, "two slots of 192 tokens per SM");
static __device__ __align__(256) unsigned char g_qmm_noalloc_scratch[kNoAllocBytes + kNoAllocSplit];

namespace {
constexpr int kMaxDevices = 64;
std::atomic<void*> g_noalloc_ptr[kMaxDevices];  // device address of the array, per device, resolved on first use (zero-initialised)
}  // namespace

extern "C" int32_t iq_qmm_noalloc(iq_ctx* ctx, void* stream, const void* x, int32_t x_dtype, int64_t ldx,
                                  const iq_qlinear* m, void* y, int32_t y_dtype, int64_t ldy, int32_t rows,
                                  uint32_t flags) {
    if (ctx == nullptr) return kErrInvalidArg;
    if (m == nullptr) return fail(ctx, kErrInvalidArg, "qmm_noalloc: null pointer");
    if (rows < 1 || m->k < 1) return fail(ctx, kErrInvalidArg, "qmm_noalloc: rows = %d, k = %d", rows, m->k);
    const size_t need = (size_t)rows * (size_t)m->k * 2;
    if (need > kNoAllocBytes)
        return fail(ctx, kErrWorkspace,
                    "qmm_noalloc: rows * k = %zu activations exceed the built-in scratch (%zu); use iq_qmm with a "
                    "caller-provided workspace", (size_t)rows * (size_t)m->k, kNoAllocBytes / 2);
    const int dev = ctx->device;
    if (dev < 0 || dev >= kMaxDevices) return fail(ctx, kErrInvalidArg, "qmm_noalloc: device %d", dev);
    void* scratch = g_noalloc_ptr[dev].load(std::memory_order_acquire);
    if (scratch == nullptr) {
        // The array's name is only a host-side handle here; the kernels need its address on this device. Resolved once
        // per device with that device current (it is: the context selected it, and the caller runs on it).
        int cur = -1;
        cudaError_t e = cudaGetDevice(&cur);
        if (e != cudaSuccess) return check_cuda(ctx, e, "cudaGetDevice");
        if (cur != dev) return fail(ctx, kErrInvalidArg, "qmm_noalloc: device %d is current, the context is on %d", cur, dev);
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_qmm_noalloc_scratch);
        if (e != cudaSuccess) return check_cuda(ctx, e, "cudaGetSymbolAddress(scratch)");
        g_noalloc_ptr[dev].store(p, std::memory_order_release);  // two first callers store the same address
        scratch = p;
    }
    // Every byte that is read from the scratch is written by this call first (activations by the conversion pass, partial sums by the
    // GEMM whose sums' kernel reads them), so nothing has to be cleared; what the previous call left behind is simply overwritten.
    return iq_qmm(ctx, stream, x, x_dtype, ldx, m, y, y_dtype, ldy, rows, flags, scratch, kNoAllocBytes + kNoAllocSplit);
}
