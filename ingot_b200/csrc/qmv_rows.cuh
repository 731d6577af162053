// Decode linears of several rows and wide inputs on the 5th-generation tensor cores with integers (affine weights, 4 and 8 bits).
//
// The arithmetic, the digits and the order of the sums are those of the ring kernel (qmv_ring.cuh), which takes these shapes at fewer rows: a row
// has the same bits alone and among sixteen. That kernel holds the digits of all inputs in every CTA beside sixteen rings of weights: of wide inputs
// few rows fit (rows_kernel_pays in qmv.cu: two of 11000 inputs), and sixteen rows are up to eight launches that each read the weights. Here a cluster
// shares a tile of 128 weight rows, each CTA holding the digits of its K slices only, and one thread issues tcgen05.mma (kind::i8) for 128 weight
// rows against all (digit, row) columns, so that sixteen rows are one launch: 4096 x 14336 (4 bits) at 8 rows 53.7 -> 27.3 us, at
// 16 106 -> 62.3, 4096 x 11008 at 12 62.5 -> 26.6, 8 bits 66.5 -> 31.8 at 16. How many clusters run at once is asked of the driver: thirty-three of four CTAs,
// but fifteen of eight, since a cluster stays in one group of SMs (2048 x 7680 at 8 rows 20 us as sixteen clusters of eight, 14.3 of four). Inputs that the staged kernel takes
// (2048, 4096, 8 bits 6144) stay there: a step of 256 inputs takes this machine 1000 to 2000 cycles whatever its rows (waits on barriers, loads from tensor memory and sums
// of one step follow one another in a warp), and 14336 x 4096 at 8 rows took 29.0 us instead of 20.4.
//
// Unit of work: a cluster of two to eight CTAs takes a tile, each its share of the K slices (the digits of all of K fit one CTA only where a cluster is
// faster). K is walked slice by slice as the ring kernel cuts it (every wk-th
// column; a column is 128 bytes of a row's codes), so that every slice's sum is one accumulator's; the slices are added in their order
// at the end, through the cluster's shared memory. The activations' digits for the CTA's columns are made once, by the warps
// that later finish the sums, while the first weights arrive, and stay in shared memory.
//
// Warp roles (512 threads): 1 tensor memory and tcgen05.mma; 2 codes; 3 scales and biases; 4-11 digits, then sums to floats, half of the rows
// each; 12-15 codes to bytes (8-bit codes need none: the MMA reads them from shared memory as they came).
// Every wait is bounded: on a timeout the kernel writes a status word, all roles drain and tensor memory is released.
//
// Same operator as vnax_qmv* (Shaders/verify_nax.metal:105-230) of the reference.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"
#include "qmv_imma.cuh"
#include "qmv_ring.cuh"
#include "umma_i8.cuh"

namespace iq {

constexpr int kQwThreads = 512;
constexpr int kQwMaxStages = 8;
constexpr int kQwMaxCols = 512;  // columns of a CTA
constexpr int kQwFixed = 1024 + 512 + 2 * kQwMaxCols;

// What a format makes of it. GS: inputs per group, CI: inputs per column, GPC: groups per column
template <int FMT>
struct QwFmt {
    static constexpr bool W8 = FMT == kFmtAffine8, G32 = FMT == kFmtAffine4G32;
    static constexpr int GS = G32 ? 32 : 64, CI = W8 ? 128 : 256, GPC = CI / GS, SPB = 2 * GPC;
    static constexpr int ND = W8 ? 2 : 3;  // digits of an input (see qmv_ring.cuh)
    static constexpr int STAGE = kQtCodes + 2 * 128 * SPB;
};
// Columns of the MMA: digits x rows, in steps of 16
constexpr int qw_cols(int t, int nd) { return (t * nd + 15) / 16 * 16; }
inline size_t qw_x_bytes(int ci, int gpc, int t, int nd) { return (size_t)ci * t * nd + (size_t)gpc * t * 8; }  // of a column: digits, {scale, sum}

struct QwParams {
    const void* s;
    const void* b;
    int32_t N, K, M;
    const void* x;
    int32_t x_dtype;
    int64_t ldx;
    void* y;
    int32_t y_dtype;
    int64_t ldy;
    int32_t accumulate;
    int32_t wk;        // K slices: every wk-th column
    int32_t cluster;   // CTAs that share a tile's slices
    int32_t xcols;     // columns whose digits a CTA holds, at most
    int32_t stages;
    int32_t vec;       // scales by asynchronous copies
    int32_t* status;
};

__device__ __forceinline__ float ld_dsmem_f32(uint32_t addr, uint32_t cta) {
    uint32_t remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(cta));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}
// (both as one asm with the registers passing through the wait, see qt_ld_wait)
template <int H>
__device__ __forceinline__ void qw_wait_ld(int (&a)[H]) {
    static_assert(H == 4 || H == 8, "tokens of a warp");
    if constexpr (H == 4)
        asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]) : : "memory");
    else
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]) : : "memory");
}

__device__ __forceinline__ void qw_store(const QwParams& p, size_t o, float f) {
    if (p.y_dtype == kF32) {
        float* yp = reinterpret_cast<float*>(p.y) + o;
        *yp = p.accumulate ? *yp + f : f;
    } else if (p.y_dtype == kF16) {
        __half* yp = reinterpret_cast<__half*>(p.y) + o;
        *yp = __float2half_rn(p.accumulate ? __half2float(*yp) + f : f);
    } else {
        uint16_t* yp = reinterpret_cast<uint16_t*>(p.y) + o;
        *yp = (uint16_t)f32_to_bf16_bits(p.accumulate ? bf16_bits_to_f32(*yp) + f : f);
    }
}

// FMT: kFmtAffine4, kFmtAffine4G32, kFmtAffine8; T: rows (8 or 16)
template <int FMT, int T>
__global__ void __launch_bounds__(kQwThreads, 1) qmv_rows_kernel(const __grid_constant__ CUtensorMap map, const QwParams p) {
    using F = QwFmt<FMT>;
    constexpr int GS = F::GS, CI = F::CI, GPC = F::GPC, SPB = F::SPB, KK = GS / 32;
    constexpr bool W8 = F::W8;
    constexpr int ND = F::ND;
    constexpr int NB = qw_cols(T, ND);
    constexpr int UG = 2;                                     // groups per hand-over
    constexpr int UPC = GPC / UG;
    constexpr int AC = W8 ? 0 : UG * GS / 4;                  // columns of a slot of A
    constexpr int DC = UG * NB;
    constexpr int NA = W8 ? 0 : (256 - 2 * DC) / AC >= 4 ? 4 : 2;
    constexpr int D0 = NA * AC;
    static_assert(D0 + 2 * DC <= 256, "tensor memory");
    constexpr int NROWS = 128;
    constexpr int XT = ND * T * 128;                          // digits of 128 inputs
    constexpr int H = T / 2, PAIRS = T / 4;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int NST = p.stages;
    const uint32_t codes0 = smem_u32(smem), x0 = codes0 + NST * kQtCodes, scales0 = x0 + p.xcols * (CI / 128) * XT;
    const uint32_t xs0 = scales0 + NST * 2 * 128 * SPB;
    unsigned char* xd = smem + (size_t)NST * kQtCodes;
    float* xs = reinterpret_cast<float*>(smem + (size_t)(xs0 - codes0));
    float* part = xs + (size_t)p.xcols * GPC * T * 2;         // [slice][token][128 lanes]
    const int rank = (int)cluster_rank();
    const int j0 = p.wk * rank / p.cluster, j1 = p.wk * (rank + 1) / p.cluster, jmax = (p.wk + p.cluster - 1) / p.cluster;
    uint64_t* bars = reinterpret_cast<uint64_t*>(part + (size_t)jmax * T * 128);
    const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * kQwMaxStages, bar_aready = bar_empty + 8 * kQwMaxStages, bar_aempty = bar_aready + 32;
    const uint32_t bar_dfull = bar_aempty + 32, bar_dempty = bar_dfull + 16, bar_x = bar_dempty + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kQwMaxStages + 13);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* ncols = abort_flag + 1;
    volatile uint16_t* cols = reinterpret_cast<volatile uint16_t*>(bars + 64);  // column, bit 15: the last one of its slice

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = p.K / GS, ncol = (p.K + CI - 1) / CI;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NST; i++) {
            mbar_init(bar_full + 8 * i, 1 + 32);
            mbar_init(bar_empty + 8 * i, (W8 ? 0 : 4) + 1 + 8);  // codes to bytes, the MMAs (8-bit codes), sums to floats
        }
        for (int i = 0; i < 4; i++) {
            mbar_init(bar_aready + 8 * i, 4);
            mbar_init(bar_aempty + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(bar_dfull + 8 * i, 1);
            mbar_init(bar_dempty + 8 * i, 8);
        }
        mbar_init(bar_x, 256);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    {  // this CTA's columns, slice by slice
        int li = threadIdx.x, j = j0;
        for (; j < j1; j++) {
            const int cnt = (ncol - j + p.wk - 1) / p.wk;
            if (li < cnt) break;
            li -= cnt;
        }
        if (j < j1) cols[threadIdx.x] = (uint16_t)((j + li * p.wk) | (j + (li + 1) * p.wk >= ncol ? 0x8000 : 0));
        else if (li == 0) *ncols = threadIdx.x;  // (fewer than the threads)
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int nloc = *ncols;
    pdl_launch_dependents();

    const int n0 = (int)blockIdx.x / p.cluster * NROWS;  // of the cluster's tile

    if (warp == 2) {
        // ================= packed codes =================
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            for (int li = 0; li < nloc; li++) {
                if (!mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag)) break;
                mbar_arrive_expect_tx(bar_full + 8 * s, kQtCodes);
                tma_load_2d(codes0 + s * kQtCodes, &map, bar_full + 8 * s, (cols[li] & 0x7FFF) * 128, n0);
                if (++s == NST) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 3) {
        // ================= scales and biases: SPB bytes of each per row and column; row = lane of the sums =================
        const size_t pitch = (size_t)G * 2;
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        const char* src[4][2];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int n = min(n0 + i * 32 + lane, p.N - 1);
            src[i][0] = static_cast<const char*>(p.s) + (size_t)n * pitch;
            src[i][1] = static_cast<const char*>(p.b) + (size_t)n * pitch;
        }
        for (int li = 0; li < nloc; li++) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag));
            if (!ok) break;
            const uint32_t dst = scales0 + s * (2 * 128 * SPB) + lane * SPB;
            const int off = (cols[li] & 0x7FFF) * SPB, left = (int)pitch - off;
            if (p.vec) {
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int m = 0; m < 2; m++) cp_async_ca<SPB>(dst + (m * 128 + i * 32) * SPB, src[i][m] + off);
                cp_async_arrive_noinc(bar_full + 8 * s);
            } else {
                uint32_t v[4][2][GPC];
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int m = 0; m < 2; m++)
#pragma unroll
                        for (int e = 0; e < GPC; e++) v[i][m][e] = ldg_nc_u16(src[i][m] + off + min(2 * e, left - 2));
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int m = 0; m < 2; m++)
#pragma unroll
                        for (int e = 0; e < GPC / 2; e++)
                            sts32(dst + (m * 128 + i * 32) * SPB + 4 * e, v[i][m][2 * e] | (v[i][m][2 * e + 1] << 16));
                mbar_arrive(bar_full + 8 * s);
            }
            if (++s == NST) { s = 0; ph ^= 1; }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        if (elect_one()) {
            int s = 0, as = 0, ds = 0;
            uint32_t ph = 0, aph = 0, dph = 0;
            const uint32_t idesc = qt_idesc(NB), xdesc0 = (x0 & 0x3FFFFu) >> 4, cdesc0 = (codes0 & 0x3FFFFu) >> 4;
            bool ok = mbar_wait_hint(0, bar_x, 0, abort_flag);
            for (int li = 0; li < nloc && ok; li++) {
                if (W8 && !(ok = mbar_wait_hint(0, bar_full + 8 * s, ph, abort_flag))) break;
#pragma unroll
                for (int u = 0; u < UPC; u++) {
                    if (!W8 && !(ok = mbar_wait_hint(0, bar_aready + 8 * as, aph, abort_flag))) break;
                    if (!(ok = mbar_wait_hint(0, bar_dempty + 8 * ds, dph ^ 1, abort_flag))) break;
                    tc_fence_after();
                    const uint32_t ta = tmem + as * AC, td = tmem + D0 + ds * DC;
#pragma unroll
                    for (int g = 0; g < UG; g++) {
                        const int k0 = (u * UG + g) * GS;  // of the column
                        const uint32_t xdesc = xdesc0 + (li * (CI / 128) + k0 / 128) * (XT >> 4) + (k0 % 128) / 16;
#pragma unroll
                        for (int kk = 0; kk < KK; kk++) {
                            const uint64_t bd = kQtDescHi | (uint64_t)(xdesc + 2 * kk);
                            if (W8) umma_i8(td + g * NB, kQtDescHi | (uint64_t)(cdesc0 + s * (kQtCodes >> 4) + k0 / 16 + 2 * kk), bd, idesc, kk);
                            else umma_i8_ta(td + g * NB, ta + g * (GS / 4) + kk * 8, bd, idesc, kk);
                        }
                    }
                    if (!W8) {
                        umma_commit(bar_aempty + 8 * as);
                        if (++as == NA) { as = 0; aph ^= 1; }
                    }
                    umma_commit(bar_dfull + 8 * ds);
                    if (++ds == 2) { ds = 0; dph ^= 1; }
                }
                if (!ok) break;
                umma_commit(bar_empty + 8 * s);
                if (++s == NST) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp >= 12) {
        // ================= codes to bytes =================
        if constexpr (!W8) {
            const int q = warp & 3;
            const int row = q * 32 + lane;  // of the stage
            const uint32_t sw = row & 7;
            const uint32_t my_a = tmem + ((uint32_t)(32 * q) << 16);
            int s = 0, as = 0;
            uint32_t ph = 0, aph = 0, s_hint = 0, a_hint = 0;
            bool ok = true;
            for (int li = 0; li < nloc; li++) {
                ok = __all_sync(0xffffffffu, s_hint || mbar_wait(bar_full + 8 * s, ph, abort_flag));
                if (!ok) break;
                const uint32_t codes = codes0 + s * kQtCodes + row * 128;
#pragma unroll
                for (int u = 0; u < UPC; u++) {
                    ok = __all_sync(0xffffffffu, a_hint || mbar_wait(bar_aempty + 8 * as, aph ^ 1, abort_flag));
                    if (!ok) break;
                    tc_fence_after();
                    constexpr int PC = UG * GS / 32;  // 16-byte pieces (32 codes) of a unit
#pragma unroll
                    for (int i0 = 0; i0 < PC; i0 += 2) {
                        uint4 v[2];
#pragma unroll
                        for (int j = 0; j < 2; j++) v[j] = lds128(codes + (((uint32_t)(u * PC + i0 + j) ^ sw) << 4));
                        const uint32_t w[8] = {v[0].x, v[0].y, v[0].z, v[0].w, v[1].x, v[1].y, v[1].z, v[1].w};
                        uint32_t o[16];
                        constexpr uint32_t MSK = 0x0F0F0F0Fu;
#pragma unroll
                        for (int j = 0; j < 8; j++) {  // even inputs, odd inputs of eight
                            o[2 * j] = w[j] & MSK;
                            o[2 * j + 1] = (w[j] >> 4) & MSK;
                        }
                        qt_st16(my_a + as * AC + i0 * 8, o);
                    }
                    qt_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(bar_aready + 8 * as);
                        if (u == UPC - 1) mbar_arrive(bar_empty + 8 * s);
                    }
                    if (++as == NA) { as = 0; aph ^= 1; }
                    a_hint = mbar_test(bar_aempty + 8 * as, aph ^ 1);
                }
                if (!ok) break;
                if (++s == NST) { s = 0; ph ^= 1; }
                s_hint = mbar_test(bar_full + 8 * s, ph);
            }
        }
    } else if (warp >= 4) {
        pdl_wait();
        // ================= digits of the activations =================
        {
            // a lane takes eight inputs of a column, a warp 256 inputs of a row at a time, four rows under way
            constexpr int UC = CI / 8, CPW = 32 / UC, TPG = GS / 8;  // lanes per column, columns per warp, lanes per group
            const int w8 = lane % TPG;
            for (int l0 = (warp - 4) * CPW; l0 < nloc; l0 += 8 * CPW) {
                const int li = min(l0 + lane / UC, nloc - 1), kc = lane % UC * 8, k = (cols[li] & 0x7FFF) * CI + kc;
                const bool live = l0 + lane / UC < nloc && k < p.K;
                unsigned char* const rec = xd + (size_t)(li * (CI / 128) + kc / 128) * XT - 8 * w8;
                float* const sc_out = xs + (size_t)(li * GPC + kc / GS) * (T / 2) * 4;
                const int chunk = (kc & 127) >> 4;
                for (int m0 = 0; m0 < p.M; m0 += 4) {
                    RawX8 raw[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) raw[q] = load_raw_x8(p.x, p.x_dtype, (size_t)min(m0 + q, p.M - 1) * p.ldx + min(k, p.K - 8));
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (m0 + q >= p.M) break;
                        float v[8];
                        unpack_x8(raw[q], p.x_dtype, v);
                        const int col = qt_col(T, m0 + q);
                        unsigned char* dst = rec + col * 128 + ((chunk ^ (col & 7)) << 4) + (kc & 8);
                        float2 sc = make_float2(0.f, 0.f);
                        // (the digits of eight inputs go to dst + 8 * w8, the next digit T rows further)
                        qr_convert<W8, F::G32, W8 ? 8 : 23, T * 128, 1>(v, w8, live, dst, &sc);
                        if (live && w8 == 0) {
                            float* o = sc_out + (col >> 1) * 4 + (col & 1);
                            o[0] = sc.x;
                            o[2] = sc.y;
                        }
                    }
                }
            }
            fence_async_smem();
            mbar_arrive(bar_x);
            if (!mbar_wait(bar_x, 0, abort_flag)) {}  // (a wait that gives up sets the flag, which ends the loops below)
        }
        // ================= sums to floats =================
        const int q = warp & 3, half = (warp - 4) >> 2;
        const int live = (p.M - 2 * half + 3) >> 2;  // pairs with a row
        const uint32_t my_d = tmem + D0 + ((uint32_t)(32 * q) << 16) + half * H;
        int s = 0, ds = 0;
        uint32_t ph = 0, dph = 0, s_hint = 0, d_hint = 0;
        bool ok = true;
        float acc[H], low[ND == 3 ? H : 1];
#pragma unroll
        for (int j = 0; j < H; j++) acc[j] = 0.f;
#pragma unroll
        for (int j = 0; j < (ND == 3 ? H : 1); j++) low[j] = 0.f;
        int slice = 0;
        for (int li = 0; li < nloc; li++) {
            const int cw = cols[li], ng = min(GPC, G - (cw & 0x7FFF) * GPC);
            ok = s_hint || mbar_wait(bar_full + 8 * s, ph, abort_flag);
            const uint32_t sa = scales0 + s * (2 * 128 * SPB) + (q * 32 + lane) * SPB;
            uint32_t scw[GPC / 2], biw[GPC / 2];
#pragma unroll
            for (int b = 0; b < 2; b++) {
                uint32_t (&o)[GPC / 2] = b ? biw : scw;
                const uint32_t a = sa + b * 128 * SPB;
                if constexpr (GPC == 8) {
                    const uint4 r = lds128(a);
                    o[0] = r.x; o[1] = r.y; o[2] = r.z; o[3] = r.w;
                } else if constexpr (GPC == 4) {
                    const uint2 r = lds64(a);
                    o[0] = r.x; o[1] = r.y;
                } else {
                    o[0] = lds32(a);
                }
            }
            const uint32_t xsb = xs0 + li * (GPC * T * 8) + half * (PAIRS * 16);
#pragma unroll
            for (int u = 0; u < UPC; u++) {
                ok = __all_sync(0xffffffffu, ok && (d_hint || mbar_wait(bar_dfull + 8 * ds, dph, abort_flag)));
                if (!ok) break;
                tc_fence_after();
                // a unit's sums in one go, tensor memory handed back before they are used, the next barriers asked (see qmv_tile.cuh)
                int d[UG][ND][H];
                if (live > 0) {
                    const uint32_t td = my_d + ds * DC;
#pragma unroll
                    for (int g = 0; g < UG; g++)
#pragma unroll
                        for (int i = 0; i < ND; i++) qt_ld(td + g * NB + i * T, d[g][i]);
#pragma unroll
                    for (int g = 0; g < UG; g++)
#pragma unroll
                        for (int i = 0; i < ND; i++) qw_wait_ld(d[g][i]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_dempty + 8 * ds);
                if (++ds == 2) { ds = 0; dph ^= 1; }
                d_hint = mbar_test(bar_dfull + 8 * ds, dph);
                if (u == UPC - 1) s_hint = mbar_test(bar_full + 8 * (s + 1 == NST ? 0 : s + 1), s + 1 == NST ? ph ^ 1 : ph);
                auto body = [&](auto np_c, auto full_c) {  // FULL: no branches between the groups' operations
                    constexpr int NP = decltype(np_c)::value;
                    constexpr bool FULL = decltype(full_c)::value;
#pragma unroll
                    for (int g = 0; g < UG; g++) {
                        const int gs = u * UG + g;
                        if (FULL || gs < ng) {
                            const float sc = __uint_as_float(gs & 1 ? scw[gs / 2] & 0xFFFF0000u : scw[gs / 2] << 16);
                            const float bi = __uint_as_float(gs & 1 ? biw[gs / 2] & 0xFFFF0000u : biw[gs / 2] << 16);
#pragma unroll
                            for (int j = 0; j < NP; j++) {
                                const uint4 xv = lds128(xsb + (gs * (T / 2) + j) * 16);
                                const float x0f = __uint_as_float(xv.x), x1f = __uint_as_float(xv.y);
                                scaled_add2(acc[2 * j], acc[2 * j + 1], (float)(d[g][0][2 * j] * 256 + d[g][1][2 * j]),
                                            (float)(d[g][0][2 * j + 1] * 256 + d[g][1][2 * j + 1]),
                                            sc, sc, x0f, x1f);
                                fma2(acc[2 * j], acc[2 * j + 1], bi, bi, __uint_as_float(xv.z), __uint_as_float(xv.w));
                                if constexpr (ND == 3)
                                    scaled_add2(low[2 * j], low[2 * j + 1], (float)d[g][ND - 1][2 * j], (float)d[g][ND - 1][2 * j + 1], sc, sc, x0f * 0.0078125f, x1f * 0.0078125f);
                            }
                        }
                    }
                };
                if (live <= 0) continue;
                if (ng < GPC) body(std::integral_constant<int, PAIRS>{}, std::false_type{});
                else if (live >= PAIRS) body(std::integral_constant<int, PAIRS>{}, std::true_type{});
                else if (PAIRS == 4 && live == 3) body(std::integral_constant<int, PAIRS == 4 ? 3 : 1>{}, std::true_type{});
                else body(std::integral_constant<int, PAIRS == 4 ? 2 : 1>{}, std::true_type{});
            }
            if (!ok) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_empty + 8 * s);
            if (++s == NST) { s = 0; ph ^= 1; }
            if (cw & 0x8000) {  // the slice is complete
#pragma unroll
                for (int j = 0; j < H; j++) {
                    const float v = ND == 3 ? acc[j] + low[ND == 3 ? j : 0] : acc[j];
                    part[(size_t)(slice * T + 4 * (j >> 1) + 2 * half + (j & 1)) * 128 + q * 32 + lane] = v;
                    acc[j] = 0.f;
                    if (ND == 3) low[ND == 3 ? j : 0] = 0.f;
                }
                slice++;
            }
        }
    }

    __syncwarp();
    if (*abort_flag && warp == 2) {  // copies in flight land before the shared memory is given back
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
    }
    // ---- the slices meet: CTA r finishes rows r, r + cluster, ... of the activations ----
    cluster_sync_all();
    pdl_wait();
    const int mine = (p.M - rank + p.cluster - 1) / p.cluster;
    const uint32_t part0 = smem_u32(part);
    auto sum = [&](int m, int l) {
        float v = 0.f;
        for (int j = 0; j < p.wk; j++) {
            const int r = ((j + 1) * p.cluster - 1) / p.wk;
            v += ld_dsmem_f32(part0 + (((j - p.wk * r / p.cluster) * T + m) * 128 + l) * 4, (uint32_t)r);
        }
        return v;
    };
    if (*abort_flag == 0)
        for (int o = threadIdx.x; o < mine * NROWS; o += kQwThreads) {
            const int m = rank + o / NROWS * p.cluster, f = o % NROWS, n = n0 + f;
            if (n >= p.N) continue;
            qw_store(p, (size_t)m * p.ldy + n, sum(m, f));
        }
    cluster_sync_all();  // (the others read this CTA's slices)
    if (*abort_flag && threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, kErrTimeout);
}

}  // namespace iq
