// MoE decode tiles on the 5th-generation tensor cores with integers: the expert tiles' gate + up + activation and down projections
// for up to eight routed rows, affine 4-bit experts in groups of 64.
//
//   P[128 weight rows, digits x tokens] = Q[128, 64] * X[digits x tokens, 64]^T     per group of 64 inputs, exact in int32
//   y[row, token] += s[row, group] * 2^(e - 15) * (256 * P_hi + P_lo) + b[row, group] * sum(x)
//
// Same arithmetic as qmv_imma_grouped.cuh: the codes enter the MMA unconverted, the activations as two signed 8-bit digits per input,
// block fixed point per group (fixed_rows.cuh). What differs is who does the work. On mma.sync every warp loads fragments, scatters scales by
// shuffles and holds chains of dependent MMAs: 77 instructions per 16 rows and group at 0.48 issued per cycle, 3.3 TB/s. Here one
// thread issues tcgen05.mma (kind::i8) for 128 rows; a lane is a weight row for good, so that a row's scale and bias are that
// lane's own, and what is left are two streams of independent instructions: codes to bytes (16-byte shared-memory loads, masks,
// tcgen05.st: 24 instructions per 32 rows and group) and sums to floats (tcgen05.ld, four instructions per pair of tokens).
//
// With two digits K is walked in the slices that the grouped kernel cuts it into, each with an accumulator of its own, and h is rounded to halves before the
// down projection's digits are made, as there: a layer has the same bits whole and in expert-parallel pieces (sums in one accumulator and h's digits from
// 32 bits had been 3.2e-4 away from them).
//
// A step is 256 inputs: four groups, 128 bytes of codes per row. Warp roles of one of two persistent CTAs per SM:
//   warp 0      the tile's activation rows (digits, scales), gathered by asynchronous copies into the MMA's swizzled layout
//   warp 1      allocates tensor memory, issues tcgen05.mma
//   warp 2      packed codes: tensor copies, 128-byte swizzle
//   warp 3      the rows' scales and biases
//   4-7 (4-11)  sums to floats, a thread per weight row; at the end of a tile activation and stores
//   the last 4  codes to bytes: A operand in tensor memory, a thread per weight row
// Tensor memory (256 columns per CTA): the sums twice, the A operand in two slots of four groups (three digits: four of two), so that conversion, MMA and
// sums of three steps overlap.
// The gate/up form takes 64 gate rows and the matching 64 up rows (lanes 0-15 of a quadrant gate, lanes 16-31 up), as qmm_ta.cuh does.
// Every wait is bounded: on a timeout the kernel writes a status word, all roles drain and tensor memory is released.
//
// Replaces the reference's vnax_moe_gateup* / vnax_moe_down_split* decode kernels (Shaders/verify_nax.metal:258-509).
#pragma once

#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "fixed_rows.cuh"
#include "gqmv.cuh"
#include "ptx.cuh"
#include "umma_i8.cuh"

namespace iq {

constexpr int qt_sums(int nd) { return nd - 1; }       // sets of four warps that turn sums into floats
constexpr int qt_threads(int nd) { return 256 + 128 * qt_sums(nd); }
constexpr int kQtRows = 8;                          // token rows per tile
constexpr int kQtXs = 4 * kQtRows * 8;              // [group][pair of tokens]{scale, scale, sum, sum}
constexpr int kQtScales = 2 * 128 * 8;              // scales and biases of the weight rows
constexpr int qt_x_bytes(int nd) { return 2 * nd * kQtRows * 128; }  // digits of a step: [pair of groups][digit][token][128]
constexpr int qt_stage(int nd) { return kQtCodes + qt_x_bytes(nd) + kQtScales + kQtXs; }
// Four stages, 64 KB of codes per CTA. Beside two digits a fifth would fit, but would take the L1 that serves a row's four pieces of a sector of scales
// (MoE of 128 experts 2048 x 768, 64 tokens: 106.9 us with five, 99.9 with four, 101.7 with three)
constexpr int kQtStages = 4;
constexpr int qt_smem(int nd) { return 1024 + kQtStages * qt_stage(nd) + 256; }  // alignment, stages, barriers

struct QtParams {
    const void* s[2];
    const void* b[2];
    int32_t expert_lo;
    int32_t N, K;              // weight rows per expert (gate/up: of each matrix), inputs
    FixedRows x;
    const uint32_t* row_map;   // sorted position -> pair id (row of x = pair / topk); null: rows are in place
    int32_t topk;
    int32_t slice;             // steps of 256 inputs whose sums are one accumulator's (two digits; gate/up: 1)
    const Tile* tiles;
    const uint32_t* ntiles;
    __half* y;
    int64_t ldy;
    const float* ebias[2];
    float limit;
    int32_t act;
    int32_t early;             // the tile list is complete when this kernel starts
    int32_t vec;               // scales by asynchronous copies of eight bytes (else in pairs of bytes)
    int32_t* status;
};
struct QtMaps {
    CUtensorMap w[2];
};

// EPI: 0 store, 1 gate + up + activation. ND: digits of an input, two or three (16 or 23 bits, see qmv_ring.cuh)
template <int EPI, int ND>
__global__ void __launch_bounds__(qt_threads(ND), 2) qmv_tile_kernel(const __grid_constant__ QtMaps maps, const QtParams p) {
    constexpr int T = kQtRows, NB = ND == 2 ? 16 : 32;         // MMA columns: digit, token (of three digits 24 are used)
    constexpr int UG = ND == 2 ? 4 : 2, NA = ND == 2 ? 2 : 4;  // groups per hand-over to the MMA and back; slots of A
    constexpr int UPS = 4 / UG;                                // hand-overs per step
    // Three digits: two sets of warps for the sums, with half of the pairs of tokens each (128 experts of 2880 x 768, 64
    // tokens: 225 us with one set, 210 with two)
    constexpr int SG = qt_sums(ND), H = T / SG;
    auto col_of = [](int m) { return SG == 2 ? qt_col(T, m) : m; };  // column of token m among its digit's
    constexpr uint32_t kACols = UG * 16, kDCols = UG * NB, kD0 = NA * kACols;
    static_assert(kD0 + 2 * kDCols <= 256, "256 columns per CTA");
    constexpr int kQtX = qt_x_bytes(ND), kQtStage = qt_stage(ND);
    constexpr int NST = kQtStages;
    constexpr int NROWS = EPI ? 64 : 128;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t codes0 = smem_u32(smem), x0 = codes0 + NST * kQtCodes, scales0 = x0 + NST * kQtX, xs0 = scales0 + NST * kQtScales;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)NST * kQtStage);
    const uint32_t bar_full = smem_u32(bars), bar_xfull = bar_full + 8 * kQtStages, bar_empty = bar_xfull + 8 * kQtStages;
    const uint32_t bar_aready = bar_empty + 8 * kQtStages, bar_aempty = bar_aready + 32, bar_dfull = bar_aempty + 32, bar_dempty = bar_dfull + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * kQtStages + 12);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NST; i++) {
            mbar_init(bar_full + 8 * i, 1 + 32);   // the codes' copy, the lanes' copies of scales
            mbar_init(bar_xfull + 8 * i, 32);
            mbar_init(bar_empty + 8 * i, 4 + 1 + 4 * SG);  // codes to bytes, the MMAs, sums to floats
        }
        for (int i = 0; i < NA; i++) {
            mbar_init(bar_aready + 8 * i, 4);
            mbar_init(bar_aempty + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(bar_dfull + 8 * i, 1);
            mbar_init(bar_dempty + 8 * i, 4 * SG);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // With p.early (the kernel before this one lets its dependents start after its own wait) the tile list and the weights may be read at once
    const bool weights_only = warp == 2 || warp == 3 || warp >= 4 + 4 * SG;
    if (!p.early || !weights_only) pdl_wait();
    pdl_launch_dependents();

    const int G = p.K / 64, steps = (G + 3) / 4;
    const int nblk = (p.N + NROWS - 1) / NROWS;
    const int total = (int)(*p.ntiles) * nblk;
    struct Item {
        int expert, row0, rows, n0;
    };
    auto item = [&](int i, Item& t) -> bool {
        if (i >= total) return false;
        const Tile l = p.tiles[i / nblk];
        t.expert = (int)l.expert - p.expert_lo; t.row0 = (int)l.start; t.rows = min((int)l.count, T);
        t.n0 = (i % nblk) * NROWS;
        return true;
    };
    const int first = blockIdx.x, stride = gridDim.x;

    if (warp == 0) {
        // ================= activation rows =================
        // A token's digits of a step (four groups) are one stretch of memory: 16 bytes per lane, 32 pieces in one copy instruction (three digits: the
        // last 16 pieces of two tokens in another). Offsets are worked out once per tile: with them in the loop this warp was what the
        // others waited for (128 experts of 2880 x 768, three digits, 64 tokens: 210 us, 174 so; 2048 x 768, two digits: 99.9, 97). The MMA reads the digits through the asynchronous proxy: each lane waits for its copies, fences and arrives, a stage behind.
        constexpr int LAG = 1, STEP = 4 * ND * 64;  // bytes of a token and step
        auto place = [](int pc, int col) {          // of piece pc (group, digit, quarter) in the stage
            const int gi = pc / (4 * ND), d = pc / 4 % ND, c = pc & 3;
            return (uint32_t)((gi >> 1) * (ND * T * 128) + (d * T + col) * 128 + ((((gi & 1) * 4 + c) ^ col) << 4));
        };
        const int g_a = lane / (4 * ND), pc_b = 32 + (lane & 15), g_b = pc_b / (4 * ND);  // pieces of the two kinds of copies, their groups
        int s = 0, sd = 0, pending = 0;
        uint32_t ph = 0;
        bool ok = true;
        auto done = [&]() {
            fence_async_smem();
            mbar_arrive(bar_xfull + 8 * sd);
            if (++sd == NST) sd = 0;
            pending--;
        };
        Item t;
        for (int i = first; ok && item(i, t); i += stride) {
            // lane m: the row of token m
            uint32_t row = t.row0 + min(lane, t.rows - 1);
            if (p.row_map != nullptr) row = p.row_map[row] / (uint32_t)p.topk;
            const unsigned char* src[T];
            uint32_t dst_b[T / 2];
            const unsigned char* src_b[T / 2];
#pragma unroll
            for (int m = 0; m < T; m++) src[m] = p.x.digits + (size_t)__shfl_sync(0xffffffffu, row, m) * G * (ND * 64) + lane * 16;
#pragma unroll
            for (int m = 0; m < (ND == 3 ? T / 2 : 0); m++) {
                const int mb = 2 * m + (lane >> 4);
                src_b[m] = p.x.digits + (size_t)__shfl_sync(0xffffffffu, row, mb) * G * (ND * 64) + pc_b * 16;
                dst_b[m] = place(pc_b, col_of(mb));
            }
            const int mx = lane >> 2, gx = lane & 3;  // scales: token and group
            const float2* sx = p.x.scale + (size_t)__shfl_sync(0xffffffffu, row, mx) * G + gx;
            const uint32_t dst_x = (gx * (T / 2) + (col_of(mx) >> 1)) * 16 + (mx & 1) * 4;
            for (int st = 0; st < steps; st++) {
                ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag));
                if (!ok) break;
                const int ng = min(4, G - 4 * st);
                const uint32_t xb = x0 + s * kQtX, xsb = xs0 + s * kQtXs;
#pragma unroll
                for (int m = 0; m < T; m++)
                    if (m < t.rows && g_a < ng) cp_async_cg16(xb + place(lane, col_of(m)), src[m] + (size_t)st * STEP);
                if constexpr (ND == 3) {
#pragma unroll
                    for (int m = 0; m < T / 2; m++)
                        if (2 * m + (lane >> 4) < t.rows && g_b < ng) cp_async_cg16(xb + dst_b[m], src_b[m] + (size_t)st * STEP);
                }
                if (mx < t.rows && gx < ng) {
                    cp_async_ca<4>(xsb + dst_x, &sx[4 * st].x);
                    cp_async_ca<4>(xsb + dst_x + 8, &sx[4 * st].y);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                pending++;
                if (pending > LAG) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(LAG) : "memory");
                    done();
                }
                if (++s == NST) { s = 0; ph ^= 1; }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        while (pending > 0) done();
    } else if (warp == 2) {
        // ================= packed codes =================
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            Item t;
            for (int i = first; ok && item(i, t); i += stride) {
                const int wrow = t.expert * p.N + t.n0;
                for (int st = 0; st < steps; st++) {
                    if (!(ok = mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag))) break;
                    mbar_arrive_expect_tx(bar_full + 8 * s, kQtCodes);
                    const uint32_t dst = codes0 + s * kQtCodes;
                    tma_load_2d(dst, &maps.w[0], bar_full + 8 * s, st * 128, wrow);
                    if (EPI) tma_load_2d(dst + kQtCodes / 2, &maps.w[1], bar_full + 8 * s, st * 128, wrow);
                    if (++s == NST) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 3) {
        // ================= scales and biases: eight bytes of each per row and step =================
        const size_t pitch = (size_t)G * 2;
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        Item t;
        for (int it = first; ok && item(it, t); it += stride) {
            const char* src[4][2];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                // (rows beyond the matrix take the last row's: nothing of theirs is stored)
                const int row = lane + 32 * i, mi = EPI ? i >> 1 : 0, n = min(t.n0 + (EPI ? row & 63 : row), p.N - 1);
                const size_t o = ((size_t)t.expert * p.N + n) * pitch;
                src[i][0] = static_cast<const char*>(p.s[mi]) + o;
                src[i][1] = static_cast<const char*>(p.b[mi]) + o;
            }
            for (int st = 0; st < steps; st++) {
                ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag));
                if (!ok) break;
                const uint32_t dst = scales0 + s * kQtScales + lane * 8;
                if (p.vec) {
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int m = 0; m < 2; m++) cp_async_ca<8>(dst + m * 1024 + i * 256, src[i][m] + st * 8);
                    cp_async_arrive_noinc(bar_full + 8 * s);
                } else {
                    const int left = (int)pitch - st * 8;
                    uint32_t v[4][2][4];
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int m = 0; m < 2; m++)
#pragma unroll
                            for (int e = 0; e < 4; e++) v[i][m][e] = ldg_nc_u16(src[i][m] + st * 8 + min(2 * e, left - 2));
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int m = 0; m < 2; m++)
#pragma unroll
                            for (int e = 0; e < 2; e++) sts32(dst + m * 1024 + i * 256 + 4 * e, v[i][m][2 * e] | (v[i][m][2 * e + 1] << 16));
                    mbar_arrive(bar_full + 8 * s);
                }
                if (++s == NST) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        if (elect_one()) {
            int s = 0, as = 0, ds = 0;
            uint32_t ph = 0, aph = 0, dph = 0;
            const uint32_t idesc = qt_idesc(NB), xdesc0 = (x0 & 0x3FFFFu) >> 4;
            bool ok = true;
            Item t;
            for (int i = first; ok && item(i, t); i += stride) {
                for (int st = 0; st < steps && ok; st++) {
                    if (!(ok = mbar_wait_hint(0, bar_xfull + 8 * s, ph, abort_flag))) break;
#pragma unroll
                    for (int u = 0; u < UPS; u++) {
                        if (!(ok = mbar_wait_hint(0, bar_aready + 8 * as, aph, abort_flag))) break;
                        if (!(ok = mbar_wait_hint(0, bar_dempty + 8 * ds, dph ^ 1, abort_flag))) break;
                        tc_fence_after();
                        const uint32_t ta = tmem + as * kACols, td = tmem + kD0 + ds * kDCols;
#pragma unroll
                        for (int g = 0; g < UG; g++) {
                            const int gs = u * UG + g;  // of the step: its pair's tile, its half of the rows' 128 bytes
                            const uint32_t xdesc = xdesc0 + s * (kQtX >> 4) + (gs >> 1) * (ND * T * 8) + (gs & 1) * 4;
#pragma unroll
                            for (int kk = 0; kk < 2; kk++)
                                umma_i8_ta(td + g * NB, ta + g * 16 + kk * 8, kQtDescHi | (uint64_t)(xdesc + 2 * kk), idesc, kk);
                        }
                        umma_commit(bar_aempty + 8 * as);
                        umma_commit(bar_dfull + 8 * ds);
                        if (++as == NA) { as = 0; aph ^= 1; }
                        if (++ds == 2) { ds = 0; dph ^= 1; }
                    }
                    if (!ok) break;
                    umma_commit(bar_empty + 8 * s);
                    if (++s == NST) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp >= 4 + 4 * SG) {
        // ================= codes to bytes =================
        const int q = warp & 3;
        const int row = EPI ? (lane >> 4) * 64 + q * 16 + (lane & 15) : q * 32 + lane;  // row of the stage
        const uint32_t sw = row & 7;
        const uint32_t my_a = tmem + ((uint32_t)(32 * q) << 16);
        int s = 0, as = 0;
        uint32_t ph = 0, aph = 0, s_hint = 0, a_hint = 0;
        bool ok = true;
        Item t;
        for (int i = first; ok && item(i, t); i += stride) {
            for (int st = 0; st < steps; st++) {
                ok = s_hint || mbar_wait(bar_full + 8 * s, ph, abort_flag);
                const uint32_t codes = codes0 + s * kQtCodes + row * 128;
#pragma unroll
                for (int u = 0; u < UPS; u++) {
                    ok = __all_sync(0xffffffffu, ok && (a_hint || mbar_wait(bar_aempty + 8 * as, aph ^ 1, abort_flag)));
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int g0 = 0; g0 < UG; g0 += 2) {
                        uint4 v[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) v[j] = lds128(codes + (((uint32_t)(2 * (u * UG + g0) + j) ^ sw) << 4));
#pragma unroll
                        for (int g = 0; g < 2; g++) {
                            const uint32_t w[8] = {v[2 * g].x, v[2 * g].y, v[2 * g].z, v[2 * g].w, v[2 * g + 1].x, v[2 * g + 1].y, v[2 * g + 1].z, v[2 * g + 1].w};
                            uint32_t o[16];
                            constexpr uint32_t MSK = 0x0F0F0F0Fu;
#pragma unroll
                            for (int j = 0; j < 8; j++) {  // even inputs, odd inputs of eight
                                o[2 * j] = w[j] & MSK;
                                o[2 * j + 1] = (w[j] >> 4) & MSK;
                            }
                            qt_st16(my_a + as * kACols + (g0 + g) * 16, o);
                        }
                    }
                    qt_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(bar_aready + 8 * as);
                        if (u == UPS - 1) mbar_arrive(bar_empty + 8 * s);
                    }
                    if (++as == NA) { as = 0; aph ^= 1; }
                    a_hint = mbar_test(bar_aempty + 8 * as, aph ^ 1);
                }
                if (!ok) break;
                if (++s == NST) { s = 0; ph ^= 1; }
                s_hint = mbar_test(bar_full + 8 * s, ph);
            }
        }
    } else {
        // ================= sums to floats =================
        const int q = warp & 3;
        const int mi = EPI ? lane >> 4 : 0;
        const int nl = EPI ? q * 16 + (lane & 15) : q * 32 + lane;
        const int row = EPI ? mi * 64 + nl : nl;
        const int half = (warp - 4) >> 2;  // SG 2: tokens 4 j + 2 half and the next one
        auto token = [half](int j) { return SG == 2 ? 4 * (j >> 1) + 2 * half + (j & 1) : j; };  // of accumulator j
        const uint32_t my_d = tmem + kD0 + ((uint32_t)(32 * q) << 16) + half * H;
        int s = 0, ds = 0;
        uint32_t ph = 0, dph = 0;
        bool ok = true;
        Item t;
        for (int i = first; ok && item(i, t); i += stride) {
            float acc[H], low[ND == 3 ? H : 1], tot[ND == 2 ? H : 1];
#pragma unroll
            for (int j = 0; j < H; j++) acc[j] = low[ND == 3 ? j : 0] = tot[ND == 2 ? j : 0] = 0.f;
            int left = p.slice;
            const int n = t.n0 + nl, live = SG == 2 ? (t.rows - 2 * half + 3) >> 2 : (t.rows + 1) >> 1;  // pairs with a token
            const bool n_ok = n < p.N;
            const float* eb = mi ? p.ebias[1] : p.ebias[0];
            const float bias = eb != nullptr && n_ok ? eb[(size_t)(t.expert) * p.N + n] : 0.f;
            for (int st = 0; st < steps; st++) {
                const int ng = min(4, G - 4 * st);
                ok = mbar_wait(bar_full + 8 * s, ph, abort_flag) && mbar_wait(bar_xfull + 8 * s, ph, abort_flag);
                const uint2 scw = lds64(scales0 + s * kQtScales + row * 8), biw = lds64(scales0 + s * kQtScales + 1024 + row * 8);
                const uint32_t xsb = xs0 + s * kQtXs + half * (H / 2 * 16);
#pragma unroll
                for (int u = 0; u < UPS; u++) {
                    ok = __all_sync(0xffffffffu, ok && mbar_wait(bar_dfull + 8 * ds, dph, abort_flag));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t td = my_d + ds * kDCols;
                    // NP: the pairs of tokens that the tile has. FULL: a step of four groups. The next group's sums are under way while one's are used; tensor
                    // memory is handed back with the last ones in registers. Two pairs at a time over the unit's groups: with all four at once the sums under
                    // way, the slices' and the tile's take more than the 80 registers (MoE block of 128 experts 2048 x 768, 64 tokens: 105.2 us, 97.9 so).
                    auto body = [&](auto np_c, auto full_c) {
                        constexpr int NP = decltype(np_c)::value;
                        constexpr bool FULL = decltype(full_c)::value;
                        constexpr int PP = ND == 2 ? 2 : H / 2, NQ = (NP + PP - 1) / PP * UG;  // pairs per pass, loads
                        int d[2][ND][2 * PP];
                        auto fetch = [&](int q) {
#pragma unroll
                            for (int i = 0; i < ND; i++) qt_ld(td + q % UG * NB + i * T + q / UG * 2 * PP, d[q & 1][i]);
                        };
                        fetch(0);
#pragma unroll
                        for (int q = 0; q < NQ; q++) {
                            const int e = q & 1, g = q % UG, j0 = q / UG * PP, gs = u * UG + g;
                            qt_ld_wait(d[e][0], d[e][1]);
                            if (ND == 3) qt_ld_wait(d[e][0], d[e][ND - 1]);
                            if (q + 1 < NQ) fetch(q + 1);
                            if (q + 1 == NQ) {
                                tc_fence_before();
                                __syncwarp();
                                if (lane == 0) mbar_arrive(bar_dempty + 8 * ds);
                            }
                            if (!FULL && gs >= ng) continue;
                            const uint32_t sw = gs < 2 ? scw.x : scw.y, bw = gs < 2 ? biw.x : biw.y;
                            const float sc = __uint_as_float(gs & 1 ? sw & 0xFFFF0000u : sw << 16), bi = __uint_as_float(gs & 1 ? bw & 0xFFFF0000u : bw << 16);
#pragma unroll
                            for (int j = j0; j < NP && j < j0 + PP; j++) {
                                const int c = 2 * (j - j0);
                                const uint4 xv = lds128(xsb + (gs * (T / 2) + j) * 16);
                                const float x0f = __uint_as_float(xv.x), x1f = __uint_as_float(xv.y);
                                // The third digit's sum keeps the first ones' factor and is divided by 128 at the end: no products of its own (MoE block of 64
                                // experts of 7168 x 2048 at 32 tokens 501 -> 475 us, 128 of 2880 x 768 152.7 -> 150.9)
                                const float h0 = (float)(d[e][0][c] * 256 + d[e][1][c]), h1 = (float)(d[e][0][c + 1] * 256 + d[e][1][c + 1]);
                                if constexpr (ND == 3)
                                    scaled_add2_low(acc[2 * j], acc[2 * j + 1], low[2 * j], low[2 * j + 1], h0, h1, (float)d[e][2][c], (float)d[e][2][c + 1], sc, x0f, x1f);
                                else if (EPI && g == 0)  // (the first one of a slice: no zeros)
                                    scaled_mul2(acc[2 * j], acc[2 * j + 1], h0, h1, sc, x0f, x1f);
                                else
                                    scaled_add2(acc[2 * j], acc[2 * j + 1], h0, h1, sc, sc, x0f, x1f);
                                fma2(acc[2 * j], acc[2 * j + 1], bi, bi, __uint_as_float(xv.z), __uint_as_float(xv.w));
                                if (EPI && ND == 2 && g == UG - 1)  // the slice (a step) is complete
                                    fma2(tot[ND == 2 ? 2 * j : 0], tot[ND == 2 ? 2 * j + 1 : 0], acc[2 * j], acc[2 * j + 1], 1.f, 1.f);
                            }
                        }
                    };
                    constexpr int PAIRS = H / 2;
                    if (live <= 0) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_dempty + 8 * ds);
                    } else if (ng < 4) {
                        body(std::integral_constant<int, PAIRS>{}, std::false_type{});
                    } else if (live >= PAIRS) {
                        body(std::integral_constant<int, PAIRS>{}, std::true_type{});
                    } else if (PAIRS == 4 && live == 3) {
                        body(std::integral_constant<int, PAIRS == 4 ? 3 : 1>{}, std::true_type{});
                    } else if (PAIRS == 4 && live == 2) {
                        body(std::integral_constant<int, PAIRS == 4 ? 2 : 1>{}, std::true_type{});
                    } else {
                        body(std::integral_constant<int, 1>{}, std::true_type{});
                    }
                    if (++ds == 2) { ds = 0; dph ^= 1; }
                }
                if (!ok) break;
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_empty + 8 * s);
                if (++s == NST) { s = 0; ph ^= 1; }
                if (ND == 2 && !EPI && --left == 0) {  // the slice is complete
#pragma unroll
                    for (int j = 0; j < H; j++) {
                        tot[ND == 2 ? j : 0] += acc[j];
                        acc[j] = 0.f;
                    }
                    left = p.slice;
                }
            }
            if (!ok) break;
            // ---- the tile's outputs ----
#pragma unroll
            for (int j = 0; j < H; j++) acc[j] = ND == 3 ? acc[j] + fmaf(low[ND == 3 ? j : 0], 0.0078125f, bias) : tot[ND == 2 ? j : 0] + bias;
            if (EPI) {
                // lanes l and l + 16 hold gate and up of one feature: the lower lane finishes the even tokens, the upper one the odd ones
                __half* yp = p.y + (size_t)t.row0 * p.ldy + n;
#pragma unroll
                for (int j = 0; j < H / 2; j++) {
                    if (j >= live) break;
                    const float other = __shfl_xor_sync(0xffffffffu, mi ? acc[2 * j] : acc[2 * j + 1], 16);
                    const float g = mi ? other : acc[2 * j], up = mi ? acc[2 * j + 1] : other;
                    const int m = token(2 * j) + mi;
                    if (n_ok && m < t.rows) yp[(size_t)m * p.ldy] = __float2half_rn(glu_rt(p.act, g, up, p.limit));
                }
            } else if (n_ok) {
                __half* yp = p.y + (size_t)t.row0 * p.ldy + n;
#pragma unroll
                for (int j = 0; j < H; j++) {
                    if (token(j) >= t.rows) break;
                    yp[(size_t)token(j) * p.ldy] = __float2half_rn(acc[j]);
                }
            }
        }
    }

    __syncwarp();
    // ---- teardown ----
    if (*abort_flag && (warp == 0 || warp == 2)) {  // copies in flight land before the shared memory is given back
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, kErrTimeout);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
    }
}

// Rows as block fixed point, where no other kernel leaves them so: grid-stride over the rows
template <bool WIDE>
__global__ void __launch_bounds__(256) fixed_rows_kernel(const void* x, int32_t x_dtype, int64_t ldx, int rows, int D, const FixedRows fx) {
    pdl_wait();
    pdl_launch_dependents();
    const int units = D / 8, upad = (units + 31) / 32 * 32;
    for (int r = blockIdx.x; r < rows; r += gridDim.x)
        for (int u = threadIdx.x; u < upad; u += 256) {
            const bool live = u < units;
            const size_t o = (size_t)r * ldx + (live ? u : 0) * 8, g = (size_t)r * (D / 64) + (live ? u : 0) / 8;
            float v[8];
            load_x8(x, x_dtype, o, v);
            fixed_point_unit<WIDE>(v, u & 7, live ? fx.digits + g * (WIDE ? 192 : 128) : nullptr, fx.scale + g);
        }
}

}  // namespace iq
