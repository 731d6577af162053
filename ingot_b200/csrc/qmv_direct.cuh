// Decode GEMV on int8 tensor-core MMAs for the shapes the staged kernel (qmv_imma.cuh) does not take: any K that is a
// multiple of 64, groups of 32, rows longer than its stages, and the gate + up + activation form of the dense FFN.
//
// Same arithmetic: codes enter m16n8k32 u8 x s8 unconverted, the activations are converted once per CTA to block fixed
// point per group (two signed 7-bit digits, see qmv_imma.cuh), per group y += s * 2^(e-13) * (128 * acc_hi + acc_lo) +
// b * sum(x); a row's bits do not depend on the other rows of the call. What differs is how the weights arrive: every
// consumer warp loads its fragments straight from global memory into registers, a batch of groups ahead (the next item's
// first batch included), so that nothing about a row's length or alignment has to fit a stage. Eight warps are eight K
// slices of a 16-row block (two blocks, one of each matrix, in the gate/up form); their sums meet in shared memory in slice
// order.
//
// Bound: HBM; in practice the loads in flight (16 warps of an SM hold about 32 KB of codes under way). It replaces kernels
// that dequantised to fp16 and were bound by instruction issue: the 8-bit FFN of width 2048 -> 7680 -> 2048 at three rows
// ran at 17.5 us (gate and up) + 15.6 us (down).
#pragma once

#include "common.cuh"
#include "ptx.cuh"
#include "qmv_imma.cuh"

namespace iq {

constexpr int kQdWarps = 8;
constexpr int kQdThreads = kQdWarps * 32;

struct QdParams {
    const unsigned char* w[2];
    const unsigned char* s[2];
    const unsigned char* b[2];
    int32_t N, K, M;       // weight rows (of each matrix), inputs, activation rows (<= 4 * MS)
    const void* x;
    int32_t x_dtype;
    int64_t ldx;
    void* y;
    int32_t y_dtype;
    int64_t ldy;
    int32_t accumulate;
    int32_t act;           // gate/up form: activation
    float limit;
};

// groups of a warp's K slice per batch of loads: 16 KB of codes under way per CTA and buffer (8-bit or two matrices: half
// the groups)
constexpr int qd_batch(bool w8, int nw) { return (w8 ? 2 : 4) / nw; }

// FMT: kFmtAffine4, kFmtAffine4G32 or kFmtAffine8; MS: sets of four activation rows; NW: matrices (2: gate and up); VEC: a
// batch's scales of a row can be read with one aligned load.
template <int FMT, int MS, int NW, bool VEC>
__global__ void __launch_bounds__(kQdThreads, MS == 1 ? 2 : 1) qmv_direct_kernel(const QdParams p) {
    constexpr bool W8 = FMT == kFmtAffine8, G32 = FMT == kFmtAffine4G32;
    constexpr int GS = G32 ? 32 : 64;                  // inputs per group
    constexpr int GB = W8 ? 64 : GS / 2;               // code bytes of a row per group
    constexpr int U = qd_batch(W8, NW);                // groups per batch
    static_assert(!VEC || U > 1, "one group's scale needs no vector");
    constexpr int LW = GB / 16;                        // words per lane, row and group
    constexpr int XL = GS / 4;                         // bytes of a lane's B fragment per group and row set: 8 or 16
    constexpr int TPG = GS / 8;                        // threads per group in the conversion
    constexpr int SW = VEC ? U / 2 : U;                // words of scales per row and batch: two scales each, or one
    extern __shared__ __align__(16) unsigned char smem[];
    const int G = p.K / GS;
    unsigned char* xq = smem;                                                      // [groups][MS][32 lanes] XL bytes
    float2* xsc = reinterpret_cast<float2*>(smem + (size_t)G * MS * 32 * XL);      // [groups][MS * 4 rows] {2^(e-13), sum x}
    float* red = reinterpret_cast<float*>(xsc + (size_t)G * MS * 4);               // [2][kQdWarps][NW * MS * 64]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    pdl_launch_dependents();

    const int nblk = p.N / 16;
    const int lo = (int)((int64_t)nblk * blockIdx.x / gridDim.x), hi = (int)((int64_t)nblk * (blockIdx.x + 1) / gridDim.x);
    // this warp's K slice, in batches of U groups
    const int batches = (G + U - 1) / U;
    const int b0 = min(batches * warp / kQdWarps, batches - 1), b1 = batches * (warp + 1) / kQdWarps;
    const int64_t row_bytes = (int64_t)G * GB, srow_bytes = (int64_t)G * 2;

    struct Batch {
        uint32_t q[NW][2][U][LW];                // codes of rows g and g + 8
        uint32_t s[NW][2][SW];
        uint32_t b[NW][2][SW];
    };
    auto load = [&](Batch& v, int blk, int bt) {
#pragma unroll
        for (int i = 0; i < NW; i++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int64_t row = (int64_t)blk * 16 + g + 8 * h;
                const unsigned char* wp = p.w[i] + row * row_bytes + t * (GB / 4);
                const unsigned char* sp = p.s[i] + row * srow_bytes;
                const unsigned char* bp = p.b[i] + row * srow_bytes;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int grp = VEC ? bt * U + u : min(bt * U + u, G - 1);  // a short last batch reads its last group again
                    if (LW == 4) {
                        const uint4 r = ldg_nc_u4(wp + (int64_t)grp * GB);
                        v.q[i][h][u][0] = r.x; v.q[i][h][u][LW > 1 ? 1 : 0] = r.y;
                        v.q[i][h][u][LW > 2 ? 2 : 0] = r.z; v.q[i][h][u][LW > 3 ? 3 : 0] = r.w;
                    } else if (LW == 2) {
                        const uint2 r = __ldg(reinterpret_cast<const uint2*>(wp + (int64_t)grp * GB));
                        v.q[i][h][u][0] = r.x; v.q[i][h][u][LW > 1 ? 1 : 0] = r.y;
                    } else {
                        v.q[i][h][u][0] = __ldg(reinterpret_cast<const uint32_t*>(wp + (int64_t)grp * GB));
                    }
                    if (!VEC) {
                        v.s[i][h][VEC ? 0 : u] = ldg_nc_u16(sp + 2 * grp);
                        v.b[i][h][VEC ? 0 : u] = ldg_nc_u16(bp + 2 * grp);
                    }
                }
                if (VEC && U == 4) {
                    const uint2 a = __ldg(reinterpret_cast<const uint2*>(sp + bt * 8)), c = __ldg(reinterpret_cast<const uint2*>(bp + bt * 8));
                    v.s[i][h][0] = a.x; v.s[i][h][SW - 1] = a.y;
                    v.b[i][h][0] = c.x; v.b[i][h][SW - 1] = c.y;
                } else if (VEC) {
                    v.s[i][h][0] = __ldg(reinterpret_cast<const uint32_t*>(sp + bt * 4));
                    v.b[i][h][0] = __ldg(reinterpret_cast<const uint32_t*>(bp + bt * 4));
                }
            }
    };
    // the weights do not depend on the previous kernel of the stream: the first batch is on its way before the wait
    Batch cur, nxt;
    load(cur, lo, b0);  // (the grid has at most one CTA per block: lo < hi)
    pdl_wait();

    // ---- activations -> block fixed point, two 7-bit digits, in B-fragment order (see qmv_imma.cuh) ---------------------
    for (int u = tid; u < G * TPG * (4 * MS - p.M); u += kQdThreads) {  // rows the call does not have: zero digits and scale
        const int m = p.M + u / (G * TPG), j = (u / TPG) % G, w8 = u % TPG;
        unsigned char* f = xq + ((size_t)(j * MS + (m >> 2)) * 32 + 8 * (m & 3)) * XL + (G32 ? w8 * 8 : (w8 >> 1) * 16 + (w8 & 1) * 8);
        *reinterpret_cast<uint2*>(f) = make_uint2(0, 0);
        *reinterpret_cast<uint2*>(f + 4 * XL) = make_uint2(0, 0);
        if (w8 == 0) xsc[j * 4 * MS + m] = make_float2(0.f, 0.f);
    }
    const int units = G * TPG * p.M, upad = (units + 31) / 32 * 32;  // whole warps: the groups' shuffles need their threads
    for (int u = tid; u < upad; u += kQdThreads) {
        const bool live = u < units;
        const int m = live ? u / (G * TPG) : 0, j = (u / TPG) % G, w8 = u % TPG;
        float v[8];
        load_x8(p.x, p.x_dtype, (size_t)m * p.ldx + j * GS + w8 * 8, v);
        float amax = 0.f, sum = 0.f;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            amax = fmaxf(amax, fabsf(v[k]));
            sum += v[k];
        }
#pragma unroll
        for (int o = 1; o < TPG; o <<= 1) {
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
        }
        float scale, inv;
        qi_group_scale(amax, sum, scale, inv);
        if (!live) continue;
        if (w8 == 0) xsc[j * 4 * MS + m] = make_float2(scale, sum);
        uint32_t hi_w[2] = {0, 0}, lo_w[2] = {0, 0};
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int X = __float2int_rn(v[k] * inv);
            const int hi_d = (X + 64) >> 7, lo_d = X - (hi_d << 7);
            const int half = W8 ? (k >> 2) : (k & 1), i = W8 ? (k & 3) : (k >> 1);
            hi_w[half] |= (uint32_t)(hi_d & 0xFF) << (8 * i);
            lo_w[half] |= (uint32_t)(lo_d & 0xFF) << (8 * i);
        }
        unsigned char* f = xq + ((size_t)(j * MS + (m >> 2)) * 32 + 8 * (m & 3)) * XL + (G32 ? w8 * 8 : (w8 >> 1) * 16 + (w8 & 1) * 8);
        *reinterpret_cast<uint2*>(f) = make_uint2(hi_w[0], hi_w[1]);
        *reinterpret_cast<uint2*>(f + 4 * XL) = make_uint2(lo_w[0], lo_w[1]);
    }
    __syncthreads();

    const uint32_t xq32 = smem_u32(xq) + lane * XL, xsc32 = smem_u32(xsc) + t * 8;
    auto bf = [](uint32_t w, int hi_half) { return __uint_as_float(hi_half ? (w & 0xFFFF0000u) : (w << 16)); };
    int it = 0;
    for (int blk = lo; blk < hi; blk++, it++) {
        float acc[NW][MS][2];
#pragma unroll
        for (int i = 0; i < NW; i++)
#pragma unroll
            for (int c = 0; c < MS; c++) acc[i][c][0] = acc[i][c][1] = 0.f;
        auto compute = [&](const Batch& v, int bt) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int grp = bt * U + u;
                if (grp >= G) break;
                const int z[4] = {0, 0, 0, 0};
                uint2 xb[MS][GS / 32];
                float2 xs[MS];
#pragma unroll
                for (int c = 0; c < MS; c++) {
                    if (G32) {
                        xb[c][0] = lds64(xq32 + (grp * MS + c) * 32 * XL);
                    } else {
                        const uint4 r = lds128(xq32 + (grp * MS + c) * 32 * XL);
                        xb[c][0] = make_uint2(r.x, r.y);
                        xb[c][G32 ? 0 : 1] = make_uint2(r.z, r.w);
                    }
                    const uint2 sr = lds64(xsc32 + (grp * MS + c) * 32);
                    xs[c] = make_float2(__uint_as_float(sr.x), __uint_as_float(sr.y));
                }
#pragma unroll
                for (int i = 0; i < NW; i++) {
                    constexpr uint32_t MSK = 0x0F0F0F0Fu;
                    const float sc0 = bf(v.s[i][0][VEC ? u / 2 : u], VEC ? u & 1 : 0), sc1 = bf(v.s[i][1][VEC ? u / 2 : u], VEC ? u & 1 : 0);
                    const float bi0 = bf(v.b[i][0][VEC ? u / 2 : u], VEC ? u & 1 : 0), bi1 = bf(v.b[i][1][VEC ? u / 2 : u], VEC ? u & 1 : 0);
#pragma unroll
                    for (int c = 0; c < MS; c++) {
                        int d[4];
                        const uint32_t* q0 = v.q[i][0][u];
                        const uint32_t* q1 = v.q[i][1][u];
                        if (W8) {
                            imma16832_u8s8(d, q0[0], q1[0], q0[LW > 1 ? 1 : 0], q1[LW > 1 ? 1 : 0], xb[c][0].x, xb[c][0].y, z);
                            imma16832_u8s8(d, q0[LW > 2 ? 2 : 0], q1[LW > 2 ? 2 : 0], q0[LW > 3 ? 3 : 0], q1[LW > 3 ? 3 : 0],
                                           xb[c][GS / 32 - 1].x, xb[c][GS / 32 - 1].y, d);
                        } else {
                            imma16832_u8s8(d, q0[0] & MSK, q1[0] & MSK, (q0[0] >> 4) & MSK, (q1[0] >> 4) & MSK, xb[c][0].x, xb[c][0].y, z);
                            if (!G32)
                                imma16832_u8s8(d, q0[LW > 1 ? 1 : 0] & MSK, q1[LW > 1 ? 1 : 0] & MSK, (q0[LW > 1 ? 1 : 0] >> 4) & MSK,
                                               (q1[LW > 1 ? 1 : 0] >> 4) & MSK, xb[c][GS / 32 - 1].x, xb[c][GS / 32 - 1].y, d);
                        }
                        const float v0 = (float)(d[0] * 128 + d[1]), v1 = (float)(d[2] * 128 + d[3]);
                        acc[i][c][0] = fmaf(v0, sc0 * xs[c].x, acc[i][c][0]);
                        acc[i][c][0] = fmaf(bi0, xs[c].y, acc[i][c][0]);
                        acc[i][c][1] = fmaf(v1, sc1 * xs[c].x, acc[i][c][1]);
                        acc[i][c][1] = fmaf(bi1, xs[c].y, acc[i][c][1]);
                    }
                }
            }
        };
        // the batch after (bt, blk): the next of this slice, else the first of the next item (of this one again at the end:
        // every load is unconditional and its address valid, whatever order the compiler issues them in)
        auto ahead = [&](Batch& v, int bt) {
            const bool same = bt + 1 < b1;
            load(v, same ? blk : min(blk + 1, hi - 1), same ? bt + 1 : b0);
        };
        int bt = b0;
        for (; bt + 1 < b1; bt += 2) {
            ahead(nxt, bt);
            compute(cur, bt);
            ahead(cur, bt + 1);
            compute(nxt, bt + 1);
        }
        if (bt < b1) {  // an odd number of batches: the buffers change places
            ahead(nxt, bt);
            compute(cur, bt);
            cur = nxt;
        }
        // ---- the eight K slices meet in shared memory ----------------------------------------------------------------------
        float* mine = red + ((it & 1) * kQdWarps + warp) * (NW * MS * 64);
#pragma unroll
        for (int i = 0; i < NW; i++)
#pragma unroll
            for (int c = 0; c < MS; c++) {
                mine[(i * MS + c) * 64 + lane * 2] = acc[i][c][0];
                mine[(i * MS + c) * 64 + lane * 2 + 1] = acc[i][c][1];
            }
        __syncthreads();
        if (tid < 64 * MS) {
            const int c = tid >> 6, mm = (tid >> 4) & 3, r = tid & 15, m = 4 * c + mm;
            if (m < p.M) {
                const int slot = c * 64 + (4 * (r & 7) + mm) * 2 + (r >> 3);
                float v[NW];
#pragma unroll
                for (int i = 0; i < NW; i++) {
                    v[i] = 0.f;
                    for (int k = 0; k < kQdWarps; k++) v[i] += red[((it & 1) * kQdWarps + k) * (NW * MS * 64) + i * MS * 64 + slot];
                }
                const float f = NW == 2 ? glu_rt(p.act, v[0], v[NW - 1], p.limit) : v[0];
                const size_t o = (size_t)m * p.ldy + (size_t)blk * 16 + r;
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
        }
    }
}

}  // namespace iq
