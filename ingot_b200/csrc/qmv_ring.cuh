// Decode GEMV on int8 tensor-core MMAs for the shapes the staged kernel (qmv_imma.cuh) does not take: any K that is a
// multiple of 64, groups of 32, rows longer than its stages, and the gate + up + activation form of the dense FFN.
//
// Same arithmetic: codes enter m16n8k32 u8 x s8 unconverted, the activations are converted once per CTA to block fixed
// point per group (two signed 8-bit digits, see qmv_imma.cuh), per group y += s * 2^(e-15) * (256 * acc_hi + acc_lo) +
// b * sum(x); a row's bits do not depend on the other rows of the call.
//
// Bound: HBM, which wants 45 KB and more under way per SM all the time. Weights loaded into registers a batch ahead came to 16
// to 32 KB (2.3 TB/s with eight rows' state beside them). Here every warp runs a ring of its own in shared memory: a slot is
// 128 bytes of 16 weight rows (of each matrix), one tensor copy with the 128-byte swizzle, and those rows' scales and biases
// by asynchronous copies of 4 to 16 bytes per lane; the warp issues them itself, `depth` slots ahead and across the blocks of
// rows, and waits on its own barriers, so that the only synchronisation of the CTA is where the K slices of a block of 16 rows
// meet. Warps are wk K slices (every wk-th 128-byte column, or runs of them) x row blocks; the host picks the split (csrc/qmv.cu). Against the
// register batches: 8-bit FFN 2048 -> 7680 -> 2048 at 3 rows 27.2 -> 21.2 us, at 12 rows 72.6 -> 46.9; 4-bit 4096 -> 14336 at
// one row 42.9 -> 36.2, at 8 rows 105 -> 72.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "ptx.cuh"
#include "qmv_imma.cuh"

namespace iq {

constexpr int kQrMaxWarps = 16;
constexpr int kQrBox = 2048;  // bytes of a slot's codes per matrix

// Eight inputs (unit w8 of a group, its threads neighbouring lanes) as block fixed point, in B-fragment order: the high digits
// at f, the low ones four lanes' fragments on.
template <bool W8, bool G32, int BITS>
__device__ __forceinline__ void qr_convert(const float (&v)[8], int w8, bool live, unsigned char* rec, float2* scale_out) {
    constexpr int TPG = G32 ? 4 : 8, XL = G32 ? 8 : 16;
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
    qi_group_scale<BITS>(amax, sum, scale, inv);
    if (!live) return;
    if (w8 == 0) *scale_out = make_float2(scale, sum);
    uint32_t hi_w[2], lo_w[2];
    qi_digits8<W8, BITS>(v, inv, hi_w, lo_w);
    unsigned char* f = rec + (G32 ? w8 * 8 : (w8 >> 1) * 16 + (w8 & 1) * 8);
    *reinterpret_cast<uint2*>(f) = make_uint2(hi_w[0], hi_w[1]);
    *reinterpret_cast<uint2*>(f + 4 * XL) = make_uint2(lo_w[0], lo_w[1]);
}

// The rows of a call converted once, for CTAs that would each spend longer on it: [rows][groups] records of the digits (128
// bytes; groups of 32: 64) and of {scale, sum}. 256 threads, a unit of eight inputs each.
template <bool W8, bool G32>
__global__ void __launch_bounds__(256) qr_convert_kernel(const void* x, int32_t x_dtype, int64_t ldx, int K, int M, int bits, unsigned char* digits, float2* scale) {
    constexpr int TPG = G32 ? 4 : 8, REC = G32 ? 64 : 128;
    pdl_launch_dependents();
    pdl_wait();
    const int units = M * (K / 8), u = blockIdx.x * 256 + threadIdx.x, uc = min(u, units - 1);
    float v[8];
    load_x8(x, x_dtype, (size_t)(uc / (K / 8)) * ldx + (uc % (K / 8)) * 8, v);
    const size_t rec = uc / TPG;  // (K is a multiple of the group)
    if (bits == 7) qr_convert<W8, G32, 7>(v, uc % TPG, u < units, digits + rec * REC, scale + rec);
    else qr_convert<W8, G32, 8>(v, uc % TPG, u < units, digits + rec * REC, scale + rec);
}

struct QrMaps {
    CUtensorMap w[2];
};
struct QrParams {
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
    int32_t wk, depth;     // K slices; slots per warp
    int32_t runs;          // as the staged kernel: 7-bit digits, slices are runs of columns (else every wk-th column: 5 % faster)
    const unsigned char* xd;  // the rows as qr_convert_kernel left them, or null: converted here, from x
    const float2* xs;
    int32_t* status;
};

// Words of scales (and as many of biases) per weight row and slot; rows that do not start on a word boundary take one more.
__host__ __device__ constexpr int qr_groups(int32_t fmt) { return fmt == kFmtAffine8 ? 2 : (fmt == kFmtAffine4G32 ? 8 : 4); }  // groups per 128 bytes
__host__ __device__ constexpr int qr_swords(int32_t fmt, bool vec) { return qr_groups(fmt) / 2 + (vec ? 0 : 1); }
// Shared memory of a CTA: rings, fragments and scales of the activations, two buffers of partial sums, barriers, flag.
inline size_t qr_smem(int32_t fmt, int K, int nw, int ms, bool vec, int warps, int depth) {
    const size_t gs = fmt == kFmtAffine4G32 ? 32 : 64, G = K / gs;
    return 1024 + (size_t)warps * depth * nw * (kQrBox + 2 * 16 * qr_swords(fmt, vec) * 4) + G * ms * (32 * (gs / 4) + 32) +
           (size_t)2 * warps * nw * ms * 256 + (size_t)warps * depth * 8 + 16;
}

// FMT: kFmtAffine4, kFmtAffine4G32 or kFmtAffine8; MS: sets of four activation rows; NW: matrices (2: gate and up); VEC: the
// scales of a slot's row can be copied as one aligned piece (K a multiple of 256, at 8 bits of 128).
template <int FMT, int MS, int NW, bool VEC>
__global__ void __launch_bounds__(kQrMaxWarps * 32, 1) qmv_ring_kernel(const __grid_constant__ QrMaps maps, const QrParams p) {
    constexpr bool W8 = FMT == kFmtAffine8, G32 = FMT == kFmtAffine4G32;
    constexpr int GS = G32 ? 32 : 64;                  // inputs per group
    constexpr int GPC = qr_groups(FMT);                // groups per slot
    constexpr int SPW = qr_swords(FMT, VEC);
    constexpr int XL = GS / 4;                         // bytes of a lane's B fragment per group and row set: 8 or 16
    constexpr int TPG = GS / 8;                        // threads per group in the conversion
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int nwarps = blockDim.x >> 5, depth = p.depth;
    const int G = p.K / GS, ncol = (G + GPC - 1) / GPC;
    unsigned char* xq = smem + (size_t)nwarps * depth * NW * kQrBox;               // [groups][MS][32 lanes] XL bytes
    float2* xsc = reinterpret_cast<float2*>(xq + (size_t)G * MS * 32 * XL);        // [groups][MS * 4 rows] {2^(e-15), sum x}
    float* red = reinterpret_cast<float*>(xsc + (size_t)G * MS * 4);               // [2][warps][NW * MS * 64]
    uint32_t* srings = reinterpret_cast<uint32_t*>(red + (size_t)2 * nwarps * NW * MS * 64);
    uint64_t* bars = reinterpret_cast<uint64_t*>(srings + (size_t)nwarps * depth * NW * 2 * 16 * SPW);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + nwarps * depth);
    const uint32_t ring = smem_u32(smem) + warp * depth * NW * kQrBox;
    const uint32_t sring = smem_u32(srings) + warp * depth * NW * 2 * 16 * SPW * 4;
    const uint32_t bar = smem_u32(bars) + warp * depth * 8;
    if (lane == 0) {
        for (int i = 0; i < depth; i++) mbar_init(bar + 8 * i, 1 + 32);  // the codes' copy, the lanes' copies of scales
        if (warp == 0) *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    __syncwarp();
    pdl_launch_dependents();

    // ---- this warp's items: its column of blocks of 16 rows, its share of their 128-byte columns --------------------------
    const int rbs = nwarps / p.wk, rb = warp / p.wk, ks = warp % p.wk;
    const int nblk = p.N / 16, nsup = (nblk + rbs - 1) / rbs;
    const int lo = (int)((int64_t)nsup * blockIdx.x / gridDim.x), hi = (int)((int64_t)nsup * (blockIdx.x + 1) / gridDim.x);
    auto block_of = [&](int sb) { return sb * rbs + rb; };
    const int step = p.runs ? 1 : p.wk, col0 = p.runs ? ncol * ks / p.wk : ks, col1 = p.runs ? ncol * (ks + 1) / p.wk : ncol;
    int psb = lo, pcol = col0, pslot = 0;  // the next item to ask for
    const bool odd_rows = (G & 1) != 0;
    auto issue = [&]() {
        const int blk = block_of(psb);
        if (psb >= hi || blk >= nblk) return;
        const uint32_t full = bar + 8 * pslot;
        if (elect_one()) {
            mbar_arrive_expect_tx(full, NW * kQrBox);
#pragma unroll
            for (int i = 0; i < NW; i++) tma_load_2d(ring + (pslot * NW + i) * kQrBox, &maps.w[i], full, pcol * 128, blk * 16);
        }
        // lane l: scales (l < 16) or biases of row l % 16
        const int row = lane & 15;
        const int64_t o = ((int64_t)(blk * 16 + row) * G + pcol * GPC) * 2;
#pragma unroll
        for (int i = 0; i < NW; i++) {
            const unsigned char* src = (lane < 16 ? p.s[i] : p.b[i]) + o;
            const uint32_t dst = sring + (((pslot * NW + i) * 2 + (lane >> 4)) * 16 + row) * SPW * 4;
            if (VEC) {
                cp_async_ca<SPW * 4>(dst, src);
            } else {  // the words that hold the row's remaining scales, never a byte past them
                const unsigned char* base = src - (odd_rows && (row & 1) ? 2 : 0);
                const int64_t left = (int64_t)min(GPC, G - pcol * GPC) * 2 + (src - base);
#pragma unroll
                for (int j = 0; j < SPW; j++) {
                    const int64_t n = left - 4 * j;
                    cp_async4_zfill(dst + 4 * j, base + (n > 0 ? 4 * j : 0), n >= 4 ? 4 : (n > 0 ? (int)n : 0));
                }
            }
        }
        cp_async_arrive_noinc(full);
        if (++pslot == depth) pslot = 0;
        if ((pcol += step) >= col1) { pcol = col0; psb++; }
    };
    for (int i = 0; i < depth; i++) issue();  // the weights do not depend on the previous kernel of the stream
    pdl_wait();

    // ---- activations -> block fixed point, two 8-bit digits, in B-fragment order (see qmv_imma.cuh) ---------------------
    const int nthreads = nwarps * 32;
    for (int u = tid; u < G * TPG * (4 * MS - p.M); u += nthreads) {  // rows the call does not have: zero digits and scale
        const int m = p.M + u / (G * TPG), j = (u / TPG) % G, w8 = u % TPG;
        unsigned char* f = xq + ((size_t)(j * MS + (m >> 2)) * 32 + 8 * (m & 3)) * XL + (G32 ? w8 * 8 : (w8 >> 1) * 16 + (w8 & 1) * 8);
        *reinterpret_cast<uint2*>(f) = make_uint2(0, 0);
        *reinterpret_cast<uint2*>(f + 4 * XL) = make_uint2(0, 0);
        if (w8 == 0) xsc[j * 4 * MS + m] = make_float2(0.f, 0.f);
    }
    if (p.xd != nullptr) {
        constexpr int PC = XL / 2;  // 16-byte pieces of a record
        for (int m = 0; m < p.M; m++) {
            const uint32_t d = smem_u32(xq) + ((m >> 2) * 32 + 8 * (m & 3)) * XL, sd = smem_u32(xsc) + m * 8;
            const unsigned char* src = p.xd + (size_t)m * G * PC * 16;
            for (int j = tid; j < G * PC; j += nthreads) cp_async_cg16(d + (j / PC) * (MS * 32 * XL) + (j % PC) * 16, src + (size_t)j * 16);
            for (int j = tid; j < G; j += nthreads) cp_async_ca<8>(sd + j * (4 * MS * 8), p.xs + (size_t)m * G + j);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    const int units = p.xd != nullptr ? 0 : G * TPG * p.M, upad = (units + 31) / 32 * 32;  // whole warps: the groups' shuffles need their threads
    auto convert = [&](const float (&v)[8], int u) {
        const int m = u / (G * TPG), j = (u / TPG) % G;
        unsigned char* rec = xq + ((size_t)(j * MS + (m >> 2)) * 32 + 8 * (m & 3)) * XL;
        if (p.runs) qr_convert<W8, G32, 7>(v, u % TPG, u < units, rec, xsc + j * 4 * MS + m);
        else qr_convert<W8, G32, 8>(v, u % TPG, u < units, rec, xsc + j * 4 * MS + m);
    };
    if (units <= 2 * nthreads) {
        for (int u = tid; u < upad; u += nthreads) {
            const int uc = min(u, units - 1);
            float v[8];
            load_x8(p.x, p.x_dtype, (size_t)(uc / (G * TPG)) * p.ldx + (uc % (G * TPG)) * 8, v);
            convert(v, u);
        }
    } else {  // four loads under way per thread
        for (int u0 = tid; u0 < upad; u0 += 4 * nthreads) {
            RawX8 raw[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int u = min(u0 + q * nthreads, units - 1);
                raw[q] = load_raw_x8(p.x, p.x_dtype, (size_t)(u / (G * TPG)) * p.ldx + (u % (G * TPG)) * 8);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (u0 + q * nthreads >= upad) break;  // (whole warps)
                float v[8];
                unpack_x8(raw[q], p.x_dtype, v);
                convert(v, u0 + q * nthreads);
            }
        }
    }
    __syncthreads();

    const uint32_t xq32 = smem_u32(xq) + lane * XL, xsc32 = smem_u32(xsc) + t * 8;
    auto bf = [](uint32_t w, int hi_half) { return __uint_as_float(hi_half ? (w & 0xFFFF0000u) : (w << 16)); };
    const int radix = p.runs ? 128 : 256;
    const bool shifted = odd_rows && (g & 1);  // rows g and g + 8 start in the middle of a word
    int slot = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int sb = lo, it = 0; sb < hi; sb++, it++) {
        float acc[NW][MS][2];
#pragma unroll
        for (int i = 0; i < NW; i++)
#pragma unroll
            for (int c = 0; c < MS; c++) acc[i][c][0] = acc[i][c][1] = 0.f;
        for (int col = block_of(sb) < nblk ? col0 : col1; col < col1; col += step) {
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar + 8 * slot, ph, abort_flag));
            if (ok) {
                uint32_t sc[NW][2][GPC / 2], bi[NW][2][GPC / 2];
#pragma unroll
                for (int i = 0; i < NW; i++)
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            const uint32_t a = sring + (((slot * NW + i) * 2 + q) * 16 + g + 8 * h) * SPW * 4;
                            uint32_t (&o)[GPC / 2] = q ? bi[i][h] : sc[i][h];
                            if (!VEC) {
                                uint32_t w[SPW];
#pragma unroll
                                for (int j = 0; j < SPW; j++) w[j] = lds32(a + 4 * j);
#pragma unroll
                                for (int j = 0; j < GPC / 2; j++) o[j] = shifted ? __funnelshift_r(w[j], w[j + 1 < SPW ? j + 1 : j], 16) : w[j];
                            } else if (GPC == 8) {
                                const uint4 r = lds128(a);
                                o[0] = r.x; o[GPC > 2 ? 1 : 0] = r.y; o[GPC > 4 ? 2 : 0] = r.z; o[GPC > 4 ? 3 : 0] = r.w;
                            } else if (GPC == 4) {
                                const uint2 r = lds64(a);
                                o[0] = r.x; o[GPC > 2 ? 1 : 0] = r.y;
                            } else {
                                o[0] = lds32(a);
                            }
                        }
                const uint32_t rows = ring + slot * NW * kQrBox + g * 128;
#pragma unroll
                for (int u = 0; u < GPC; u++) {
                    const int grp = col * GPC + u;
                    if (!VEC && grp >= G) break;
                    const int z[4] = {0, 0, 0, 0};
                    uint2 xb[MS][2];
                    float2 xs[MS];
#pragma unroll
                    for (int c = 0; c < MS; c++) {
                        if (G32) {
                            xb[c][0] = lds64(xq32 + (grp * MS + c) * 32 * XL);
                        } else {
                            const uint4 r = lds128(xq32 + (grp * MS + c) * 32 * XL);
                            xb[c][0] = make_uint2(r.x, r.y);
                            xb[c][1] = make_uint2(r.z, r.w);
                        }
                        const uint2 sr = lds64(xsc32 + (grp * MS + c) * 32);
                        xs[c] = make_float2(__uint_as_float(sr.x), __uint_as_float(sr.y));
                    }
#pragma unroll
                    for (int i = 0; i < NW; i++) {
                        // the A fragments of rows g and g + 8: a lane's share of the group, at its swizzled place
                        constexpr uint32_t MSK = 0x0F0F0F0Fu;
                        uint32_t a[2][4];
                        const uint32_t wa = rows + i * kQrBox;
                        if (W8) {
                            const uint32_t o = ((u * 4 + t) ^ g) << 4;
                            const uint4 r0 = lds128(wa + o), r1 = lds128(wa + 1024 + o);
                            a[0][0] = r0.x; a[0][1] = r1.x; a[0][2] = r0.y; a[0][3] = r1.y;
                            a[1][0] = r0.z; a[1][1] = r1.z; a[1][2] = r0.w; a[1][3] = r1.w;
                        } else {
                            uint32_t q0[2], q1[2];
                            if (G32) {
                                const uint32_t o = ((u ^ g) << 4) + t * 4;
                                q0[0] = q0[1] = lds32(wa + o);
                                q1[0] = q1[1] = lds32(wa + 1024 + o);
                            } else {
                                const uint32_t o = (((u * 2 + (t >> 1)) ^ g) << 4) + (t & 1) * 8;
                                const uint2 r0 = lds64(wa + o), r1 = lds64(wa + 1024 + o);
                                q0[0] = r0.x; q0[1] = r0.y; q1[0] = r1.x; q1[1] = r1.y;
                            }
#pragma unroll
                            for (int k = 0; k < 2; k++) {
                                a[k][0] = q0[k] & MSK; a[k][1] = q1[k] & MSK;
                                a[k][2] = (q0[k] >> 4) & MSK; a[k][3] = (q1[k] >> 4) & MSK;
                            }
                        }
                        const float sc0 = bf(sc[i][0][u / 2], u & 1), sc1 = bf(sc[i][1][u / 2], u & 1);
                        const float bi0 = bf(bi[i][0][u / 2], u & 1), bi1 = bf(bi[i][1][u / 2], u & 1);
                        int d[MS][4];
#pragma unroll
                        for (int c = 0; c < MS; c++) imma16832_u8s8(d[c], a[0][0], a[0][1], a[0][2], a[0][3], xb[c][0].x, xb[c][0].y, z);
                        if (!G32) {
#pragma unroll
                            for (int c = 0; c < MS; c++) imma16832_u8s8(d[c], a[1][0], a[1][1], a[1][2], a[1][3], xb[c][1].x, xb[c][1].y, d[c]);
                        }
#pragma unroll
                        for (int c = 0; c < MS; c++) {
                            const float v0 = (float)(d[c][0] * radix + d[c][1]), v1 = (float)(d[c][2] * radix + d[c][3]);
                            acc[i][c][0] = fmaf(v0, sc0 * xs[c].x, acc[i][c][0]);
                            acc[i][c][0] = fmaf(bi0, xs[c].y, acc[i][c][0]);
                            acc[i][c][1] = fmaf(v1, sc1 * xs[c].x, acc[i][c][1]);
                            acc[i][c][1] = fmaf(bi1, xs[c].y, acc[i][c][1]);
                        }
                    }
                }
            }
            __syncwarp();  // every lane has read the slot
            if (ok) issue();
            if (++slot == depth) { slot = 0; ph ^= 1; }
        }
        // ---- the K slices meet in shared memory (two buffers: one barrier per round) -------------------------------------
        float* mine = red + ((it & 1) * nwarps + warp) * (NW * MS * 64);
#pragma unroll
        for (int i = 0; i < NW; i++)
#pragma unroll
            for (int c = 0; c < MS; c++) *reinterpret_cast<float2*>(mine + (i * MS + c) * 64 + lane * 2) = make_float2(acc[i][c][0], acc[i][c][1]);
        __syncthreads();
        for (int o = tid; o < rbs * 64 * MS; o += nthreads) {
            const int rbi = o / (64 * MS), c = (o >> 6) % MS, mm = (o >> 4) & 3, r = o & 15, m = 4 * c + mm, blk = sb * rbs + rbi;
            if (m >= p.M || blk >= nblk) continue;
            const float* part = red + ((it & 1) * nwarps + rbi * p.wk) * (NW * MS * 64) + c * 64 + (4 * (r & 7) + mm) * 2 + (r >> 3);
            float v[NW];
#pragma unroll
            for (int i = 0; i < NW; i++) v[i] = 0.f;
            for (int k = 0; k < p.wk; k++)
#pragma unroll
                for (int i = 0; i < NW; i++) v[i] += part[(k * NW + i) * MS * 64];
            const float f = NW == 2 ? glu_rt(p.act, v[0], v[NW - 1], p.limit) : v[0];
            const size_t y = (size_t)m * p.ldy + (size_t)blk * 16 + r;
            if (p.y_dtype == kF32) {
                float* yp = reinterpret_cast<float*>(p.y) + y;
                *yp = p.accumulate ? *yp + f : f;
            } else if (p.y_dtype == kF16) {
                __half* yp = reinterpret_cast<__half*>(p.y) + y;
                *yp = __float2half_rn(p.accumulate ? __half2float(*yp) + f : f);
            } else {
                uint16_t* yp = reinterpret_cast<uint16_t*>(p.y) + y;
                *yp = (uint16_t)f32_to_bf16_bits(p.accumulate ? bf16_bits_to_f32(*yp) + f : f);
            }
        }
    }
    if (!ok) {  // copies in flight land before the shared memory is given back
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
        if (lane == 0 && p.status != nullptr) atomicExch(p.status, kErrTimeout);
    }
}

}  // namespace iq
