// Decode GEMV on int8 tensor-core MMAs for the shapes the staged kernel (qmv_imma.cuh) does not take: any K that is a
// multiple of 64, groups of 32, rows longer than its stages, and the gate + up + activation form of the dense FFN.
//
// Same arithmetic: codes enter m16n8k32 u8 x s8 unconverted, the activations are converted once per CTA to block fixed
// point per group (see qmv_imma.cuh), per group y += s * 2^(e-15) * (256 * acc_hi + acc_lo) + b * sum(x); a row's bits do not
// depend on the other rows of the call.
//
// Digits. 4-bit codes times bf16 scales, plus bf16 biases, are exact in fp16 but for a few, and the fp16 MMAs that ran these
// shapes took bf16 and fp16 activations as they are: 2e-7 off the 64-bit product (2880 inputs). 16 bits relative to a group's
// largest value are 8e-6 off it, and 2e-4 where a few inputs are 100 times the rest. So the 4-bit formats take 23 bits, which
// hold every bf16 value down to 2^-15 of the group's largest, in three digits. Up to four rows: the eight columns of an MMA are
// two rows of (high, middle), (low, low), so that a lane's two accumulators are digits of one product, and the row's two lanes
// meet with the K slices. From five rows on: three MMAs per eight rows, one per digit, and the lane adds the two parts itself: the
// same sums. 8-bit codes were rounded in fp16 weights (2e-4): 16 bits, four rows of (high, low) per MMA. What the third digit
// costs: 14336 x 4160 at one row nothing (15.6 -> 14.6 us), at 4 rows 17.2 -> 18.8, at 16 rows (two launches) 32 -> 42; the fp16
// kernel took 18.1, 23.8 and 40.6.
//
// Bound: HBM, which wants 45 KB and more under way per SM all the time. Weights loaded into registers a batch ahead came to 16
// to 32 KB (2.3 TB/s with eight rows' state beside them). Here every warp runs a ring of its own in shared memory: a slot is
// 128 bytes of 16 weight rows (of each matrix), one tensor copy with the 128-byte swizzle, and those rows' scales and biases
// by asynchronous copies of 4 to 16 bytes per lane; the warp issues them itself, `depth` slots ahead and across the blocks of
// rows, and waits on its own barriers, so that the only synchronisation of the CTA is where the K slices of a block of 16 rows
// meet. Warps are wk K slices (every wk-th 128-byte column, or runs of them) x row blocks; the host picks the split (csrc/qmv.cu). Against the
// register batches: 8-bit FFN 2048 -> 7680 -> 2048 at 3 rows 27.2 -> 21.2 us, at 12 rows 72.6 -> 46.9; 4-bit 4096 -> 14336 at
// one row 42.9 -> 36.0, at 8 rows 105 -> 82 (16-bit digits 72).
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "ptx.cuh"
#include "qmv_imma.cuh"

namespace iq {

constexpr int kQrMaxWarps = 16;
constexpr int kQrBox = 2048;  // bytes of a slot's codes per matrix

// How the activations' digits lie in shared memory, per group of inputs and set of rows: 16 bits, sets of four rows; 24 bits,
// sets of two rows; 23 bits, sets of eight (each digit of all rows together).
enum : int { kQr16 = 0, kQr23 = 1, kQr23Tall = 2 };
__host__ __device__ constexpr int qr_rows(int lay) { return lay == kQr16 ? 4 : (lay == kQr23 ? 2 : 8); }
__host__ __device__ constexpr int qr_record(bool g32, int lay) { return (lay == kQr16 ? 2 : 3) * (g32 ? 32 : 64); }  // digits of a group and row
__host__ __device__ constexpr int qr_scales(int lay) { return lay == kQr23Tall ? 8 : 4; }   // float2 {2^(e-15), sum x} of a group and set
__host__ __device__ constexpr int qr_sums(int lay) { return lay == kQr23Tall ? 128 : 64; }  // sums of a set and 16 weight rows

// Eight inputs (unit w8 of a group, its threads neighbouring lanes) as block fixed point, in B-fragment order: the digits from
// the highest down, four lanes' fragments each, STEP bytes from digit to digit. BITS: of a digit; 23: three digits, and SE
// scale entries (two: for the lane with the high and middle digits, with the sum, and for the one with the low digit).
template <bool W8, bool G32, int BITS, int STEP, int SE>
__device__ __forceinline__ void qr_convert(const float (&v)[8], int w8, bool live, unsigned char* rec, float2* scale_out) {
    constexpr int TPG = G32 ? 4 : 8;
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
    qi_group_scale<BITS == 23 ? 8 : BITS>(amax, sum, scale, inv);
    if (!live) return;
    unsigned char* f = rec + (G32 ? w8 * 8 : (w8 >> 1) * 16 + (w8 & 1) * 8);
    if (BITS == 23) {
        if (w8 == 0) {
            scale_out[0] = make_float2(scale, sum);
            if (SE == 2) scale_out[SE - 1] = make_float2(scale * 0.0078125f, 0.f);
        }
        uint32_t d[3][2];
        qi_digits23<W8>(v, inv, d);
#pragma unroll
        for (int i = 0; i < 3; i++) *reinterpret_cast<uint2*>(f + i * STEP) = make_uint2(d[i][0], d[i][1]);
    } else {
        if (w8 == 0) *scale_out = make_float2(scale, sum);
        uint32_t hi_w[2], lo_w[2];
        qi_digits8<W8, BITS == 23 ? 8 : BITS>(v, inv, hi_w, lo_w);
        *reinterpret_cast<uint2*>(f) = make_uint2(hi_w[0], hi_w[1]);
        *reinterpret_cast<uint2*>(f + STEP) = make_uint2(lo_w[0], lo_w[1]);
    }
}

// The rows of a call converted once, for CTAs that would each spend longer on it: [rows][groups] records of the digits and of
// {scale, sum} (two entries with 23 bits). 256 threads, a unit of eight inputs each.
template <bool W8, bool G32, bool WIDE>
__global__ void __launch_bounds__(256) qr_convert_kernel(const void* x, int32_t x_dtype, int64_t ldx, int K, int M, int bits, unsigned char* digits, float2* scale) {
    constexpr int TPG = G32 ? 4 : 8, REC = qr_record(G32, WIDE ? kQr23 : kQr16), STEP = G32 ? 32 : 64;
    pdl_launch_dependents();
    pdl_wait();
    const int units = M * (K / 8), u = blockIdx.x * 256 + threadIdx.x, uc = min(u, units - 1);
    float v[8];
    load_x8(x, x_dtype, (size_t)(uc / (K / 8)) * ldx + (uc % (K / 8)) * 8, v);
    const size_t rec = uc / TPG;  // (K is a multiple of the group)
    if (WIDE) qr_convert<W8, G32, 23, STEP, 2>(v, uc % TPG, u < units, digits + rec * REC, scale + 2 * rec);
    else if (bits == 7) qr_convert<W8, G32, 7, STEP, 1>(v, uc % TPG, u < units, digits + rec * REC, scale + rec);
    else qr_convert<W8, G32, 8, STEP, 1>(v, uc % TPG, u < units, digits + rec * REC, scale + rec);
}

struct QrMaps {
    CUtensorMap w[2];
};
struct QrParams {
    const unsigned char* s[2];
    const unsigned char* b[2];
    int32_t N, K, M;       // weight rows (of each matrix), inputs, activation rows (<= MS sets)
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
inline size_t qr_smem(int32_t fmt, int K, int nw, int lay, int ms, bool vec, int warps, int depth) {
    const size_t gs = fmt == kFmtAffine4G32 ? 32 : 64, G = K / gs;
    return 1024 + (size_t)warps * depth * nw * (kQrBox + 2 * 16 * qr_swords(fmt, vec) * 4) + G * ms * (qr_rows(lay) * qr_record(gs == 32, lay) + qr_scales(lay) * 8) +
           (size_t)2 * warps * nw * ms * qr_sums(lay) * 4 + (size_t)warps * depth * 8 + 16;
}

// FMT: kFmtAffine4, kFmtAffine4G32 or kFmtAffine8; MS: sets of activation rows; NW: matrices (2: gate and up); VEC: the
// scales of a slot's row can be copied as one aligned piece (K a multiple of 256, at 8 bits of 128); LAY: kQr16, kQr23, kQr23Tall.
template <int FMT, int MS, int NW, bool VEC, int LAY>
__global__ void __launch_bounds__(kQrMaxWarps * 32, 1) qmv_ring_kernel(const __grid_constant__ QrMaps maps, const QrParams p) {
    constexpr bool W8 = FMT == kFmtAffine8, G32 = FMT == kFmtAffine4G32;
    constexpr int GS = G32 ? 32 : 64;                  // inputs per group
    constexpr int GPC = qr_groups(FMT);                // groups per slot
    constexpr int SPW = qr_swords(FMT, VEC);
    constexpr int XL = GS / 4;                         // bytes of a lane's B fragment per group and row set: 8 or 16
    constexpr int TPG = GS / 8;                        // threads per group in the conversion
    constexpr bool WIDE = LAY != kQr16, TALL = LAY == kQr23Tall;
    constexpr int RPS = qr_rows(LAY), SPS = qr_scales(LAY), SE = SPS / RPS;  // rows, scale entries of a set; entries of a row
    constexpr int REC = qr_record(G32, LAY), SETB = RPS * REC;               // digits of a group: of a row, of a set
    constexpr int DSTEP = (TALL ? 8 : 1) * 4 * XL, RSTEP = TALL ? 4 * XL : REC;  // from digit to digit, from row to row of a set
    constexpr int FPS = qr_sums(LAY), AC = TALL ? 8 : 2;                     // sums of a set: of a warp, of a lane
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int nwarps = blockDim.x >> 5, depth = p.depth;
    const int G = p.K / GS, ncol = (G + GPC - 1) / GPC;
    unsigned char* xq = smem + (size_t)nwarps * depth * NW * kQrBox;               // [groups][MS][rows][digits][4 lanes] XL bytes (tall: [digits][rows])
    float2* xsc = reinterpret_cast<float2*>(xq + (size_t)G * MS * SETB);           // [groups][MS][SPS] {2^(e-15), sum x}
    float* red = reinterpret_cast<float*>(xsc + (size_t)G * MS * SPS);             // [2][warps][NW * MS * FPS]
    uint32_t* srings = reinterpret_cast<uint32_t*>(red + (size_t)2 * nwarps * NW * MS * FPS);
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
    // (rows the call does not have keep what the memory held: a column of B feeds its own column of D, which nobody reads)
    if (p.xd != nullptr) {
        constexpr int PC = REC / 16, PD = XL / 4;  // 16-byte pieces of a record, of a digit
        for (int m = 0; m < p.M; m++) {
            const uint32_t d = smem_u32(xq) + (m / RPS) * SETB + (m % RPS) * RSTEP, sd = smem_u32(xsc) + m * SE * 8;
            const unsigned char* src = p.xd + (size_t)m * G * REC;
            for (int j = tid; j < G * PC; j += nthreads) cp_async_cg16(d + (j / PC) * (MS * SETB) + (j % PC) / PD * DSTEP + (j % PD) * 16, src + (size_t)j * 16);
            for (int j = tid; j < G; j += nthreads) cp_async_ca<SE * 8>(sd + j * (SPS * MS * 8), p.xs + ((size_t)m * G + j) * (WIDE ? 2 : 1));
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    const int units = p.xd != nullptr ? 0 : G * TPG * p.M, upad = (units + 31) / 32 * 32;  // whole warps: the groups' shuffles need their threads
    // row of unit u (no division for a single row: it is a fair part of that call's prologue)
    auto row_of = [&](int u) { return p.M == 1 ? 0 : u / (G * TPG); };
    auto convert = [&](const float (&v)[8], int u, int m) {
        const int j = (u - m * (G * TPG)) / TPG;
        unsigned char* rec = xq + (size_t)(j * MS + m / RPS) * SETB + (m % RPS) * RSTEP;
        float2* sc = xsc + j * SPS * MS + m * SE;
        if (WIDE) qr_convert<W8, G32, 23, DSTEP, SE>(v, u % TPG, u < units, rec, sc);
        else if (p.runs) qr_convert<W8, G32, 7, DSTEP, SE>(v, u % TPG, u < units, rec, sc);
        else qr_convert<W8, G32, 8, DSTEP, SE>(v, u % TPG, u < units, rec, sc);
    };
    if (units <= 2 * nthreads) {
        for (int u = tid; u < upad; u += nthreads) {
            const int uc = min(u, units - 1), m = row_of(uc);
            float v[8];
            load_x8(p.x, p.x_dtype, (size_t)m * p.ldx + (uc - m * (G * TPG)) * 8, v);
            convert(v, u, m);
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
                convert(v, u0 + q * nthreads, (u0 + q * nthreads) / (G * TPG));
            }
        }
    }
    __syncthreads();

    // lane (g, t) feeds column g: its digit of its row (kQr23: the row's fourth column takes the low digit as well)
    const uint32_t xq32 = smem_u32(xq) + (LAY == kQr23 ? ((g >> 2) * 3 + min(g & 3, 2)) * 4 * XL + t * XL : lane * XL);
    const uint32_t xsc32 = smem_u32(xsc) + t * (TALL ? 16 : 8);
    auto bf = [](uint32_t w, int hi_half) { return __uint_as_float(hi_half ? (w & 0xFFFF0000u) : (w << 16)); };
    // a lane's two accumulators are the columns 2t and 2t + 1 (kQr23, odd t: twice the low digit, of which one counts)
    const int radix = TALL ? 256 : WIDE ? (t & 1 ? 0 : 256) : (p.runs ? 128 : 256);
    const bool shifted = odd_rows && (g & 1);  // rows g and g + 8 start in the middle of a word
    int slot = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int sb = lo, it = 0; sb < hi; sb++, it++) {
        float acc[NW][MS][AC];
#pragma unroll
        for (int i = 0; i < NW; i++)
#pragma unroll
            for (int c = 0; c < MS; c++)
#pragma unroll
                for (int q = 0; q < AC; q++) acc[i][c][q] = 0.f;
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
                    constexpr int DB = TALL ? 3 : 1, XS = TALL ? 2 : 1;  // B fragments of a set, rows of a lane's accumulators
                    uint2 xb[MS][DB][2];
                    float2 xs[MS][XS];
#pragma unroll
                    for (int c = 0; c < MS; c++) {
#pragma unroll
                        for (int i = 0; i < DB; i++) {
                            const uint32_t a = xq32 + (grp * MS + c) * SETB + i * DSTEP;
                            if (G32) {
                                xb[c][i][0] = lds64(a);
                            } else {
                                const uint4 r = lds128(a);
                                xb[c][i][0] = make_uint2(r.x, r.y);
                                xb[c][i][1] = make_uint2(r.z, r.w);
                            }
                        }
                        const uint32_t a = xsc32 + (grp * MS + c) * SPS * 8;
                        if (TALL) {
                            const uint4 sr = lds128(a);
                            xs[c][0] = make_float2(__uint_as_float(sr.x), __uint_as_float(sr.y));
                            xs[c][XS - 1] = make_float2(__uint_as_float(sr.z), __uint_as_float(sr.w));
                        } else {
                            const uint2 sr = lds64(a);
                            xs[c][0] = make_float2(__uint_as_float(sr.x), __uint_as_float(sr.y));
                        }
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
                        int d[MS][DB][4];
#pragma unroll
                        for (int c = 0; c < MS; c++)
#pragma unroll
                            for (int q = 0; q < DB; q++) imma16832_u8s8(d[c][q], a[0][0], a[0][1], a[0][2], a[0][3], xb[c][q][0].x, xb[c][q][0].y, z);
                        if (!G32) {
#pragma unroll
                            for (int c = 0; c < MS; c++)
#pragma unroll
                                for (int q = 0; q < DB; q++) imma16832_u8s8(d[c][q], a[1][0], a[1][1], a[1][2], a[1][3], xb[c][q][1].x, xb[c][q][1].y, d[c][q]);
                        }
#pragma unroll
                        for (int c = 0; c < MS; c++) {
                            if (TALL) {  // accumulator q: activation row 2 t + q % 2 of the set, weight row g + 8 (q / 2)
#pragma unroll
                                for (int q = 0; q < 4; q++) {
                                    const float s = q < 2 ? sc0 : sc1, x = xs[c][q % XS].x;
                                    float &hi = acc[i][c][q % AC], &lo = acc[i][c][(4 + q) % AC];
                                    hi = fmaf((float)(d[c][0][q] * radix + d[c][DB / 2][q]), s * x, hi);
                                    hi = fmaf(q < 2 ? bi0 : bi1, xs[c][q % XS].y, hi);
                                    lo = fmaf((float)d[c][DB - 1][q], s * (x * 0.0078125f), lo);
                                }
                            } else {
                                const float v0 = (float)(d[c][0][0] * radix + d[c][0][1]), v1 = (float)(d[c][0][2] * radix + d[c][0][3]);
                                acc[i][c][0] = fmaf(v0, sc0 * xs[c][0].x, acc[i][c][0]);
                                acc[i][c][0] = fmaf(bi0, xs[c][0].y, acc[i][c][0]);
                                acc[i][c][1] = fmaf(v1, sc1 * xs[c][0].x, acc[i][c][1]);
                                acc[i][c][1] = fmaf(bi1, xs[c][0].y, acc[i][c][1]);
                            }
                        }
                    }
                }
            }
            __syncwarp();  // every lane has read the slot
            if (ok) issue();
            if (++slot == depth) { slot = 0; ph ^= 1; }
        }
        // ---- the K slices meet in shared memory (two buffers: one barrier per round) -------------------------------------
        float* mine = red + ((it & 1) * nwarps + warp) * (NW * MS * FPS);
#pragma unroll
        for (int i = 0; i < NW; i++)
#pragma unroll
            for (int c = 0; c < MS; c++) {
                if (TALL)
                    *reinterpret_cast<float4*>(mine + (i * MS + c) * FPS + lane * 4) =
                        make_float4(acc[i][c][0] + acc[i][c][4 % AC], acc[i][c][1] + acc[i][c][5 % AC], acc[i][c][2 % AC] + acc[i][c][6 % AC], acc[i][c][3 % AC] + acc[i][c][7 % AC]);
                else *reinterpret_cast<float2*>(mine + (i * MS + c) * FPS + lane * 2) = make_float2(acc[i][c][0], acc[i][c][1]);
            }
        __syncthreads();
        for (int o = tid; o < rbs * 16 * RPS * MS; o += nthreads) {
            const int rbi = o / (16 * RPS * MS), c = o / (16 * RPS) % MS, mm = (o >> 4) % RPS, r = o & 15, m = RPS * c + mm, blk = sb * rbs + rbi;
            if (m >= p.M || blk >= nblk) continue;
            const float* part = red + ((it & 1) * nwarps + rbi * p.wk) * (NW * MS * FPS) + c * FPS +
                                (TALL ? (4 * (r & 7) + (mm >> 1)) * 4 + (r >> 3) * 2 + (mm & 1) : (4 * (r & 7) + mm * SE) * 2 + (r >> 3));
            float v[NW];
#pragma unroll
            for (int i = 0; i < NW; i++) v[i] = 0.f;
            for (int k = 0; k < p.wk; k++)
#pragma unroll
                for (int i = 0; i < NW; i++) {
                    const float* q = part + (k * NW + i) * MS * FPS;
                    v[i] += LAY == kQr23 ? q[0] + q[2] : q[0];
                }
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
