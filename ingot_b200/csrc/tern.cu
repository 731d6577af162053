// The rotated ternary format (Bonsai 2): MLX affine 2-bit codes in groups of 128 with an fp16 scale and bias = -scale,
// i.e. w = (q - 1) * s with q in {0, 1, 2}; only the scale is stored. The weights live in a rotated basis: before each
// matrix the activations go through x <- H_1024(x * signs) / 32 per block of 1024 inputs (normalised Sylvester
// Walsh-Hadamard), and the embedding applies the inverse to a table row.
//
// Replaces, on sm_100a, had_rows_h, embed_rows_t and vnax_qmvt* of the reference (Shaders/xc_tern.metal:29-65, 110-230;
// launcher Layers/Linear.swift:298-349). The prefill GEMM of the format is the tcgen05 kernel with a ternary
// dequantiser (csrc/qmm_ta.cuh). The kernels here are small: a 4096 x 4096 ternary matrix is 4 MB.
#include "common.cuh"
#include "internal.h"
#include "ptx.cuh"

namespace iq {
namespace {

// Unnormalised Walsh-Hadamard transform of 1024 floats by 256 threads, thread t holding elements 4 t .. 4 t + 3, in the
// reference's butterfly order (span 1, 2, 4, ...: a + b and a - b), so that the fp32 results are the CPU rule's bits
// (Tests/IngotTests/KernelHarness.swift:196-210). Spans below 4 are a thread's own, below 128 a warp's, and the last three run
// on elements 256 k + t, exchanged through shared memory: two barriers where a barrier per span took ten (a 1024 x 1024 GEMV, which
// is all start-up, 4.6 -> 3.7 us).
__device__ __forceinline__ void fwht1024(float (&v)[4], float* sh, int tid) {
    const int lane = tid & 31;
    float a = v[0], b = v[1], c = v[2], d = v[3];
    v[0] = a + b; v[1] = a - b; v[2] = c + d; v[3] = c - d;
    a = v[0]; b = v[1]; c = v[2]; d = v[3];
    v[0] = a + c; v[2] = a - c; v[1] = b + d; v[3] = b - d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float other = __shfl_xor_sync(0xffffffffu, v[k], o);
            v[k] = (lane & o) ? other - v[k] : v[k] + other;
        }
    __syncthreads();
    reinterpret_cast<float4*>(sh)[tid] = make_float4(v[0], v[1], v[2], v[3]);
    __syncthreads();
    // span 128: elements 256 k + t and its partner 128 away (another thread's: both read them)
    const int base = tid & 127;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float lo = sh[256 * k + base], hi = sh[256 * k + base + 128];
        v[k] = (tid & 128) ? lo - hi : lo + hi;
    }
    a = v[0]; b = v[1]; c = v[2]; d = v[3];
    v[0] = a + b; v[1] = a - b; v[2] = c + d; v[3] = c - d;  // span 256
    a = v[0]; b = v[1]; c = v[2]; d = v[3];
    v[0] = a + c; v[2] = a - c; v[1] = b + d; v[3] = b - d;  // span 512
}

// y[r, block] = half(H(x[r, block] * signs[block]) / 32). Grid (K / 1024, rows), 256 threads.
__global__ void __launch_bounds__(256) had_rows_kernel(const void* __restrict__ x, int32_t x_dtype, int64_t ldx,
                                                      const float* __restrict__ signs, __half* __restrict__ y, int64_t ldy) {
    __shared__ __align__(16) float sh[1024];
    pdl_launch_dependents();  // (ahead of the wait: the GEMV fetches codes and scales meanwhile; behind it 9216 x 5120, one row, 10.5 -> 11.0 us)
    const int tid = threadIdx.x, k0 = blockIdx.x * 1024;
    pdl_wait();
    float v[4];
    load_x4(x, x_dtype, (size_t)blockIdx.y * ldx + k0 + tid * 4, v);
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] *= signs[k0 + tid * 4 + j];
    fwht1024(v, sh, tid);
#pragma unroll
    for (int k = 0; k < 4; k++) y[(size_t)blockIdx.y * ldy + k0 + 256 * k + tid] = __float2half_rn(v[k] * (1.0f / 32.0f));
}

// Ternary embedding: row tokens[r] dequantised, inverse rotation (H / 32, then the signs), fp32 and / or fp16 out.
// One block of 256 threads per output row; a token outside the table gives a zero row.
__global__ void __launch_bounds__(256) embed_rows_tern_kernel(const uint32_t* __restrict__ tokens, const uint32_t* __restrict__ w,
                                                             const __half* __restrict__ s, const float* __restrict__ signs,
                                                             float* __restrict__ of, __half* __restrict__ oh, int64_t ldo,
                                                             int vocab, int K) {
    __shared__ __align__(16) float sh[1024];
    const int tid = threadIdx.x, row = blockIdx.x;
    const uint32_t t = tokens[row];
    const bool live = t < (uint32_t)vocab;
    const uint32_t* wr = w + (size_t)(live ? t : 0) * (K / 16);
    const __half* sr = s + (size_t)(live ? t : 0) * (K / 128);
    for (int b0 = 0; b0 < K; b0 += 1024) {
        float e[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = b0 + 4 * tid + j;
            const float q = (float)((wr[k / 16] >> (2 * (k % 16))) & 3u) - 1.0f;
            e[j] = live ? q * __half2float(sr[k / 128]) : 0.f;
        }
        fwht1024(e, sh, tid);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int i = 256 * j + tid;
            const float v = e[j] * (1.0f / 32.0f) * signs[b0 + i];
            if (of != nullptr) of[(size_t)row * ldo + b0 + i] = v;
            if (oh != nullptr) oh[(size_t)row * ldo + b0 + i] = __float2half_rn(v);
        }
    }
}

// Decode GEMV: Y[m, n] (+)= sum_k x[m, k] * (q[n, k] - 1) * s[n, k / 128] for up to 16 rows of (already rotated) fp16
// activations, on m16n8k16 fp16 tensor-core MMAs: the weights -1, 0, +1 are exact in fp16, so every product is exact, and
// the scale multiplies the fp32 sum of a group of 128.
//
// A block is 32 output features (16 where that leaves SMs idle), its eight warps take the groups of 128 inputs round robin, and their sums meet in shared
// memory in warp order. Lane (g, t) of a warp holds rows g, g + 8, ... and inputs 32 t .. 32 t + 31 of the group: eight
// bytes of codes per row, 64 bytes of each activation row. The order of the inputs inside an MMA is free as long as both
// operands agree: inputs k and k + 4 make a pair, because their codes are one byte apart, so that one shift and one mask
// turn them into the selector of the byte permutation that looks both weights up.
//
// Bound: latency, and with several rows the L1's look-ups, a line each: an activation row's pieces are 16 bytes every 64, so the rows
// of a group are 64 lines, the codes of 16 features 16, their scales (two bytes a row) 16. Hence 32 features per fragment of
// activations from one and a half such blocks per SM on, and the scales of a block, one contiguous range, by way of shared memory.
// Rotation included, us, with 16 features and scales from global memory -> now: 9216 x 5120, 1 / 5 / 16 rows 13.2 / 14.6 / 21.2 -> 10.4 /
// 11.7 / 16.5; 5120 x 9216 (16 features) 16.3 / 17.3 / 24.8 -> 14.8 / 15.6 / 24.7; 30720 x 4096 29.0 / 31.1 / 56.5 -> 27.2 / 28.4 / 38.7.
// Prefetching the activations instead gained nothing; with 32 features 5120 x 9216 takes 20.9 (160 blocks on 148 SMs).
constexpr int kTernWarps = 8;
struct TernParams {
    const __half* x;
    int64_t ldx;
    const uint32_t* w;
    const __half* s;
    void* y;
    int32_t y_dtype;
    int64_t ldy;
    int32_t M, N, K, accumulate;
    int32_t staged;  // the scales fit shared memory
};

template <int MH, int RB>  // sets of eight activation rows, blocks of 16 features
__global__ void __launch_bounds__(kTernWarps * 32, 4 / (MH * RB) > 2 ? 3 : 2) tern_qmv_kernel(const TernParams p) {
    __shared__ float red[kTernWarps][MH][16 * RB][8];
    extern __shared__ uint16_t ssc[];  // [feature of the block][group]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    pdl_launch_dependents();
    const int G = p.K / 128, n0 = blockIdx.x * 16 * RB, live_n = min(16 * RB, p.N - n0);  // (a multiple of 16)
    const unsigned char* w0 = reinterpret_cast<const unsigned char*>(p.w) + (size_t)(n0 + g) * (p.K / 4) + t * 8;
    const uint16_t* s0 = reinterpret_cast<const uint16_t*>(p.s) + (size_t)n0 * G;
    constexpr int PF = MH * RB > 2 ? 2 : 4;  // groups of codes on their way ahead of the one being used
    uint2 q[PF][RB][2];
    auto fetch = [&](int i, int grp) {  // (no condition around the loads: groups and features past the end read others again)
        grp = min(grp, G - 1);
#pragma unroll
        for (int b = 0; b < RB; b++)
#pragma unroll
            for (int r = 0; r < 2; r++)
                q[i][b][r] = *reinterpret_cast<const uint2*>(w0 + (size_t)((16 * b < live_n ? 16 * b : 0) + 8 * r) * (p.K / 4) + grp * 32);
    };
#pragma unroll
    for (int i = 0; i < PF; i++) fetch(i, warp + i * kTernWarps);
    if (p.staged) {
        for (int i = tid; i < live_n * G; i += kTernWarps * 32) ssc[i] = (uint16_t)ldg_nc_u16(s0 + i);
        __syncthreads();
    }
    pdl_wait();  // the activations are the rotation's output
    float acc[RB][MH][4];
#pragma unroll
    for (int b = 0; b < RB; b++)
#pragma unroll
        for (int h = 0; h < MH; h++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[b][h][j] = 0.f;
    for (int g0 = warp; g0 < G; g0 += PF * kTernWarps) {
#pragma unroll
        for (int i = 0; i < PF; i++) {
            const int grp = g0 + i * kTernWarps;
            if (grp >= G) break;
            uint4 xv[MH][4];  // inputs 8 j .. 8 j + 7 of the lane's 32
#pragma unroll
            for (int h = 0; h < MH; h++) {
                const bool live = 8 * h + g < p.M;
                const uint4* xp = reinterpret_cast<const uint4*>(p.x + (size_t)(live ? 8 * h + g : 0) * p.ldx + grp * 128 + t * 32);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    xv[h][j] = xp[j];
                    if (!live) xv[h][j] = make_uint4(0, 0, 0, 0);
                }
            }
            float d[RB][MH][4], f[RB][2];
            uint32_t words[RB][2][2];
#pragma unroll
            for (int b = 0; b < RB; b++) {
#pragma unroll
                for (int h = 0; h < MH; h++)
#pragma unroll
                    for (int j = 0; j < 4; j++) d[b][h][j] = 0.f;
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    words[b][r][0] = q[i][b][r].x; words[b][r][1] = q[i][b][r].y;
                    const int o = ((16 * b < live_n ? 16 * b : 0) + 8 * r + g) * G + grp;
                    f[b][r] = __half2float(__ushort_as_half(p.staged ? ssc[o] : (unsigned short)ldg_nc_u16(s0 + o)));
                }
            }
            fetch(i, grp + PF * kTernWarps);
#pragma unroll
            for (int j = 0; j < 4; j++) {  // eight inputs: two MMAs
                uint32_t x04[MH], x15[MH], x26[MH], x37[MH];
#pragma unroll
                for (int h = 0; h < MH; h++) {
                    const uint4 v = xv[h][j];
                    x04[h] = __byte_perm(v.x, v.z, 0x5410); x15[h] = __byte_perm(v.x, v.z, 0x7632);
                    x26[h] = __byte_perm(v.y, v.w, 0x5410); x37[h] = __byte_perm(v.y, v.w, 0x7632);
                }
#pragma unroll
                for (int b = 0; b < RB; b++) {
                    uint32_t a[2][4];
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        const uint32_t c8 = j & 1 ? words[b][r][j >> 1] >> 16 : words[b][r][j >> 1];  // eight codes in the low 16 bits
#pragma unroll
                        for (int pr = 0; pr < 4; pr++) {
                            // codes pr and pr + 4 to bits 4-5 and 12-13: selectors of the high bytes of -1, 0, 1, 2 as fp16
                            const uint32_t sel = ((pr < 2 ? c8 << (4 - 2 * pr) : c8 >> (2 * pr - 4)) & 0x3030u) | 0x0404u;
                            a[r][pr] = __byte_perm(0x403C00BCu, 0u, sel);
                        }
                    }
#pragma unroll
                    for (int h = 0; h < MH; h++) {
                        mma16816(d[b][h], a[0][0], a[1][0], a[0][1], a[1][1], x04[h], x15[h]);
                        mma16816(d[b][h], a[0][2], a[1][2], a[0][3], a[1][3], x26[h], x37[h]);
                    }
                }
            }
#pragma unroll
            for (int b = 0; b < RB; b++)
#pragma unroll
                for (int h = 0; h < MH; h++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[b][h][j] = fmaf(f[b][j >> 1], d[b][h][j], acc[b][h][j]);
        }
    }
#pragma unroll
    for (int b = 0; b < RB; b++)
#pragma unroll
        for (int h = 0; h < MH; h++)
#pragma unroll
            for (int j = 0; j < 4; j++) red[warp][h][16 * b + g + 8 * (j >> 1)][2 * t + (j & 1)] = acc[b][h][j];
    __syncthreads();
    for (int u = tid; u < 16 * RB * 8 * MH; u += kTernWarps * 32) {
        const int nl = u % (16 * RB), m8 = u / (16 * RB) % 8, h = u / (16 * RB * 8), m = 8 * h + m8;
        if (m >= p.M || nl >= live_n) continue;
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < kTernWarps; k++) v += red[k][h][nl][m8];
        const size_t o = (size_t)m * p.ldy + n0 + nl;
        if (p.y_dtype == kF32) {
            float* yp = reinterpret_cast<float*>(p.y) + o;
            *yp = p.accumulate ? *yp + v : v;
        } else if (p.y_dtype == kF16) {
            __half* yp = reinterpret_cast<__half*>(p.y) + o;
            *yp = __float2half_rn(p.accumulate ? __half2float(*yp) + v : v);
        } else {
            uint16_t* yp = reinterpret_cast<uint16_t*>(p.y) + o;
            *yp = (uint16_t)f32_to_bf16_bits(p.accumulate ? bf16_bits_to_f32(*yp) + v : v);
        }
    }
}

}  // namespace

// The GEMV of the ternary format (called by iq_qmv for bits = 2, group = 128). x must be fp16 (the rotation's output).
int32_t launch_tern_qmv(iq_ctx* ctx, cudaStream_t st, const void* x, int32_t x_dtype, int64_t ldx, const iq_qlinear* m, void* y,
                        int32_t y_dtype, int64_t ldy, int32_t rows, int32_t n, int32_t accumulate) {
    if (x_dtype != kF16)
        return fail(ctx, kErrInvalidArg, "qmv: ternary weights take fp16 activations (the output of iq_had_rows)");
    if (m->k % 128 != 0) return fail(ctx, kErrInvalidArg, "qmv: ternary k = %d must be a multiple of 128", m->k);
    if ((reinterpret_cast<uintptr_t>(m->w) & 15) != 0) return fail(ctx, kErrInvalidArg, "qmv: ternary codes must be 16-byte aligned");
    TernParams p;
    p.x = static_cast<const __half*>(x); p.ldx = ldx;
    p.w = static_cast<const uint32_t*>(m->w); p.s = static_cast<const __half*>(m->scales);
    p.y = y; p.y_dtype = y_dtype; p.ldy = ldy;
    p.M = rows; p.N = n; p.K = m->k; p.accumulate = accumulate;
    const int rb = n / 32 * 2 >= 3 * ctx->sms ? 2 : 1;
    const size_t scales = (size_t)16 * rb * (m->k / 128) * 2;
    p.staged = scales <= 24 * 1024;  // (inputs up to 49,152; beyond, the scales come from global memory)
    auto kernel = rb == 2 ? (rows > 8 ? tern_qmv_kernel<2, 2> : tern_qmv_kernel<1, 2>) : (rows > 8 ? tern_qmv_kernel<2, 1> : tern_qmv_kernel<1, 1>);
    return check_cuda(ctx, launch_dependent(kernel, dim3((unsigned)((n / 16 + rb - 1) / rb)), kTernWarps * 32,
                                            p.staged ? scales : 0, st, p), "tern_qmv launch");
}

}  // namespace iq

using namespace iq;

extern "C" int32_t iq_had_rows(iq_ctx* ctx, void* stream, const void* x, int32_t x_dtype, int64_t ldx, const float* signs,
                               void* y_f16, int64_t ldy, int32_t rows, int32_t k) {
    if (ctx == nullptr) return kErrInvalidArg;
    if (x == nullptr || signs == nullptr || y_f16 == nullptr || rows < 1 || k < 1024 || k % 1024 != 0 || ldx < k || ldy < k ||
        ldx % 8 != 0 || x_dtype < 0 || x_dtype > 2 || (reinterpret_cast<uintptr_t>(x) & 15) != 0)
        return fail(ctx, kErrInvalidArg, "had_rows: rows = %d, k = %d (a multiple of 1024), ldx / ldy >= k, x 16-byte aligned",
                    rows, k);
    return check_cuda(ctx, launch_dependent(had_rows_kernel, dim3(k / 1024, rows), 256, 0, reinterpret_cast<cudaStream_t>(stream), x, x_dtype, ldx,
                                            signs, static_cast<__half*>(y_f16), ldy), "had_rows launch");
}

extern "C" int32_t iq_embed_rows_ternary(iq_ctx* ctx, void* stream, const iq_qlinear* table, const float* signs,
                                         const uint32_t* tokens, int32_t rows, float* out_f32, void* out_f16, int64_t ldo) {
    if (ctx == nullptr) return kErrInvalidArg;
    if (table == nullptr || table->w == nullptr || table->scales == nullptr || signs == nullptr || tokens == nullptr ||
        (out_f32 == nullptr && out_f16 == nullptr))
        return fail(ctx, kErrInvalidArg, "embed_rows_ternary: null pointer");
    if (table->bits != 2 || table->group != 128 || table->mode != IQ_MODE_AFFINE)
        return fail(ctx, kErrUnsupported, "embed_rows_ternary: the table must be 2-bit, group 128");
    if (rows < 1 || table->n < 1 || table->k < 1024 || table->k % 1024 != 0 || ldo < table->k)
        return fail(ctx, kErrInvalidArg, "embed_rows_ternary: rows = %d, k = %d (a multiple of 1024), ldo = %lld", rows, table->k,
                    (long long)ldo);
    embed_rows_tern_kernel<<<rows, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        tokens, static_cast<const uint32_t*>(table->w), static_cast<const __half*>(table->scales), signs, out_f32,
        static_cast<__half*>(out_f16), ldo, table->n, table->k);
    return check_cuda(ctx, cudaGetLastError(), "embed_rows_ternary launch");
}
