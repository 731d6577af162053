// GEMM of operands that need no conversion on the 5th-generation tensor cores (tcgen05 + tensor memory):
//   bf16 x bf16 -> fp32   the router's approximate logits (the refinement follows in route_topk_kernel)
//   int8 x int8 -> s32    the rotated W8A8 prefill GEMM, a scale per row on both sides
//
//   D[128 weight rows, BN tokens] += W[128, 128 bytes] * X[BN, 128 bytes]^T      per K step (64 bf16 or 128 int8 inputs)
//
// Warp roles inside one persistent CTA (192 threads): warp 0 TMA producer (both tiles, 128-byte swizzle, the layout the MMA
// reads), warp 1 allocates tensor memory and issues tcgen05.mma (one lane), warps 2-5 epilogue. Two accumulators in
// tensor memory let the epilogue of one tile overlap the main loop of the next. Every wait is bounded: on a timeout the
// kernel writes a status word, all roles drain and tensor memory is released. The quantized formats have a kernel of
// their own (qmm_ta.cuh).
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "ptx.cuh"

namespace iq {

constexpr int kQmmThreads = 192;
constexpr int kWRows = 128;          // weight rows per tile (MMA M)

struct QmmParams {
    const void* s;           // int8: scale of each token row, fp32
    const void* b;           // int8: scale of each weight row, fp32
    int32_t N, K, M;         // weight rows, inputs, token rows
    void* y;
    int32_t y_dtype;
    int64_t ldy;
    int32_t accumulate;
    float limit;             // int8: factor of the result
    int32_t* status;         // device status word (0 = ok)
};

// Shared-memory matrix descriptor of a K-major tile with 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes
// apart (stride byte offset), descriptor version 1, layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t make_sw128_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;              // leading byte offset (unused with a swizzled K-major tile)
    d |= (uint64_t)(1024 >> 4) << 32;    // stride byte offset
    d |= (uint64_t)1 << 46;              // descriptor version (sm_100)
    d |= (uint64_t)2 << 61;              // SWIZZLE_128B
    return d;
}
// Instruction descriptor, kind::f16: D = f32, A and B both f16 or both bf16, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t make_idesc(int n, bool bf16) {
    return (1u << 4) | (bf16 ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kWRows >> 4) << 24);
}
// kind::i8: D = s32, A = B = signed 8-bit, both K-major (32 inputs per MMA), M = 128, N = n.
__device__ __forceinline__ uint32_t make_idesc_i8(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kWRows >> 4) << 24);
}

template <int FMT, int BN>
struct QmmSmem {
    static constexpr bool I8 = FMT == kFmtInt8Plain;
    static constexpr int BKE = I8 ? 128 : 64;                             // inputs per K step (128 bytes of a row either way)
    static constexpr int X_BYTES = BN * 128;
    static constexpr int STAGE_BYTES = X_BYTES + kWRows * 128;
    static constexpr int kMaxDyn = 232448 - 1280;                         // opt-in limit minus alignment + barriers
    static constexpr int STAGES = kMaxDyn / STAGE_BYTES > 6 ? 6 : kMaxDyn / STAGE_BYTES;
    static constexpr int TOTAL = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
};

template <int FMT, int BN>
__global__ void __launch_bounds__(kQmmThreads, 1)
    qmm_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const QmmParams p) {
    using S = QmmSmem<FMT, BN>;
    constexpr int STAGES = S::STAGES;
    extern __shared__ unsigned char smem_raw[];
    // 1024-byte alignment for the swizzled tiles
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * S::STAGE_BYTES);
    // barrier slots: full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2]
    const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * STAGES;
    const uint32_t bar_tfull = bar_empty + 8 * STAGES, bar_tempty = bar_tfull + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(bar_tfull + 8 * a, 1);
            mbar_init(bar_tempty + 8 * a, 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int m_tiles = (p.M + BN - 1) / BN;
    const int total_work = m_tiles * ((p.N + kWRows - 1) / kWRows);
    const int ksteps = p.K / S::BKE;

    if (warp == 0) {
        // ================= TMA producer =================
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int wi = blockIdx.x; wi < total_work && ok; wi += gridDim.x) {
                const int row0 = (wi % m_tiles) * BN, n0 = (wi / m_tiles) * kWRows;
                for (int ks = 0; ks < ksteps; ks++) {
                    if (!(ok = mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag))) break;
                    const uint32_t st = smem_u32(smem + s * S::STAGE_BYTES);
                    mbar_arrive_expect_tx(bar_full + 8 * s, S::STAGE_BYTES);
                    tma_load_2d(st, &map_x, bar_full + 8 * s, ks * S::BKE, row0);
                    tma_load_2d(st + S::X_BYTES, &map_w, bar_full + 8 * s, ks * S::BKE, n0);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        if (elect_one()) {
            int s = 0, a = 0;
            uint32_t ph = 0, tph = 0;
            bool ok = true;
            for (int wi = blockIdx.x; wi < total_work && ok; wi += gridDim.x) {
                const int rows = min(BN, p.M - (wi % m_tiles) * BN);
                const int nmma = (rows + 15) & ~15;
                const uint32_t idesc = S::I8 ? make_idesc_i8(nmma) : make_idesc(nmma, true);
                if (!(ok = mbar_wait(bar_tempty + 8 * a, tph ^ 1, abort_flag))) break;
                tc_fence_after();
                const uint32_t tacc = tmem_base + a * BN;
                for (int ks = 0; ks < ksteps; ks++) {
                    if (!(ok = mbar_wait(bar_full + 8 * s, ph, abort_flag))) break;
                    tc_fence_after();
                    const uint32_t st = smem_u32(smem + s * S::STAGE_BYTES);
                    const uint64_t bdesc = make_sw128_desc(st), adesc = make_sw128_desc(st + S::X_BYTES);
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {  // four MMAs of 32 bytes of K each
                        if (S::I8) umma_i8(tacc, adesc + 2 * kk, bdesc + 2 * kk, idesc, (ks | kk) ? 1u : 0u);
                        else umma_f16(tacc, adesc + 2 * kk, bdesc + 2 * kk, idesc, (ks | kk) ? 1u : 0u);
                    }
                    umma_commit(bar_empty + 8 * s);  // the stage is free once these MMAs have read it
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                if (ok) umma_commit(bar_tfull + 8 * a);
                a ^= 1;
                if (a == 0) tph ^= 1;
            }
        }
    } else {
        // ================= epilogue =================
        const int q = warp & 3;  // tensor-memory lane quadrant this warp may read
        int a = 0;
        uint32_t tph = 0;
        for (int wi = blockIdx.x; wi < total_work; wi += gridDim.x) {
            const int row0 = (wi % m_tiles) * BN, rows = min(BN, p.M - row0), n = (wi / m_tiles) * kWRows + 32 * q + lane;
            if (!__all_sync(0xffffffffu, mbar_wait(bar_tfull + 8 * a, tph, abort_flag))) break;
            tc_fence_after();
            const bool n_ok = n < p.N;  // weight row = output feature of this thread
            const float sw = S::I8 && n_ok ? reinterpret_cast<const float*>(p.b)[n] : 0.f;
            const uint32_t tbase = tmem_base + ((uint32_t)(32 * q) << 16) + a * BN;
            for (int c0 = 0; c0 < rows; c0 += 32) {
                uint32_t r[32];
                tmem_ld32(tbase + c0, r);
                tmem_ld_wait();
                const int live = n_ok ? rows - c0 : 0;  // columns j < live are stored
                float v[32];
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    // int8: ((sum * sx[token]) * sw[feature]) / n, in the order of the CPU emulation
                    v[j] = S::I8 ? ((float)(int)r[j] * (j < live ? reinterpret_cast<const float*>(p.s)[row0 + c0 + j] : 0.f)) * sw * p.limit
                                 : __uint_as_float(r[j]);
                }
                const size_t o0 = (size_t)(row0 + c0) * p.ldy + n;
                if (p.y_dtype == kF32) {
                    float* yp = reinterpret_cast<float*>(p.y) + o0;
                    if (p.accumulate) {  // all loads before the first store
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (j < live) v[j] = yp[(size_t)j * p.ldy] + v[j];
                    }
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (j < live) yp[(size_t)j * p.ldy] = v[j];
                } else if (p.y_dtype == kF16) {
                    __half* yp = reinterpret_cast<__half*>(p.y) + o0;
                    if (p.accumulate) {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (j < live) v[j] = __half2float(yp[(size_t)j * p.ldy]) + v[j];
                    }
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (j < live) yp[(size_t)j * p.ldy] = __float2half_rn(v[j]);
                } else {
                    uint16_t* yp = reinterpret_cast<uint16_t*>(p.y) + o0;
                    if (p.accumulate) {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (j < live) v[j] = bf16_bits_to_f32(yp[(size_t)j * p.ldy]) + v[j];
                    }
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (j < live) yp[(size_t)j * p.ldy] = (uint16_t)f32_to_bf16_bits(v[j]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_tempty + 8 * a);
            a ^= 1;
            if (a == 0) tph ^= 1;
        }
    }
    __syncwarp();
    // ---- teardown ------------------------------------------------------------------------------------------------
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, kErrTimeout);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

// fp32 / bf16 activations -> fp16, row-major [rows, k] contiguous (the MMA's B operand type)
__global__ void __launch_bounds__(256) convert_x_f16_kernel(const void* __restrict__ x, int32_t x_dtype, int64_t ldx, __half* __restrict__ out,
                                                           int rows, int k) {
    pdl_wait();
    pdl_launch_dependents();  // (after the wait: what runs before this kernel has ended when the GEMM starts on its weights)
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (i >= (size_t)rows * k) return;
    const size_t r = i / k, c = i % k;
    float v[8];
    load_x8(x, x_dtype, r * ldx + c, v);
    uint4 o;
    o.x = pack_half2(v[0], v[1]); o.y = pack_half2(v[2], v[3]); o.z = pack_half2(v[4], v[5]); o.w = pack_half2(v[6], v[7]);
    *reinterpret_cast<uint4*>(out + i) = o;
}

}  // namespace iq
