// Streaming MXFP4 GEMV (plain, and gate + up + activation): the weight stream goes HBM -> shared memory through a ring of bulk (TMA) copies, so the
// bytes in flight per SM are set by the ring (3-6 stages of 24-64 KB), not by registers. One persistent CTA per SM:
//   warp 8       producer: per stage one block of R consecutive weight rows over the whole K (codes and scales
//                are each one contiguous range, so a block is two bulk copies and more per matrix)
//   warps 0..7   consumers: RGS row groups of 16 rows x WK K-slices; dequantise from shared memory and multiply on
//                m16n8k16 fragments exactly as gqmv_kernel does (same fragment order, same fixed-order K reduction,
//                hence the same row-invariant bits)
// A CTA takes a contiguous range of the blocks. With programmatic dependent launch the producer starts streaming weights while
// the previous kernel of the stream is still draining; activations are only read after the dependency wait.
//
// Same operators as gqmv.cuh (the reference's vnax_qmv*, Shaders/verify_nax.metal:105-257); this is the path taken when a block of 16+ rows over the whole K fits a stage.
#pragma once

#include "common.cuh"
#include "gqmv.cuh"
#include <type_traits>

#include "ptx.cuh"

namespace iq {

constexpr int kQsConsumers = 256;
constexpr int kQsThreads = 288;
constexpr int kQsPiece = 8192;  // bytes per bulk copy

struct QsParams {
    const unsigned char* w[2];
    const unsigned char* s[2];
    int32_t N, K;
    const void* x;
    int32_t x_dtype;
    int64_t ldx;
    int32_t M;
    void* y;
    int32_t y_dtype;
    int64_t ldy;
    int32_t accumulate;
    float limit;
    int32_t act;
    // blocking
    int32_t R;          // weight rows per block (16 * rgs)
    int32_t NB;         // blocks of the matrix
    int32_t rgs, wk;    // row groups x K slices = 8 consumer warps
    int32_t row_bytes;  // code bytes per weight row
    int32_t srow_bytes; // scale bytes per weight row
    int32_t mat_bytes;  // bytes of one matrix inside a stage (codes + scales of R rows)
    int32_t stage_bytes;
    int32_t nstages;
    // shared-memory layout
    int32_t xs_bytes, red_bytes;
    int32_t* status;
};

__device__ __forceinline__ void consumer_barrier() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ bool consumer_barrier_or(bool pred) {
    uint32_t r;
    asm volatile(
        "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.or.pred q, 1, 256, p;\nselp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"((uint32_t)pred)
        : "memory");
    return r != 0;
}

template <int MH, int MODE>
__global__ void __launch_bounds__(kQsThreads, (MH == 1 && MODE != kModeGateUp) ? 2 : 1) qmv_stream_kernel(const QsParams p) {
    constexpr int FMT = kFmtMxfp4;
    using F = FmtTraits<FMT>;
    constexpr int NW = MODE == kModeGateUp ? 2 : 1;
    extern __shared__ __align__(128) unsigned char smem[];
    uint4* xs = reinterpret_cast<uint4*>(smem);
    float* red = reinterpret_cast<float*>(smem + p.xs_bytes);
    unsigned char* stages = smem + p.xs_bytes + p.red_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(stages + (size_t)p.nstages * p.stage_bytes);
    const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * p.nstages;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * p.nstages);
    uint4* zero16 = reinterpret_cast<uint4*>(bars + 2 * p.nstages + 2);  // 16 bytes of zeros for idle fragment lanes

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < p.nstages; s++) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 8);
        }
        *abort_flag = 0;
        *zero16 = make_uint4(0, 0, 0, 0);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    __syncthreads();
    pdl_launch_dependents();

    const int codes_bytes = p.R * p.row_bytes;
    const int nch = p.row_bytes / 16;              // 16-byte chunks per weight row
    const int nsteps = (nch + 3) / 4;

    const int total = p.NB;
    const int per = (total + gridDim.x - 1) / gridDim.x;
    const int lo = min(total, (int)blockIdx.x * per), hi = min(total, lo + per);

    if (warp == 8) {
        // ================= producer =================
        bool ok = true;
        for (int item = lo, it = 0; item < hi && ok; item++, it++) {
            const int s = it % p.nstages;
            const uint32_t ph = (it / p.nstages) & 1;
            const int r0 = item * p.R;
            const int rows = min(p.R, p.N - r0);
            ok = mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const uint32_t cb = rows * p.row_bytes, sb = rows * p.srow_bytes;
            if (lane == 0) mbar_arrive_expect_tx(bar_full + 8 * s, NW * (cb + sb));
            __syncwarp();
            const uint32_t st = smem_u32(stages + (size_t)s * p.stage_bytes);
            const int npc = (cb + kQsPiece - 1) / kQsPiece;  // code pieces per matrix
            const int per_mat = npc + 1;
            for (int pc = lane; pc < NW * per_mat; pc += 32) {
                const int i = pc / per_mat, j = pc % per_mat;
                const uint32_t dst = st + i * p.mat_bytes;
                if (j < npc) {
                    const uint32_t off = j * kQsPiece;
                    bulk_g2s(dst + off, p.w[i] + (int64_t)r0 * p.row_bytes + off,
                             min((uint32_t)kQsPiece, cb - off), bar_full + 8 * s);
                } else {
                    bulk_g2s(dst + codes_bytes, p.s[i] + (int64_t)r0 * p.srow_bytes, sb, bar_full + 8 * s);
                }
            }
        }
        if (!ok) {  // give copies in flight time to land before the CTA's shared memory is released
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {}
        }
    } else {
        // ================= consumers =================
        const int g = lane >> 2, t = lane & 3;
        const int rg = warp / p.wk, wk = warp % p.wk;
        const int spw = (nsteps + p.wk - 1) / p.wk;
        const int jb = wk * spw, je = min(nsteps, jb + spw);
        pdl_wait();  // activations (and y) belong to the previous kernel until here
        const int M = p.M;
        {
            // ---- stage the activations (fp16, fragment order) ----------------------------------------------------------
            const int units_per_row = p.K / 8;
            const int total_units = M * units_per_row;
            for (int uidx = tid; uidx < total_units; uidx += kQsConsumers) {
                const int m = uidx / units_per_row, ku = uidx % units_per_row;
                float v[8];
                load_x8(p.x, p.x_dtype, (size_t)m * p.ldx + ku * 8, v);
                uint4 o;
                o.x = pack_half2(v[0], v[1]); o.y = pack_half2(v[2], v[3]);
                o.z = pack_half2(v[4], v[5]); o.w = pack_half2(v[6], v[7]);
                const int kl = ku * 8, cl = kl / F::CK, q = (kl % F::CK) / 8;
                xs[(((cl >> 2) * F::QU + q) * M + m) * 4 + (cl & 3)] = o;
            }
            consumer_barrier();
        }
        for (int item = lo, it = 0; item < hi; item++, it++) {
            const int s = it % p.nstages;
            const uint32_t ph = (it / p.nstages) & 1;
            const int r0 = item * p.R;
            const int rows = min(p.R, p.N - r0);
            const bool rows_ok = rg * 16 < rows;
            const unsigned char* st = stages + (size_t)s * p.stage_bytes;

            // two independent accumulation chains per output (even / odd MMAs), added at the end in a fixed order
            float acc2[NW][MH][2][4];
#pragma unroll
            for (int i = 0; i < NW; i++)
#pragma unroll
                for (int h = 0; h < MH; h++)
#pragma unroll
                    for (int c2 = 0; c2 < 2; c2++)
#pragma unroll
                        for (int e = 0; e < 4; e++) acc2[i][h][c2][e] = 0.f;
            float acc[NW][MH][4];

            const bool ok = mbar_wait(bar_full + 8 * s, ph, abort_flag);
            const int lr = rg * 16 + g;  // this lane's first row inside the block
            if (ok && rows_ok) {
                const uint32_t st32 = smem_u32(st);
                // per-lane shared-memory addresses of the codes and scales of rows lr and lr + 8
                uint32_t ca[NW][2], sa[NW][2];
#pragma unroll
                for (int i = 0; i < NW; i++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        ca[i][h] = st32 + i * p.mat_bytes + (lr + 8 * h) * p.row_bytes + t * 16;
                        sa[i][h] = st32 + i * p.mat_bytes + codes_bytes + (lr + 8 * h) * p.srow_bytes + t;
                    }
                // activation fragments: live lanes walk the staged x, the others keep reading one block of zeros
                uint32_t xa[MH], xstep[MH];
#pragma unroll
                for (int h = 0; h < MH; h++) {
                    const int m = g + 8 * h;
                    xa[h] = m < M ? smem_u32(xs) + (m * 4 + t) * 16 : smem_u32(zero16);
                    xstep[h] = m < M ? M * 64 : 0;
                }
                auto step = [&](int j, auto full_tag) {
                    constexpr bool FULL = decltype(full_tag)::value;
                    const bool c_ok = FULL || 4 * j + t < nch;
                    uint4 cv[NW][2];
                    DqConst dq[NW][2];
#pragma unroll
                    for (int i = 0; i < NW; i++)
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            if (c_ok) {
                                cv[i][h] = lds128(ca[i][h] + j * 64);
                                dq[i][h] = make_dq<FMT>(lds_u8(sa[i][h] + j * 4));  // (four chunks per step, a scale each)
                            } else {
                                cv[i][h] = make_uint4(0, 0, 0, 0);
                                dq[i][h] = make_dq<FMT>(127u);
                            }
                        }
#pragma unroll
                    for (int q = 0; q < F::QU; q++) {
                        uint4 xf[MH];
#pragma unroll
                        for (int h = 0; h < MH; h++)
                            xf[h] = c_ok ? lds128(xa[h] + (j * F::QU + q) * xstep[h]) : make_uint4(0, 0, 0, 0);
#pragma unroll
                        for (int i = 0; i < NW; i++) {
                            uint32_t pa[4], pb[4];
                            dequant_word<FMT>(word_of(cv[i][0], q), dq[i][0], pa);
                            dequant_word<FMT>(word_of(cv[i][1], q), dq[i][1], pb);
#pragma unroll
                            for (int h = 0; h < MH; h++) {
                                mma16816(acc2[i][h][0], pa[0], pb[0], pa[1], pb[1], xf[h].x, xf[h].y);
                                mma16816(acc2[i][h][1], pa[2], pb[2], pa[3], pb[3], xf[h].z, xf[h].w);
                            }
                        }
                    }
                };
                const int jfull = min(je, nch / 4);  // steps whose four chunks all exist
#pragma unroll 2
                for (int j = jb; j < jfull; j++) step(j, std::true_type{});
                for (int j = max(jb, jfull); j < je; j++) step(j, std::false_type{});
            }
#pragma unroll
            for (int i = 0; i < NW; i++)
#pragma unroll
                for (int h = 0; h < MH; h++)
#pragma unroll
                    for (int e = 0; e < 4; e++) acc[i][h][e] = acc2[i][h][0][e] + acc2[i][h][1][e];
            // the stage is free as soon as every warp has read its part
            __syncwarp();
            if (lane == 0 && ok) mbar_arrive(bar_empty + 8 * s);

            // ---- fixed-order reduction over the K slices, then the epilogue in the slice-0 warps ---------------------
            float* mine = red + (size_t)((it & 1) * 8 + warp) * (NW * MH * 4 * 32);
            if (p.wk > 1) {
#pragma unroll
                for (int i = 0; i < NW; i++)
#pragma unroll
                    for (int h = 0; h < MH; h++)
#pragma unroll
                        for (int e = 0; e < 4; e++) mine[((i * MH + h) * 4 + e) * 32 + lane] = acc[i][h][e];
            }
            if (consumer_barrier_or(!ok)) break;  // a wait gave up somewhere: everybody leaves together
            if (wk != 0 || !rows_ok) continue;
            if (p.wk > 1) {
#pragma unroll
                for (int i = 0; i < NW; i++)
#pragma unroll
                    for (int h = 0; h < MH; h++)
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            float sum = 0.f;
                            for (int k = 0; k < p.wk; k++)
                                sum += red[(size_t)((it & 1) * 8 + warp + k) * (NW * MH * 4 * 32) + ((i * MH + h) * 4 + e) * 32 + lane];
                            acc[i][h][e] = sum;
                        }
            }
            const int n0 = r0 + rg * 16;
#pragma unroll
            for (int h = 0; h < MH; h++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int n = n0 + g + 8 * (e >> 1);
                    const int m = 2 * t + (e & 1) + 8 * h;
                    if (m >= M) continue;
                    float v = acc[0][h][e];
                    if (MODE == kModeGateUp) {
                        v = glu_rt(p.act, v, acc[NW - 1][h][e], p.limit);
                    }
                    const size_t o = (size_t)m * p.ldy + n;
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
    }
    __syncthreads();
    if (*abort_flag && tid == 0 && p.status != nullptr) atomicExch(p.status, kErrTimeout);
}

}  // namespace iq
