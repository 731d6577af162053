// The MoE block for one token, and for two or three of small experts, in three kernels, where a decode step is a chain of latencies and not
// of bytes (one token of the 128-expert layer reads 21 MB, 3 us, and took 59 us in eight kernels, 26 in three). Beyond 24 million weights of all
// tokens' experts only the first of them runs here, then the decode tiles, which stage the weights (use_experts_small in moe.cu):
//
//   moe_route_small_kernel   router logits, top-k and the permutation in one cluster of eight blocks; also the activations as
//                            block fixed point (the int8 kernels' operand, see qmv_imma.cuh), once per token
//   moe_gateup_small_kernel  h = act(gate x, up x) per (expert tile, 64 features): weights straight from global memory into
//                            registers, and h leaves as fp16 and as the down projection's block fixed point, group by group
//   moe_down_small_kernel    per (token, 16 features) the down projections of all the token's experts side by side in the
//                            block's warps, then their weighted sum: the combine needs no kernel and no round trip
//
// Each starts while its predecessor runs (programmatic dependent launch); the down kernel has its first weights on the way
// before h exists. Affine 4-bit experts, all of them on this GPU. The results are those of the separate kernels: exact
// float64 logits, sums in fixed orders. The activations and h are fixed point of 23 bits (three digits: the columns of an MMA are two
// rows of (high, middle), (low, low), as in qmv_ring.cuh), which keeps bf16 activations and halves of h whole as fp16 kernels do: with 16 bits a
// layer of 2880 x 768 with input channels 100 times the rest was 8.5e-4 off the 64-bit result instead of 4.9e-4. The decode tiles take three digits
// of both for two and three tokens too.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "fixed_rows.cuh"
#include "gqmv.cuh"
#include "moe_aux.cuh"
#include "ptx.cuh"
#include "qmv_imma.cuh"

namespace iq {

constexpr int kSmallTokens = 3;
constexpr int kSmallThreads = 512;
constexpr int kSmallCluster = 8;

struct RouteSmallParams {
    RouteParams r;               // logits_rw, inds, wts, T, E, ld, topk, D and the scoring rule
    RouterIn in;
    uint32_t *counts, *offsets, *row_map, *pos, *ntiles;
    Tile *tiles_a, *tiles_b;
    FixedRows fx;                // the activations as block fixed point, or null
    int32_t wide;                // its form: 23 bits (moe_gateup_small_kernel's), or 16
};
constexpr size_t route_small_smem(int tt, int D, int E) {
    return router_block_smem(tt, D, E / kSmallCluster) + (size_t)tt * E * 4 + 16 * kSmallTokens * 4 + 64 * 4 + (size_t)E * 4;
}

// WFMT: 0 bf16 router, 1 8-bit affine. TT: tokens rounded up to 1, 2, 4. VPL: experts per lane of the selection.
// A block of the cluster takes E / 8 experts (router_block: the other router kernels' bits). The logits meet in the
// first block's shared memory, which then selects (a warp per token) and groups.
template <int WFMT, int TT, int VPL>
__global__ void __launch_bounds__(kSmallThreads, 1) __cluster_dims__(kSmallCluster, 1, 1) moe_route_small_kernel(const RouteSmallParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int T = p.r.T, E = p.r.E, D = p.r.D, topk = p.r.topk, epc = E / kSmallCluster;
    double2* xs = reinterpret_cast<double2*>(smem);
    double* part = reinterpret_cast<double*>(smem + (size_t)TT * D * 8);
    float* lg = reinterpret_cast<float*>(part + (size_t)router_slices(epc) * epc * TT);  // [TT][E], the first block's
    uint32_t* sinds = reinterpret_cast<uint32_t*>(lg + (size_t)TT * E);                  // [16 * kSmallTokens]
    uint32_t* wsum = sinds + 16 * kSmallTokens;                                          // [2][32]
    uint32_t* soff = wsum + 64;                                                          // [E] exclusive offsets
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x;
    pdl_launch_dependents();
    cluster_sync_all();  // every block of the cluster runs: the first one's shared memory may be written
    router_block<WFMT, TT>(p.in, xs, part, 0, T, rank * epc, epc, [&](int e, int t, float f) {
        st_dsmem_u32(reinterpret_cast<uint32_t*>(lg + (size_t)t * E + e), 0, __float_as_uint(f));
        p.r.logits_rw[(size_t)t * p.r.ld + e] = f;
    });
    if (rank == kSmallCluster - 1)
        for (int i = tid; i < T * (p.r.ld - E); i += kSmallThreads) p.r.logits_rw[(size_t)(i / (p.r.ld - E)) * p.r.ld + E + i % (p.r.ld - E)] = 0.f;
    cluster_sync_all();
    // the other blocks turn the activations into fixed point
    if (rank != 0) {
        if (p.fx.digits == nullptr) return;
        for (int t = rank - 1; t < T; t += kSmallCluster - 1) {
            if (p.wide) fixed_point_row<true>(p.in.x, p.in.x_dtype, (size_t)t * p.in.ldx, D, p.fx, t, tid, kSmallThreads);
            else fixed_point_row<false>(p.in.x, p.in.x_dtype, (size_t)t * p.in.ldx, D, p.fx, t, tid, kSmallThreads);
        }
        return;
    }
    if (warp < T) {
        const int t = warp;
        float v[VPL], pv[VPL];
        uint32_t taken = 0;
#pragma unroll
        for (int j = 0; j < VPL; j++) {
            const int e = j * 32 + lane;
            float f = e < E ? lg[(size_t)t * E + e] : -INFINITY;
            if (e < E && p.r.logit_bias != nullptr) f += p.r.logit_bias[e];
            pv[j] = 0.f;
            if (p.r.sigmoid) {
                f = (float)(1.0 / (1.0 + exp(-(double)f)));
                pv[j] = f;
                if (e < E && p.r.select_bias != nullptr) f += p.r.select_bias[e];
            }
            if (f != f) f = -INFINITY;
            v[j] = f;
            if (e >= E) taken |= 1u << j;
        }
        const uint32_t mine = route_select<VPL>(v, pv, taken, topk, lane, p.r.sigmoid != 0, p.r.eps, p.r.scale, p.r.pes,
                                                p.r.inds + (size_t)t * topk, p.r.wts + (size_t)t * topk, true);
        if (lane < topk) sinds[t * topk + lane] = mine;
    }
    __syncthreads();
    // ---- the permutation: a thread per expert counts and places, a thread per pair finds its position --------------------
    const int P = T * topk;
    uint32_t c = 0;
    if (tid < E)
        for (int i = 0; i < P; i++) c += sinds[i] == (uint32_t)tid;
    uint32_t off = c, til = c > 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, off, o), b = __shfl_up_sync(0xffffffffu, til, o);
        if (lane >= o) { off += a; til += b; }
    }
    if (lane == 31) { wsum[warp] = off; wsum[32 + warp] = til; }
    __syncthreads();
    for (int k = 0; k < warp; k++) { off += wsum[k]; til += wsum[32 + k]; }
    if (tid < E) {
        soff[tid] = off - c;
        p.counts[tid] = c;
        p.offsets[tid] = off - c;
        if (c > 0) p.tiles_a[til - 1] = p.tiles_b[til - 1] = Tile{(uint32_t)tid, off - c, c, 0};  // (c <= T: one tile)
        if (tid == E - 1) {
            p.offsets[E] = off;
            p.ntiles[0] = p.ntiles[1] = til;
        }
    }
    __syncthreads();
    if (tid < P) {
        const uint32_t e = sinds[tid];
        uint32_t r = soff[e];
        for (int j = 0; j < tid; j++) r += sinds[j] == e;
        p.row_map[r] = (uint32_t)tid;
        p.pos[tid] = r;
    }
}

struct GateUpSmallParams {
    const unsigned char *w[2], *s[2], *b[2];  // stacked gate and up
    int32_t D, I, topk;
    FixedRows x;               // the tokens
    const uint32_t* row_map;
    const Tile* tiles;
    const uint32_t* ntiles;
    const float* ebias[2];     // [E, I] or null
    int32_t act;
    float limit;
    __half* h;                 // [P, I]
    FixedRows fh;              // h as block fixed point
};

// Codes, scales and biases of two neighbouring groups of 64 inputs of weight rows g and g + 8 (a lane's share), straight from
// global memory. Groups past the end read the last one again. even: the pair's scales are one aligned word.
struct SmallBatch {
    uint2 q[2][2];         // [group][row]
    uint32_t s[2], b[2];   // [row]: two bf16
};
__device__ __forceinline__ void small_load(SmallBatch& v, const unsigned char* w, const unsigned char* s, const unsigned char* b, int64_t row,
                                           int G, int g0, bool even, int t) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int64_t r = row + 8 * h;
        const int ga = min(g0, G - 1), gb = min(g0 + 1, G - 1);
        v.q[0][h] = __ldg(reinterpret_cast<const uint2*>(w + (r * G + ga) * 32 + t * 8));
        v.q[1][h] = __ldg(reinterpret_cast<const uint2*>(w + (r * G + gb) * 32 + t * 8));
        const uint16_t* sp = reinterpret_cast<const uint16_t*>(s) + r * G;
        const uint16_t* bp = reinterpret_cast<const uint16_t*>(b) + r * G;
        if (even) {
            v.s[h] = __ldg(reinterpret_cast<const uint32_t*>(sp + ga));
            v.b[h] = __ldg(reinterpret_cast<const uint32_t*>(bp + ga));
        } else {
            v.s[h] = (uint32_t)__ldg(sp + ga) | ((uint32_t)__ldg(sp + gb) << 16);
            v.b[h] = (uint32_t)__ldg(bp + ga) | ((uint32_t)__ldg(bp + gb) << 16);
        }
    }
}
// One group of the batch against one set of two activation rows: xb the lane's digits (column g: digit g % 4 of row g / 4, the last
// digit twice), xs its part's scale and sum: lanes of even t hold the high and middle digits' sums of row t / 2, those of odd t the
// low one's (radix 0: one of the two).
__device__ __forceinline__ float2 small_part(const float2& row, int t) { return t & 1 ? make_float2(row.x * 0.0078125f, 0.f) : row; }
__device__ __forceinline__ void small_mma(float (&acc)[2], const SmallBatch& v, int u, const uint4& xb, const float2& xs, int radix) {
    constexpr uint32_t MSK = 0x0F0F0F0Fu;
    const int z[4] = {0, 0, 0, 0};
    int d[4];
    const uint2 w0 = v.q[u][0], w1 = v.q[u][1];
    imma16832_u8s8(d, w0.x & MSK, w1.x & MSK, (w0.x >> 4) & MSK, (w1.x >> 4) & MSK, xb.x, xb.y, z);
    imma16832_u8s8(d, w0.y & MSK, w1.y & MSK, (w0.y >> 4) & MSK, (w1.y >> 4) & MSK, xb.z, xb.w, d);
    const float v0 = (float)(d[0] * radix + d[1]), v1 = (float)(d[2] * radix + d[3]);
    const float s0 = __uint_as_float(u ? (v.s[0] & 0xFFFF0000u) : (v.s[0] << 16)), s1 = __uint_as_float(u ? (v.s[1] & 0xFFFF0000u) : (v.s[1] << 16));
    const float b0 = __uint_as_float(u ? (v.b[0] & 0xFFFF0000u) : (v.b[0] << 16)), b1 = __uint_as_float(u ? (v.b[1] & 0xFFFF0000u) : (v.b[1] << 16));
    acc[0] = fmaf(v0, s0 * xs.x, acc[0]);
    acc[0] = fmaf(b0, xs.y, acc[0]);
    acc[1] = fmaf(v1, s1 * xs.x, acc[1]);
    acc[1] = fmaf(b1, xs.y, acc[1]);
}

// A block's item: 64 features (gate and up) of one tile of up to three rows, in sets of two; its sixteen warps are four blocks of
// 16 rows x four slices of the inputs.
__global__ void __launch_bounds__(kSmallThreads, 1) moe_gateup_small_kernel(const GateUpSmallParams p) {
    constexpr int RS = 72;  // floats between activation rows of the slices' sums (the lanes of a store in different banks)
    __shared__ float red[4][2][8][RS];  // [slice][matrix][row, part]
    __shared__ float gmax[16], gsum[16];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int rb = warp & 3, ks = warp >> 2;
    const int G = p.D / 64, NB = p.I / 64;
    const int pairs = (G + 1) / 2, p0 = pairs * ks / 4, p1 = pairs * (ks + 1) / 4;  // this slice, in pairs of groups
    const bool even = (G & 1) == 0;
    const int radix = t & 1 ? 0 : 256;
    pdl_wait();
    pdl_launch_dependents();  // (after the wait: what the down kernel reads early is then complete)
    const int total = (int)__ldcg(p.ntiles) * NB;
    for (int it = blockIdx.x; it < total; it += gridDim.x) {
        const uint4 tw = __ldcg(reinterpret_cast<const uint4*>(p.tiles) + it / NB);
        const Tile tile = Tile{tw.x, tw.y, tw.z, tw.w};
        const int n0 = (it % NB) * 64, M = (int)tile.count;
        const int64_t row = (int64_t)tile.expert * p.I + n0 + rb * 16 + g;
        SmallBatch cur[2], nxt[2];
#pragma unroll
        for (int i = 0; i < 2; i++) small_load(cur[i], p.w[i], p.s[i], p.b[i], row, G, 2 * min(p0, pairs - 1), even, t);
        const unsigned char* xd[2];
        const float2* xs[2];
        bool live[2];
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const int m = 2 * c + (g >> 2), mt = 2 * c + (t >> 1);
            live[c] = m < M;
            const uint32_t tok = __ldcg(p.row_map + tile.start + min(m, M - 1)) / (uint32_t)p.topk;
            const uint32_t tks = __ldcg(p.row_map + tile.start + min(mt, M - 1)) / (uint32_t)p.topk;
            xd[c] = p.x.digits + (size_t)tok * G * 192 + min(g & 3, 2) * 64 + t * 16;
            xs[c] = p.x.scale + (size_t)tks * G;
        }
        float acc[2][2][2] = {{{0.f, 0.f}, {0.f, 0.f}}, {{0.f, 0.f}, {0.f, 0.f}}};  // [matrix][set]
        auto slice = [&](auto sets) {  // (their number outside the loop: no branch between the groups' loads)
            auto compute = [&](const SmallBatch (&v)[2], int pr) {
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int grp = 2 * pr + u;
                    if (grp >= G) break;
#pragma unroll
                    for (int c = 0; c < decltype(sets)::value; c++) {
                        uint4 xb = *reinterpret_cast<const uint4*>(xd[c] + grp * 192);
                        if (!live[c]) xb = make_uint4(0, 0, 0, 0);
                        const float2 sv = small_part(xs[c][grp], t);
                        small_mma(acc[0][c], v[0], u, xb, sv, radix);
                        small_mma(acc[1][c], v[1], u, xb, sv, radix);
                    }
                }
            };
            int pr = p0;
            for (; pr + 1 < p1; pr += 2) {
#pragma unroll
                for (int i = 0; i < 2; i++) small_load(nxt[i], p.w[i], p.s[i], p.b[i], row, G, 2 * (pr + 1), even, t);
                compute(cur, pr);
#pragma unroll
                for (int i = 0; i < 2; i++) small_load(cur[i], p.w[i], p.s[i], p.b[i], row, G, 2 * min(pr + 2, pairs - 1), even, t);
                compute(nxt, pr + 1);
            }
            if (pr < p1) compute(cur, pr);
        };
        if (M > 2) slice(std::integral_constant<int, 2>{});
        else slice(std::integral_constant<int, 1>{});
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
                red[ks][i][4 * c + t][rb * 16 + g] = acc[i][c][0];
                red[ks][i][4 * c + t][rb * 16 + 8 + g] = acc[i][c][1];
            }
        __syncthreads();
        // a thread per (feature, row): the slices in order, the activation, and the group of 64 features as block fixed point
        const int f = tid & 63, m = tid >> 6;
        float gv = 0.f, uv = 0.f;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            gv += red[k][0][2 * m & 7][f] + red[k][0][(2 * m & 7) + 1][f];  // (rows past the fourth: nothing is stored)
            uv += red[k][1][2 * m & 7][f] + red[k][1][(2 * m & 7) + 1][f];
        }
        if (p.ebias[0] != nullptr) {
            gv += p.ebias[0][(size_t)tile.expert * p.I + n0 + f];
            uv += p.ebias[1][(size_t)tile.expert * p.I + n0 + f];
        }
        const __half h16 = __float2half_rn(glu_rt(p.act, gv, uv, p.limit));
        const float hv = m < M ? __half2float(h16) : 0.f;
        float amax = fabsf(hv), sum = hv;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
        }
        if (lane == 0) { gmax[warp] = amax; gsum[warp] = sum; }
        __syncthreads();  // (also: every sum of this item has been read)
        if (m < M) {
            const size_t pos = tile.start + m;
            amax = fmaxf(gmax[warp & ~1], gmax[warp | 1]);
            sum = gsum[warp & ~1] + gsum[warp | 1];
            float sc, inv;
            qi_group_scale<8>(amax, sum, sc, inv);
            const size_t rec = pos * NB + n0 / 64;
            if (f == 0) p.fh.scale[rec] = make_float2(sc, sum);
            const int X = __float2int_rn(hv * inv);
            const int hi_d = (X + 128) >> 8, lo_d = X - (hi_d << 8);
            const int lo7 = __float2int_rn(fmaf(hv, inv, -(float)X) * 128.f);
            unsigned char* d = p.fh.digits + rec * 192 + ((f >> 4) & 3) * 16 + ((f >> 3) & 1) * 8 + (f & 1) * 4 + ((f & 7) >> 1);
            d[0] = (unsigned char)(hi_d & 0xFF);
            d[64] = (unsigned char)(lo_d & 0xFF);
            d[128] = (unsigned char)(lo7 & 0xFF);
            p.h[pos * p.I + n0 + f] = h16;
        }
    }
}

struct DownSmallParams {
    const unsigned char *w, *s, *b;
    int32_t D, I, topk, T;
    FixedRows fh;
    const uint32_t *inds, *pos;
    const float* wts;
    const float* ebias;        // [E, D] or null
    __half* yd;                // [P, D]
    void* out;
    int32_t out_dtype;
    int64_t ldo;
    int32_t accumulate;
    int32_t slices;            // of the inputs per pair: 16 warps / pairs
};

// A block's item: 16 features of one token; warp j * slices + k is slice k of the token's j-th expert.
__global__ void __launch_bounds__(kSmallThreads, 1) moe_down_small_kernel(const DownSmallParams p) {
    __shared__ float part[2][16][2][16];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int j = warp / p.slices, ks = warp % p.slices;
    const int G = p.I / 64, NB = p.D / 16, total = p.T * NB;
    const int pairs = (G + 1) / 2, p0 = pairs * ks / p.slices, p1 = pairs * (ks + 1) / p.slices;
    const bool even = (G & 1) == 0, mine = j < p.topk;
    const int radix = t & 1 ? 0 : 256;
    pdl_launch_dependents();
    // the routing was complete before the gate/up kernel let this one start (it is read past the L1 cache), and the weights
    // depend on nothing else
    auto row_of = [&](int it) {
        return (int64_t)__ldcg(p.inds + (it / NB) * p.topk + (mine ? j : 0)) * p.D + (it % NB) * 16 + g;
    };
    SmallBatch cur, nxt;
    int it = blockIdx.x;
    int64_t row = it < total ? row_of(it) : 0;
    if (it >= total) row = g;
    small_load(cur, p.w, p.s, p.b, row, G, 2 * min(p0, pairs - 1), even, t);
    pdl_wait();
    for (int n = 0; it < total; it += gridDim.x, n++) {
        const int tok = it / NB, next = it + gridDim.x;
        const int64_t next_row = row_of(next < total ? next : it);
        float acc[2] = {0.f, 0.f};
        if (mine) {
            const uint32_t pos = __ldcg(p.pos + tok * p.topk + j);
            // one activation row: its digits are the first four columns, the others zero
            const unsigned char* hd = p.fh.digits + (size_t)pos * G * 192 + min(g & 3, 2) * 64 + t * 16;
            const float2* hs = p.fh.scale + (size_t)pos * G;
            auto compute = [&](const SmallBatch& v, int pr) {
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int grp = 2 * pr + u;
                    if (grp >= G) break;
                    uint4 xb = *reinterpret_cast<const uint4*>(hd + grp * 192);
                    if (g > 3) xb = make_uint4(0, 0, 0, 0);
                    small_mma(acc, v, u, xb, small_part(hs[grp], t), radix);
                }
            };
            int pr = p0;
            for (; pr + 1 < p1; pr += 2) {
                small_load(nxt, p.w, p.s, p.b, row, G, 2 * (pr + 1), even, t);
                compute(cur, pr);
                const bool same = pr + 2 < p1;
                small_load(cur, p.w, p.s, p.b, same ? row : next_row, G, 2 * (same ? pr + 2 : min(p0, pairs - 1)), even, t);
                compute(nxt, pr + 1);
            }
            if (pr < p1) {
                small_load(nxt, p.w, p.s, p.b, next_row, G, 2 * min(p0, pairs - 1), even, t);
                compute(cur, pr);
                cur = nxt;
            }
        }
        row = next_row;
        if (t < 2) {  // row 0 of the set
            part[n & 1][warp][t][g] = acc[0];
            part[n & 1][warp][t][g + 8] = acc[1];
        }
        __syncthreads();
        if (tid < 16) {
            const int d = (it % NB) * 16 + tid;
            float sum = 0.f;
            for (int k = 0; k < p.topk; k++) {
                const uint32_t pos = __ldcg(p.pos + tok * p.topk + k);
                float y = 0.f;
                for (int q = 0; q < p.slices; q++) y += part[n & 1][k * p.slices + q][0][tid] + part[n & 1][k * p.slices + q][1][tid];
                if (p.ebias != nullptr) y += p.ebias[(size_t)__ldcg(p.inds + tok * p.topk + k) * p.D + d];
                const __half y16 = __float2half_rn(y);
                p.yd[(size_t)pos * p.D + d] = y16;
                sum = fmaf(__ldcg(p.wts + tok * p.topk + k), __half2float(y16), sum);
            }
            const size_t o = (size_t)tok * p.ldo + d;
            if (p.out_dtype == kF32) {
                float* op = reinterpret_cast<float*>(p.out) + o;
                *op = p.accumulate ? sum + *op : sum;
            } else if (p.out_dtype == kBF16) {
                uint16_t* op = reinterpret_cast<uint16_t*>(p.out) + o;
                *op = (uint16_t)f32_to_bf16_bits(p.accumulate ? bf16_bits_to_f32(*op) + sum : sum);
            } else {
                __half* op = reinterpret_cast<__half*>(p.out) + o;
                *op = __float2half_rn(p.accumulate ? __half2float(*op) + sum : sum);
            }
        }
    }
}

}  // namespace iq
