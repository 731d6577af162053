// What follows the lm_head GEMV on the decode path: the arg-max of each row of logits, and the 64 best candidates of
// each row with the row's maximum and softmax denominator (what the sampler needs; the rest of the vocabulary never
// leaves the GPU).
//
// Replaces the reference's argmax_rows (Shaders/verify.metal:525-547) and TopK64 (topk64_part + topk64_merge,
// Shaders/zz_sample.metal; contract in Tests/IngotTests/TopK64Tests.swift:8-63): candidates are the logits
// x >= -FLT_MAX, ordered by value descending with ties to the lower id, padded with (id 0xFFFFFFFF, -FLT_MAX); the values
// are the logits' own bits; z[2r] is the row maximum (exact), z[2r+1] = sum_i exp((x_i - max) / T_r).
#include <float.h>
#include <math.h>

#include <algorithm>

#include "internal.h"
#include "ptx.cuh"

namespace iq {
namespace {

constexpr int kTopK = 64;
constexpr int kChunk = 4096;   // logits per part
constexpr int kMaxParts = 64;  // parts per row: up to 262,144 logits
constexpr int kSortThreads = 1024;

// Sort key of a logit: an unsigned that orders like the float (-0 taken as +0 so that it ties with it); 0 = not a candidate.
__device__ __forceinline__ uint32_t order_key(float v) {
    if (!(v >= -FLT_MAX)) return 0u;  // -inf and NaN
    const uint32_t u = __float_as_uint(v == 0.f ? 0.f : v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

constexpr int kPerThread = kChunk / kSortThreads;
constexpr int kSteps = 16;  // two bits of the key per step

struct SelectSmem {
    uint32_t count[kSteps][3];
    uint32_t above[kPerThread][kSortThreads / 32];  // accepted above the threshold / equal to it, per (k, warp)
    uint32_t equal[kPerThread][kSortThreads / 32];
};

// The 64 largest of the block's kChunk keys (key k of thread t has index t + k * kSortThreads; equal keys count the lower
// index as the larger), fewer when there are fewer candidates: emit(k, position) for each, positions in index order from 0.
// Returns how many. The threshold is found two bits at a time by counting the keys at or above three trial values (a ballot
// per key and value, one barrier per step), and the search stops as soon as exactly 64 are left: about 10 steps for
// ordinary logits. A full bitonic sort of the 4096 keys took 78 barriers and 69 us for eight rows of 128,000.
template <class Emit>
__device__ __forceinline__ int select64(const uint32_t (&u)[kPerThread], SelectSmem& sm, int tid, Emit emit) {
    const int lane = tid & 31, warp = tid >> 5;
    if (tid < kSteps * 3) sm.count[tid / 3][tid % 3] = 0;
    __syncthreads();
    uint32_t thr = 0, n_at = 0xFFFFFFFFu;  // the keys at or above thr are at least 64, if there are that many candidates
    for (int st = 0; st < kSteps; st++) {
        const int sh = 30 - 2 * st;
        uint32_t c[3] = {0, 0, 0};
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const uint32_t trial = thr | ((uint32_t)(j + 1) << sh);
#pragma unroll
            for (int k = 0; k < kPerThread; k++) c[j] += __popc(__ballot_sync(0xffffffffu, u[k] >= trial));
        }
        if (lane < 3) {
            const uint32_t mine = lane == 0 ? c[0] : (lane == 1 ? c[1] : c[2]);
            if (mine != 0) atomicAdd(&sm.count[st][lane], mine);
        }
        __syncthreads();
        const uint32_t n1 = sm.count[st][0], n2 = sm.count[st][1], n3 = sm.count[st][2];
        if (n3 >= kTopK) { thr |= 3u << sh; n_at = n3; }
        else if (n2 >= kTopK) { thr |= 2u << sh; n_at = n2; }
        else if (n1 >= kTopK) { thr |= 1u << sh; n_at = n1; }
        if (n_at == kTopK) break;
    }
    if (thr == 0) thr = 1;  // fewer than 64 candidates: all of them
    // positions in index order: keys above the threshold all count, keys equal to it the first ones
    uint32_t ba[kPerThread], be[kPerThread];
#pragma unroll
    for (int k = 0; k < kPerThread; k++) {
        ba[k] = __ballot_sync(0xffffffffu, u[k] > thr);
        be[k] = __ballot_sync(0xffffffffu, u[k] == thr);
        if (lane == 0) {
            sm.above[k][warp] = __popc(ba[k]);
            sm.equal[k][warp] = __popc(be[k]);
        }
    }
    __syncthreads();
    uint32_t total_above = 0, total_equal = 0, above[kPerThread], equal[kPerThread];  // accepted before this (k, warp)
#pragma unroll
    for (int k = 0; k < kPerThread; k++) {
        const uint32_t a = sm.above[k][lane], e = sm.equal[k][lane];
        uint32_t pa = lane < warp ? a : 0, pe = lane < warp ? e : 0, ta = a, te = e;
        pa = __reduce_add_sync(0xffffffffu, pa);
        pe = __reduce_add_sync(0xffffffffu, pe);
        ta = __reduce_add_sync(0xffffffffu, ta);
        te = __reduce_add_sync(0xffffffffu, te);
        above[k] = total_above + pa;
        equal[k] = total_equal + pe;
        total_above += ta;
        total_equal += te;
    }
    // (when the search stopped early, keys between the threshold and the 64th are all above: total_above + total_equal = 64)
    const uint32_t room = kTopK - total_above;  // equal keys that still fit
    const uint32_t below = (1u << lane) - 1u;
#pragma unroll
    for (int k = 0; k < kPerThread; k++) {
        const uint32_t na = above[k] + __popc(ba[k] & below), ne = equal[k] + __popc(be[k] & below);
        if (u[k] > thr) emit(k, (int)(na + min(ne, room)));
        else if (u[k] == thr && ne < room) emit(k, (int)(na + ne));
    }
    return (int)(total_above + min(total_equal, room));
}

struct TopkParams {
    const float* x;
    int64_t ldx;
    int32_t rows, V, parts;
    float inv_t[16];
    unsigned long long* part_keys;  // [rows, parts, 64] key << 32 | ~id, 0 where a part has fewer
    float* part_mz;                 // [rows, parts, 2] part maximum and sum exp((x - part max) / T)
    uint32_t* idx;                  // [rows, 64]
    float* val;                     // [rows, 64]
    float* z;                       // [rows, 2]
};

__global__ void __launch_bounds__(kSortThreads) topk64_part_kernel(const TopkParams p) {
    __shared__ SelectSmem sel;
    __shared__ float red[32];
    const int part = blockIdx.x, row = blockIdx.y, tid = threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    const float* xr = p.x + (size_t)row * p.ldx;
    const int i0 = part * kChunk;
    float v[kPerThread];
    uint32_t u[kPerThread];
    float m = -INFINITY;
#pragma unroll
    for (int k = 0; k < kPerThread; k++) {
        const int id = i0 + tid + k * kSortThreads;
        v[k] = id < p.V ? xr[id] : -INFINITY;
        u[k] = order_key(v[k]);
        m = fmaxf(m, v[k]);
    }
    // part maximum
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((tid & 31) == 0) red[tid >> 5] = m;
    __syncthreads();
    m = red[tid & 31];
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __syncthreads();
    // sum exp((x - part max) / T) in a fixed order: per thread, warp tree, then the warps in order
    float s = 0.f;
    if (m > -INFINITY) {
        const float it = p.inv_t[row];
#pragma unroll
        for (int k = 0; k < kPerThread; k++)
            if (i0 + tid + k * kSortThreads < p.V) s += expf((v[k] - m) * it);
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((tid & 31) == 0) red[tid >> 5] = s;
    unsigned long long* out = p.part_keys + ((size_t)row * p.parts + part) * kTopK;
    const int n = select64(u, sel, tid, [&](int k, int pos) {  // starts with a barrier
        out[pos] = ((unsigned long long)u[k] << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)(i0 + tid + k * kSortThreads));
    });
    if (tid >= n && tid < kTopK) out[tid] = 0ull;
    if (tid == 0) {
        float tot = 0.f;
        for (int i = 0; i < kSortThreads / 32; i++) tot += red[i];
        p.part_mz[((size_t)row * p.parts + part) * 2] = m;
        p.part_mz[((size_t)row * p.parts + part) * 2 + 1] = tot;
    }
}

__global__ void __launch_bounds__(kSortThreads) topk64_merge_kernel(const TopkParams p) {
    __shared__ SelectSmem sel;
    __shared__ unsigned long long best[kTopK];
    const int row = blockIdx.x, tid = threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    // the parts' candidates in part order, and in id order inside a part: index order is id order
    unsigned long long key[kPerThread];
    uint32_t u[kPerThread];
#pragma unroll
    for (int k = 0; k < kPerThread; k++) {
        const int i = tid + k * kSortThreads;
        key[k] = i < p.parts * kTopK ? p.part_keys[(size_t)row * p.parts * kTopK + i] : 0ull;
        u[k] = (uint32_t)(key[k] >> 32);
    }
    if (tid < kTopK) best[tid] = 0ull;
    const int n = select64(u, sel, tid, [&](int k, int pos) { best[pos] = key[k]; });  // starts with a barrier
    __syncthreads();
    if (tid < kTopK) {
        // one thread per candidate: its place is the number of larger keys (the keys are distinct: they hold the id)
        const unsigned long long k = best[tid];
        int place = tid;
        uint32_t id = 0xFFFFFFFFu;
        float v = -FLT_MAX;
        if (tid < n) {
            place = 0;
            for (int i = 0; i < n; i++) place += best[i] > k;
            id = 0xFFFFFFFFu - (uint32_t)(k & 0xFFFFFFFFull);
            v = p.x[(size_t)row * p.ldx + id];  // the logit's own bits (-0 stays -0)
        }
        p.idx[(size_t)row * kTopK + place] = id;
        p.val[(size_t)row * kTopK + place] = v;
    }
    if (tid >= kSortThreads - 32) {  // the last warp: two parts per lane
        const int lane = tid & 31;
        const float* mz = p.part_mz + (size_t)row * p.parts * 2;
        float mq[kMaxParts / 32], zq[kMaxParts / 32], M = -INFINITY;
#pragma unroll
        for (int j = 0; j < kMaxParts / 32; j++) {
            const int q = lane + 32 * j;
            mq[j] = q < p.parts ? mz[2 * q] : -INFINITY;
            zq[j] = q < p.parts ? mz[2 * q + 1] : 0.f;
            M = fmaxf(M, mq[j]);
        }
        for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        double Z = 0.0;
        const float it = p.inv_t[row];
#pragma unroll
        for (int j = 0; j < kMaxParts / 32; j++)
            if (mq[j] > -INFINITY) Z += (double)zq[j] * exp((double)(mq[j] - M) * (double)it);
        for (int o = 16; o > 0; o >>= 1) Z += __shfl_xor_sync(0xffffffffu, Z, o);
        if (lane == 0) {
            p.z[row * 2] = M;
            p.z[row * 2 + 1] = (float)Z;
        }
    }
}

// arg-max of each row, ties to the lower index (verify.metal:525-547). The eight blocks of a cluster share a row and meet in
// the first one's shared memory: one block alone reads a row of 128,000 logits at the latency of its own loads (16 us).
constexpr int kArgmaxBlocks = 8;
__global__ void __launch_bounds__(1024) __cluster_dims__(kArgmaxBlocks, 1, 1)
    argmax_rows_kernel(const float* __restrict__ x, int64_t ldx, uint32_t* __restrict__ out, int N) {
    __shared__ float bv[32];
    __shared__ uint32_t bi[32];
    __shared__ float cv[kArgmaxBlocks];
    __shared__ uint32_t ci[kArgmaxBlocks];
    // (rows on the x dimension: the others end at 65,535)
    const int row = blockIdx.x / kArgmaxBlocks, part = blockIdx.x % kArgmaxBlocks, tid = threadIdx.x;
    pdl_launch_dependents();
    cluster_sync_all();  // the first block runs: its shared memory may be written
    pdl_wait();
    const float* xr = x + (size_t)row * ldx;
    float m = -INFINITY;
    uint32_t mi = 0;
    constexpr int U = 8;  // loads in flight per thread
    for (uint32_t i = part * 1024 + tid; i < (uint32_t)N; i += U * kArgmaxBlocks * 1024) {  // (unsigned: i and j pass N)
        float v[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
            const uint32_t j = i + k * kArgmaxBlocks * 1024;
            v[k] = j < (uint32_t)N ? xr[j] : -INFINITY;
        }
#pragma unroll
        for (int k = 0; k < U; k++)
            if (v[k] > m) { m = v[k]; mi = i + k * kArgmaxBlocks * 1024; }
    }
    float sm = m;
    for (int o = 16; o > 0; o >>= 1) sm = fmaxf(sm, __shfl_xor_sync(0xffffffffu, sm, o));
    uint32_t si = m == sm ? mi : 0xFFFFFFFFu;
    for (int o = 16; o > 0; o >>= 1) si = min(si, __shfl_xor_sync(0xffffffffu, si, o));
    if ((tid & 31) == 0) { bv[tid >> 5] = sm; bi[tid >> 5] = si; }
    __syncthreads();
    if (tid == 0) {
        float b = bv[0];
        uint32_t ix = bi[0];
        for (int i = 1; i < 32; i++)
            if (bv[i] > b || (bv[i] == b && bi[i] < ix)) { b = bv[i]; ix = bi[i]; }
        st_dsmem_u32(reinterpret_cast<uint32_t*>(&cv[part]), 0, __float_as_uint(b));
        st_dsmem_u32(&ci[part], 0, ix);
    }
    cluster_sync_all();
    if (part == 0 && tid == 0) {
        float b = cv[0];
        uint32_t ix = ci[0];
        for (int i = 1; i < kArgmaxBlocks; i++)
            if (cv[i] > b || (cv[i] == b && ci[i] < ix)) { b = cv[i]; ix = ci[i]; }
        out[row] = ix;
    }
}

}  // namespace
}  // namespace iq

using namespace iq;

extern "C" int32_t iq_argmax_rows(iq_ctx* ctx, void* stream, const float* x, int64_t ldx, int32_t rows, int32_t n,
                                  uint32_t* out) {
    if (ctx == nullptr) return kErrInvalidArg;
    if (x == nullptr || out == nullptr || rows < 1 || n < 1 || ldx < n) return fail(ctx, kErrInvalidArg, "argmax_rows: arguments");
    constexpr int32_t kRows = 1 << 27;  // of one launch: kArgmaxBlocks blocks each
    int32_t st = kOk;
    for (int64_t r = 0; r < rows && st == kOk; r += kRows)
        st = check_cuda(ctx, launch_dependent(argmax_rows_kernel, dim3((unsigned)std::min<int64_t>(rows - r, kRows) * kArgmaxBlocks), 1024, 0,
                                              reinterpret_cast<cudaStream_t>(stream), x + r * ldx, ldx, out + r, n),
                        "argmax_rows launch");
    return st;
}

extern "C" int32_t iq_topk64_scratch_bytes(int32_t rows, int32_t vocab, size_t* bytes) {
    if (bytes == nullptr || rows < 1 || rows > 16 || vocab < 1 || vocab > kChunk * kMaxParts) return kErrInvalidArg;
    const size_t parts = (size_t)(vocab + kChunk - 1) / kChunk;
    *bytes = (size_t)rows * parts * (kTopK * 8 + 2 * 4) + 256;
    return kOk;
}

extern "C" int32_t iq_topk64(iq_ctx* ctx, void* stream, const float* x, int64_t ldx, int32_t rows, int32_t vocab,
                             const float* temperatures, int32_t n_temperatures, uint32_t* idx, float* val, float* z,
                             void* scratch, size_t scratch_bytes) {
    if (ctx == nullptr) return kErrInvalidArg;
    size_t need = 0;
    if (x == nullptr || idx == nullptr || val == nullptr || z == nullptr || temperatures == nullptr || ldx < vocab ||
        (n_temperatures != 1 && n_temperatures != rows) || iq_topk64_scratch_bytes(rows, vocab, &need) != kOk)
        return fail(ctx, kErrInvalidArg, "topk64: arguments (1..16 rows, up to %d logits, one temperature or one per row)",
                    kChunk * kMaxParts);
    if (scratch == nullptr || scratch_bytes < need || (reinterpret_cast<uintptr_t>(scratch) & 7) != 0)
        return fail(ctx, kErrWorkspace, "topk64: scratch %zu < %zu (8-byte aligned)", scratch_bytes, need);
    TopkParams p;
    p.x = x; p.ldx = ldx; p.rows = rows; p.V = vocab;
    p.parts = (vocab + kChunk - 1) / kChunk;
    for (int r = 0; r < 16; r++) {
        const float t = temperatures[n_temperatures == 1 ? 0 : (r < rows ? r : 0)];
        if (!(t > 0.f)) return fail(ctx, kErrInvalidArg, "topk64: temperature %g", (double)t);
        p.inv_t[r] = 1.0f / t;
    }
    p.part_keys = static_cast<unsigned long long*>(scratch);
    p.part_mz = reinterpret_cast<float*>(p.part_keys + (size_t)rows * p.parts * kTopK);
    p.idx = idx; p.val = val; p.z = z;
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(stream);
    cudaError_t e = launch_dependent(topk64_part_kernel, dim3(p.parts, rows), kSortThreads, 0, cs, p);
    if (e == cudaSuccess) e = launch_dependent(topk64_merge_kernel, dim3(rows), kSortThreads, 0, cs, p);
    return check_cuda(ctx, e, "topk64 launch");
}
