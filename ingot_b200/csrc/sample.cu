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
constexpr int kMaxVocab = 262144;
constexpr int kTopBlocks = 8;      // blocks of a cluster, which share a row
constexpr int kTopThreads = 1024;
constexpr int kTopList = 1024;     // keys of a block's list of candidates

// Sort key of a logit: an unsigned that orders like the float (-0 taken as +0 so that it ties with it); 0 = not a candidate.
__device__ __forceinline__ uint32_t order_key(float v) {
    if (!(v >= -FLT_MAX)) return 0u;  // -inf and NaN
    const uint32_t u = __float_as_uint(v == 0.f ? 0.f : v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// With its id: keys are distinct, and of equal logits the lower id has the larger one.
__device__ __forceinline__ unsigned long long full_key(uint32_t u, uint32_t id) {
    return u == 0 ? 0ull : ((unsigned long long)u << 32) | (unsigned long long)(0xFFFFFFFFu - id);
}
__device__ __forceinline__ unsigned long long max_u64(unsigned long long a, unsigned long long b) { return a > b ? a : b; }

struct TopkParams {
    const float* x;
    int64_t ldx;
    int32_t V, span;  // logits of a row, and of a block: a multiple of kTopThreads
    float inv_t[16];
    uint32_t* idx;    // [rows, 64]
    float* val;       // [rows, 64]
    float* z;         // [rows, 2]
};

// The 64 largest keys of a row, its maximum and its softmax denominator, by the eight blocks of a cluster.
//
// A block reads its span once (KPT logits per thread, in registers). The largest keys of 128 groups of its logits (eight lanes
// each) are distinct, so that the 64th of them is not above the block's 64th largest key, and the keys from there on (about 90
// of ordinary logits, whatever the span) are the list from which the block's 64 best are ranked by counting, several threads per
// key. Where the list would not fit (orders made for it), the bound is searched by halving until it does. The first block gets
// the eight sorted runs through distributed shared memory and ranks what is not below the smallest eighth-best.
//
// Bound: latency (a row of 128,000 is 0.5 MB). Two kernels of 4096-logit parts, searching the 64th key two bits and one block-wide
// barrier at a time, took 23 us for one row of 128,000, 34 for eight and 51 for sixteen; now 11.4, 11.5 and 21.
// KEEP: the span stays in registers; where more than eight rows want two blocks per SM (sixteen rows of 128,000 23 -> 21 us), it is read
// again instead. KPT = 0 (spans of more than 16 logits per thread): read again, eight logits a turn of a loop. Unrolled for 32 the
// passes are some 50 KB of instructions, which a decode step's GEMV has driven out of the caches: behind the GEMV of a 151,936 x 2048 4-bit
// head one row took 24.8 us of candidates, rolled 17.3 (four rows 31.5 -> 16.8, eight 78 -> 63 with the GEMV; 262,144: 32.5 -> 21.5). Spans of
// up to 16 stay unrolled (131,072 with its GEMV 40.6 us, rolled 41.9).
template <int KPT, bool KEEP>
__global__ void __launch_bounds__(kTopThreads, KEEP || KPT == 0 ? 1 : 2) __cluster_dims__(kTopBlocks, 1, 1)
    topk64_kernel(const __grid_constant__ TopkParams p) {
    __shared__ unsigned long long list[kTopList], group_max[128], bound_;
    __shared__ unsigned long long run[kTopBlocks][kTopK];  // the first block's: sorted candidates of every block
    __shared__ double part_z[kTopBlocks];                  // likewise
    __shared__ float part_max[kTopBlocks];
    __shared__ float red[32], redz[32];
    __shared__ uint32_t count[2], larger[kTopList];
    const int row = blockIdx.x / kTopBlocks, part = blockIdx.x % kTopBlocks, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    larger[tid] = 0;
    if (tid < 2) count[tid] = 0;
    if (tid == 0) bound_ = 1;  // (where fewer than 64 groups have a candidate: all that there are)
    cluster_sync_all();  // the first block runs: its shared memory may be written
    pdl_wait();
    const float* xr = p.x + (size_t)row * p.ldx;
    const int i0 = part * p.span + tid, end = min(p.V, (part + 1) * p.span);
    auto read = [&](int k) {
        const int i = i0 + k * kTopThreads;
        return i < end ? xr[i] : -INFINITY;
    };
    float kept[KEEP ? KPT : 1];
    if (KEEP) {
#pragma unroll
        for (int k = 0; k < KPT; k++) kept[KEEP ? k : 0] = read(k);
    }
    // every logit of the thread in order of id, eight loads at a time
    auto each = [&](auto f) {
        if constexpr (KPT == 0) {
#pragma unroll 1
            for (int k0 = 0; k0 * kTopThreads < p.span; k0 += 8) {  // (read() ends at the span: its last turn may be short)
                float v[8];
#pragma unroll
                for (int k = 0; k < 8; k++) v[k] = read(k0 + k);
#pragma unroll
                for (int k = 0; k < 8; k++) f(k0 + k, v[k]);
            }
            return;
        }
#pragma unroll
        for (int k0 = 0; k0 < KPT; k0 += 8) {
            float v[8];
#pragma unroll
            for (int k = k0; k < min(KPT, k0 + 8); k++) v[k - k0] = KEEP ? kept[KEEP ? k : 0] : read(k);
#pragma unroll
            for (int k = k0; k < min(KPT, k0 + 8); k++) f(k, v[k - k0]);
        }
    };
    float m = -INFINITY;
    uint32_t best = 0, best_id = 0;
    each([&](int k, float v) {
        const uint32_t u = order_key(v);
        if (u > best) { best = u; best_id = i0 + k * kTopThreads; }
        m = fmaxf(m, v);
    });
    unsigned long long gm = full_key(best, best_id);
    for (int o = 4; o > 0; o >>= 1) gm = max_u64(gm, __shfl_xor_sync(0xffffffffu, gm, o));
    if ((lane & 7) == 0) group_max[4 * warp + (lane >> 3)] = gm;
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) red[warp] = m;
    __syncthreads();
    {  // the 64th of the groups' keys: eight threads count the larger ones of one
        const unsigned long long mine = group_max[tid >> 3];
        uint32_t c = 0;
#pragma unroll
        for (int j = 0; j < 16; j++) c += group_max[(tid & 7) + 8 * j] > mine;
        for (int o = 1; o < 8; o <<= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if ((tid & 7) == 0 && c == kTopK - 1 && mine != 0) bound_ = mine;
    }
    m = red[lane];
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __syncthreads();
    unsigned long long bound = bound_;
    // the keys from the bound on, in any order (few threads have one)
    auto collect = [&](unsigned long long from, uint32_t* n) {
        const uint32_t high = (uint32_t)(from >> 32);
        each([&](int k, float v) {
            const uint32_t u = order_key(v);
            if (u >= high) {
                const unsigned long long key = full_key(u, (uint32_t)(i0 + k * kTopThreads));
                if (key >= from) {
                    const uint32_t at = atomicAdd(n, 1u);
                    if (at < kTopList) list[at] = key;
                }
            }
        });
    };
    collect(bound, &count[0]);
    // sum exp((x - block maximum) / T) in a fixed order: four sums per thread, trees over the warp and the warps (in float64)
    const float inv_t = p.inv_t[row];
    float z = 0.f;
    if (m > -INFINITY) {
        float e[4] = {0.f, 0.f, 0.f, 0.f};
        each([&](int k, float v) { e[k & 3] += i0 + k * kTopThreads < end ? expf((v - m) * inv_t) : 0.f; });
        z = (e[0] + e[1]) + (e[2] + e[3]);
        for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    }
    if (lane == 0) redz[warp] = z;
    __syncthreads();
    uint32_t n = count[0];
    if (n > kTopList) {  // halve between the bound (too many keys) and the top (none) until the list fits; the keys are distinct
        unsigned long long lo = bound, hi = ~0ull;
        while (true) {
            const unsigned long long mid = lo + (hi - lo) / 2;
            uint32_t c = 0;
            each([&](int k, float v) { c += full_key(order_key(v), (uint32_t)(i0 + k * kTopThreads)) >= mid; });
            c = __reduce_add_sync(0xffffffffu, c);
            __syncthreads();
            if (tid == 0) count[1] = 0;
            __syncthreads();
            if (lane == 0) atomicAdd(&count[1], c);
            __syncthreads();
            n = count[1];
            if (n > kTopList) lo = mid;
            else if (n < kTopK) hi = mid;
            else { bound = mid; break; }
        }
        __syncthreads();
        if (tid == 0) count[1] = 0;
        __syncthreads();
        collect(bound, &count[1]);
        __syncthreads();
    }
    // a key's place is the number of larger ones: all threads count, several for a key
    if (n != 0) {
        const uint32_t per = max(1u, kTopThreads / n), c = tid % n, j = tid / n;
        const unsigned long long mine = list[c];
        if (j < per) {
            uint32_t l = 0;
            for (uint32_t i = j; i < n; i += per) l += list[i] > mine;
            if (l != 0) atomicAdd(&larger[c], l);
        }
        __syncthreads();
        if (j == 0 && larger[c] < kTopK) st_dsmem_u64(&run[part][larger[c]], 0, mine);
    }
    if (tid < kTopK && tid >= n) st_dsmem_u64(&run[part][tid], 0, 0ull);
    if (warp == kTopThreads / 32 - 1) {
        double tot = (double)redz[lane];
        for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
        if (lane == 0) {
            st_dsmem_u64(reinterpret_cast<unsigned long long*>(&part_z[part]), 0, (unsigned long long)__double_as_longlong(tot));
            st_dsmem_u32(reinterpret_cast<uint32_t*>(&part_max[part]), 0, __float_as_uint(m));
        }
    }
    cluster_sync_all();
    if (part != 0) return;
    // ---- the first block: two threads per key, four runs each ----------------------------------------------------------
    unsigned long long floor8 = run[lane & 7][7];
    for (int o = 4; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, floor8, o);
        floor8 = other < floor8 ? other : floor8;
    }
    const unsigned long long mine = run[tid >> 7][(tid >> 1) & 63];
    uint32_t place = 0;
    if (mine != 0 && mine >= floor8) {
#pragma unroll
        for (int j = 0; j < kTopBlocks / 2; j++) {
            const unsigned long long* r = run[(tid & 1) * (kTopBlocks / 2) + j];
            int c = 0;
#pragma unroll
            for (int o = 32; o > 0; o >>= 1) c += r[c + o - 1] > mine ? o : 0;
            place += c + (r[c] > mine);
        }
    }
    place += __shfl_xor_sync(0xffffffffu, place, 1);
    const int found = min(__syncthreads_count(mine != 0 && (tid & 1) == 0), kTopK);
    if ((tid & 1) == 0 && mine != 0 && mine >= floor8 && place < kTopK) {
        const uint32_t id = 0xFFFFFFFFu - (uint32_t)(mine & 0xFFFFFFFFull);
        p.idx[(size_t)row * kTopK + place] = id;
        p.val[(size_t)row * kTopK + place] = xr[id];  // the logit's own bits (-0 stays -0)
    }
    if (tid < kTopK && tid >= found) {
        p.idx[(size_t)row * kTopK + tid] = 0xFFFFFFFFu;
        p.val[(size_t)row * kTopK + tid] = -FLT_MAX;
    }
    if (warp == kTopThreads / 32 - 1) {
        const float mq = lane < kTopBlocks ? part_max[lane] : -INFINITY;
        float M = mq;
        for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        double Z = mq > -INFINITY ? part_z[lane & (kTopBlocks - 1)] * exp((double)(mq - M) * (double)inv_t) : 0.0;
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

// (the kernel needs no scratch; what the contract asks for stays as it is)
extern "C" int32_t iq_topk64_scratch_bytes(int32_t rows, int32_t vocab, size_t* bytes) {
    if (bytes == nullptr || rows < 1 || rows > 16 || vocab < 1 || vocab > kMaxVocab) return kErrInvalidArg;
    const size_t parts = (size_t)(vocab + 4095) / 4096;
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
        return fail(ctx, kErrInvalidArg, "topk64: arguments (1..16 rows, up to %d logits, one temperature or one per row)", kMaxVocab);
    if (scratch == nullptr || scratch_bytes < need || (reinterpret_cast<uintptr_t>(scratch) & 7) != 0)
        return fail(ctx, kErrWorkspace, "topk64: scratch %zu < %zu (8-byte aligned)", scratch_bytes, need);
    TopkParams p;
    p.x = x; p.ldx = ldx; p.V = vocab;
    p.span = round_up((vocab + kTopBlocks - 1) / kTopBlocks, kTopThreads);
    for (int r = 0; r < 16; r++) {
        const float t = temperatures[n_temperatures == 1 ? 0 : (r < rows ? r : 0)];
        if (!(t > 0.f)) return fail(ctx, kErrInvalidArg, "topk64: temperature %g", (double)t);
        p.inv_t[r] = 1.0f / t;
    }
    p.idx = idx; p.val = val; p.z = z;
    const int kpt = p.span / kTopThreads;
    auto kernel = kpt <= 4 ? topk64_kernel<4, true> : kpt <= 8 ? topk64_kernel<8, true> : kpt > 16 ? topk64_kernel<0, false>
                  : rows <= 8 ? topk64_kernel<16, true> : topk64_kernel<16, false>;
    return check_cuda(ctx, launch_dependent(kernel, dim3(rows * kTopBlocks), kTopThreads, 0, reinterpret_cast<cudaStream_t>(stream), p), "topk64 launch");
}
