// Quantized GEMM on the 5th-generation tensor cores with the dequantised weights in tensor memory, dense and grouped
// (MoE):
//
//   D[128 weight rows, up to 192 tokens] += Wd[128, 64] * X[tokens, 64]^T      per K step of 64 inputs
//
// Why tensor memory. With the fp16 weight tile in shared memory the K step moved 104 KB through the shared-memory port
// (tile stores 16, MMA reads of the tile 16 and of X 32, TMA writes of X 32, codes 8: 832 cycles at 128 B per cycle) for 512
// cycles of MMA, and ran at that port's rate. tcgen05.mma takes its A operand from tensor memory: the dequantisers write
// there with tcgen05.st, a thread per weight row and 64 weights at a time, and what is left for the port is X (written
// and read once) and the packed codes. A step of 64 inputs with N tokens is 2 N cycles of MMA, whatever else the SM does (measured with
// operands resident, beside tcgen05.st, shared-memory loads and spinning warps).
//
// Tensor memory (512 columns): two accumulators of up to 192 columns and four A stages of 32 columns (64 fp16 inputs per
// lane), or two of up to 128 columns and eight A stages. Two accumulators always: the epilogue of a tile runs under the
// next tile's main loop, which one accumulator of 256 columns could not offer beside the A stages.
//
// Warp roles of one persistent CTA (768 threads):
//   warp 0       producer of X tiles: one tensor copy brings two or four K steps of the tile (128-byte swizzle). A step of its
//                own per copy does not do: the wait, the expected bytes and the copy's issue are a chain of 500 cycles in one
//                thread, whatever the box
//   warp 1       allocates tensor memory, issues tcgen05.mma (one lane; in a pair the even CTA's), commits stages and accumulators
//   warp 2       producer of the packed codes: a stage is 128 bytes of 128 weight rows (two to eight K steps), so that DRAM
//                and L2 see whole lines; 128-byte swizzle, so that the dequantisers' row-wise 16-byte loads are free of bank
//                conflicts
//   warp 3       producer of the stage's scales and biases (asynchronous copies of a row's 4-16 bytes)
//   warps 4-7    epilogue
//   warps 8-23   dequantisers, four groups of four warps on every fourth K step (two CTAs per SM: two groups)
// The gate/up form takes 64 gate rows and the matching 64 up rows as one tile of 128: lanes 0-15 of every warp's quadrant
// hold gate rows, lanes 16-31 the same rows of up, so that the activation needs one shuffle per two tokens and
// everything else is the plain form.
// Pairs of CTAs (cta_group::2). One CTA's step of 176 tokens and more takes 500 to 530 cycles of the 2 N that the MMA needs, with A
// and X always there: the issuing thread's loop runs beside sixteen warps that convert codes, and X goes through every SM's port
// twice (written, then read) for 128 features. Two CTAs take 256 features: each holds half of the tile's tokens, the tensor cores
// read both halves, one thread issues for both SMs, and every SM copies half as much X, which the clock feels as well (these
// kernels run into the power limit: 2048 x 4096 x 14336 at 8 bits 1300 MHz with X copied, 1440 without). Copies of X of both CTAs
// count on the even one's barrier, dequantisers and epilogue warps of the odd one arrive there, and commits go to both. 2048 x
// 4096 x 14336 (8 bits, added) 228 -> 210 us, 4096 x 4096 x 7680 225 -> 202, FFN 4096 x 14336 of 1088 rows 338 -> 314 (sustained, at
// the power limit: 284 -> 246 and 426 -> 368 with the K split below). Tiles below some 150 rows
// mostly go to single CTAs, whose finer tiles fill the rounds better; the cost model takes pairs for them too where they save a round (64 rows
// x 19456 x 4096 34.6 -> 28.3 us, K split included). On the way:
// arrivals that release at cluster scope cost the dequantisers 10 to 25 %, reporting the odd CTA's X by a thread of its own 20 %.
// Tiles of a list that hold up to 64 tokens (MoE decode and short prefills) leave the MMA idle: a step of 16 tokens is 72 cycles
// of it, and the 400 cycles of the issuing thread and of its hand-overs are the time. Two CTAs per SM, each with two
// dequantiser groups, half of the shared memory and 256 columns (two accumulators of 64, four A stages), run two such
// chains side by side: 32 experts of 2880 x 2880 (MXFP4) at 64 tokens, gate/up 102 -> 78 us (3.6 TB/s) and down 53 -> 45;
// 128 experts of 2048 x 768 (4 bits) at 200 tokens 100 -> 90 and 51 -> 46. Three groups per CTA were slower (48 registers).
// What bounds it now is issue slots: 70 % busy, two thirds of them the conversion of the codes. With 64 registers a thread it takes the
// plainer form of what it shares with the tall tiles (SPLIT below): tile numbers for work items, no K split, codes converted half a step at a
// time, an issuer that asks its barriers ahead of the MMAs, a guard per stored column. With the tall tiles' forms the MoE block of 32
// experts of 2880 x 2880 (MXFP4, 64 tokens) took 140.8 instead of 137.8 us, 128 of 3584 x 768 at 16 tokens 125 instead of 118, 512 of 3264 x 640
// (4 bits, 64 tokens) 553 instead of 538. The other way round, one issuer loop for both cost 64-row dense calls 5 to 20 %.
// Every wait is bounded: on a timeout the kernel writes a status word, all roles drain and tensor memory is released.
//
// Replaces qmm_t_nax3* (Shaders/qmm_nax_v3.metal:107-256) and, with a tile list, moe_gateup_swiglu2* / moe_down2*
// (Shaders/qmm_nax_moe.metal:442-717) of the reference.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "gqmv.cuh"
#include "ptx.cuh"

namespace iq {

constexpr int kTaGroups = 4;               // dequantiser groups of four warps: one CTA per SM
constexpr int kTaGroupsLow = 2;            // ... two CTAs per SM (tiles of up to 64 tokens)
constexpr int kTaLowRows = 64;
constexpr int ta_threads(int groups) { return 256 + 128 * groups; }
constexpr int kTaMaxRows = 192;            // token rows per tile
constexpr int kTaCodeStage = 128 * 128;    // bytes of a stage of packed codes
constexpr int kTaMaxStages = 12;
constexpr int kTaSmemMax = 232448;
constexpr int kTaSmemLow = 115712;         // two CTAs per SM: half of 228 KB each, less the system's KB
constexpr int kTaSmemFixed = 1024 + 1024;  // alignment, barriers

// K split of the tiles that fill no whole round (below)
struct TaSplit {
    int32_t tiles, units, ctas;  // split tiles (the first ones of the list), units per tile, CTAs that share them
};

struct TaParams {
    const void* s[2];
    const void* b[2];
    int32_t expert_lo;       // first expert held here: tile.expert - expert_lo indexes the stacked tensors
    int32_t N, K;            // weight rows per expert (gate/up: of each matrix), inputs
    int32_t M;               // token rows (dense)
    int32_t tile_rows;       // dense tiling: token rows per tile
    const Tile* tiles;       // work list; null: dense tiling
    const uint32_t* ntiles;
    void* y;
    int32_t y_dtype;
    int64_t ldy;
    int32_t accumulate;
    const float* ebias[2];   // fp32 [E, N] or null
    float limit;
    int32_t act;
    // X copies: a tile of r rows takes the smallest box of xbox * (i + 1) rows, i < nbox, that holds it, xk K steps at a time
    int32_t xbox, nbox, xk;
    int32_t nx, nc;          // stages of X and of codes
    int32_t x_stage;         // bytes of an X stage
    int32_t dcols;           // columns per accumulator: 64, 128 or 192
    int32_t early;           // the tile list is complete when the kernel starts
    TaSplit split;           // dense
    float* part;             // its partial sums
    int32_t ustep;           // K steps per unit of the split
    int32_t pair;            // pairs of CTAs: tiles, rounds and the split count pairs
    int32_t vec;             // how scales are read: 1 by asynchronous copies, 0 in pairs of bytes, -1 (MXFP4) byte by byte
    int32_t* status;
};

struct TaMaps {
    CUtensorMap x[4], w[2];
};

// ---- split of the last round ------------------------------------------------------------------------------------------
// T tiles over G CTAs take ceil(T / G) rounds, the last one with T % G tiles: 336 tiles on 148 CTAs spend a third of the time on
// 40 of them, and a 64-row call has 52 tiles in all. So the R tiles beyond the whole rounds are divided along K: their
// R x units units of `ustep` K steps are dealt to the CTAs in equal contiguous runs (a run touches two tiles at most). A piece of
// a tile goes to a slot of fp32 sums, and ta_sum_kernel behind the GEMM adds a tile's slots in the order of K and stores.
// Measured and taken back: sums by whichever piece ends last (four epilogue warps read 98 KB per piece at the latency of their
// loads: 20 us for four pieces of 192 tokens, under which the next tile's accumulator waits); tile lists (a round is one of many).
// On one B200, us: 64 rows x 4096 x 14336 (8 bits) 72.7 -> 25.9, 128 x 7744 x 11520 (4 bits) 52.8 -> 36.6, 320 x 4096 x 14336
// 65.5 -> 44.6, 4096 x 1024 x 7680 80.4 -> 72.8, 2048 x 4096 x 14336 (8 bits, added) 248 -> 239; dense FFN of 256 rows, 2048 x 7680 81 -> 65.
constexpr int kTaSplitPieces = 8;    // pieces per tile at most (one more where a run begins in the tile before)
// Cycles of a K step of tiles of `rows` tokens (fitted to dense calls of 64 to 4096 rows; `low`: two CTAs share the SM), and of a split:
// the sums' kernel, and the partial sums that are written and read at some 1900 bytes per cycle.
inline int ta_step_cycles(int rows, bool low, bool pair) {
    const int over = rows > 64 ? rows - 64 : 0;
    return pair ? 420 + over * 9 / 20 : low ? 880 + over * 2 : 400 + over;
}
inline long long ta_split_cycles(const TaSplit& s, int rows, bool pair) { return 7000 + (long long)(s.ctas + s.tiles) * rows * (pair ? 2048 : 1024) / 1900; }
inline TaSplit ta_split(int total, int ctas, int ksteps, int ustep, int rows, bool pair) {
    TaSplit r;
    r.units = (ksteps + ustep - 1) / ustep;
    r.tiles = total < ctas ? total : total % ctas;
    r.ctas = r.tiles * kTaSplitPieces < ctas ? r.tiles * kTaSplitPieces : ctas;
    if (r.tiles * r.units < r.ctas) r.ctas = r.tiles * r.units;
    // the round saved, less the CTA's share of it, has to be longer than what the split costs
    if (r.tiles == 0 || (long long)(r.ctas - r.tiles) * ksteps * ta_step_cycles(rows, false, pair) <= ta_split_cycles(r, rows, pair) * r.ctas) r.tiles = r.ctas = 0;
    return r;
}
// What a CTA does, worked out once and read from shared memory at every item (in registers it made the roles' loops spill): its
// pieces of split tiles, then whole tiles.
struct TaSched {
    int32_t total, n_tiles, m_tiles, split;  // work items, tiles of features, tiles of tokens, split tiles
    int32_t np;
    struct Piece {
        int32_t tile, ks0, ks1;
        int32_t slot;  // of the partial sums, -1: the whole tile
    } piece[2];
};
// The CTAs [c0, c1) share split tile t; a CTA's piece is in the slot of its number, or of ctas + t where the tile is its second
__host__ __device__ inline void ta_split_tile(const TaSplit& s, int t, int& c0, int& c1, int& slot0) {
    const int all = s.tiles * s.units, ua = t * s.units;
    c0 = ((ua + 1) * s.ctas - 1) / all;  // the last CTA whose run starts at or before the tile's first unit
    c1 = ((ua + s.units) * s.ctas - 1) / all + 1;
    slot0 = c0 * all / s.ctas < ua ? s.ctas + t : c0;
}
// floats of a slot for tiles of up to `rows` tokens; slots: one per CTA, one per split tile
__host__ __device__ constexpr int ta_slot(int rows) { return 128 * ((rows + 15) & ~15); }
inline size_t ta_split_bytes(const TaSplit& s, int rows, bool pair) { return (size_t)(s.ctas + s.tiles) * ta_slot(rows) * (pair ? 8 : 4); }

// Shared-memory and instruction descriptors: K-major B tile with 128-byte swizzle (rows of 128 bytes, 8-row groups 1024
// bytes apart; the low 14 bits take the address in units of 16 bytes), fp16 operands, fp32 accumulator, M = 128.
constexpr uint64_t kTaDescHi = ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
// n: 16 to 256 in steps of 16, for M = 128 and for a pair's 256, whose CTAs then hold whole groups of eight rows each. (Steps of 32 on pairs,
// which is all that CUTLASS's form with A in tensor memory offers, cost lists 0.3 to 1 %; tiles of all counts of rows are tested.)
__device__ __forceinline__ uint32_t ta_idesc(int n, int ctas) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((8u * ctas) << 24); }

// D[128, N] (+)= A[128, 16] (tensor memory: lane = row, two inputs per column) * B[N, 16]^T (shared memory)
// (PAIR: 256 rows, the upper 128 of A and D in the tensor memory of the pair's other CTA, half of B's rows in its shared memory)
template <bool PAIR>
__device__ __forceinline__ void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    if (PAIR) {
        asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
            ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(acc)
            : "memory");
        return;
    }
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// ---- formats ----------------------------------------------------------------------------------------------------------
// KPS: K steps of 64 inputs per stage of codes (128 bytes of a row); BPS: code bytes of a row per step.
template <int FMT>
struct TaFmt {
    static constexpr int BPS = FMT == kFmtAffine8 ? 64 : (FMT == kFmtTernary ? 16 : 32);
    static constexpr int KPS = 128 / BPS;
    static constexpr int GROUP = (FMT == kFmtMxfp4 || FMT == kFmtAffine4G32) ? 32 : (FMT == kFmtTernary ? 128 : 64);
    static constexpr bool BIAS = FMT == kFmtAffine4 || FMT == kFmtAffine8 || FMT == kFmtAffine4G32;
    static constexpr int ES = FMT == kFmtMxfp4 ? 1 : 2;           // bytes of a scale
    static constexpr int SPB = 64 * KPS / GROUP * ES;             // scale bytes of a row per stage of codes: 4, 8 or 16
    static constexpr int STAGE = kTaCodeStage + 128 * SPB * (BIAS ? 2 : 1);
};
inline int ta_code_stage(int32_t fmt) {
    switch (fmt) {
        case kFmtAffine4: return TaFmt<kFmtAffine4>::STAGE;
        case kFmtAffine8: return TaFmt<kFmtAffine8>::STAGE;
        case kFmtMxfp4: return TaFmt<kFmtMxfp4>::STAGE;
        case kFmtAffine4G32: return TaFmt<kFmtAffine4G32>::STAGE;
        default: return TaFmt<kFmtTernary>::STAGE;
    }
}

// 32 consecutive inputs of one weight row -> 16 registers of two fp16 weights each, in input order. codes: the row's
// 128-byte line in the stage (sw = row % 8: the swizzle), unit: the first 16-byte piece of them in it (ternary: of the 64
// inputs, half h). sc / bi: the scale and bias bits. small: every lane's scales are below 2^-4 (4-bit affine codes).
//
// 4-bit affine codes with such scales: a code in the bits 4-7 of a half is a subnormal, q * 2^-20, so that one fma with the scale times 2^20
// is w = fma(q, s, b), rounded once as before: 13 instructions for eight codes instead of 16 (1024 + q brought to q by an exact fma
// first, which scales that overflow a half times 2^20 still take, a warp at a time). The conversion bounds the low tiles and shares the issue slots with
// the MMA's thread in the tall ones: 64 rows x 8192 x 4096 16.9 -> 15.8 us, 512 rows 36.8 -> 34.1, FFN 4096 x 14336 of 256 rows 103.0 -> 95.7, of
// 1088 318 -> 308, the MoE block of 128 experts of 2048 x 768 at 512 tokens 178 -> 162, at 4096 474 -> 456.
template <int FMT>
__device__ __forceinline__ void ta_dequant32(uint32_t codes, uint32_t unit, int h, uint32_t sw, uint32_t sc, uint32_t bi, bool small,
                                             uint32_t (&o)[16]) {
    if (FMT == kFmtAffine4 || FMT == kFmtAffine4G32) {
        const uint4 v = lds128(codes + ((unit ^ sw) << 4));
        const float s = bf16_bits_to_f32(sc), b = bf16_bits_to_f32(bi);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        const uint32_t b2 = pack_half2(b, b);
        if (small) {
            const float s20 = s * 1048576.0f;
            const uint32_t s2 = pack_half2(s20, s20);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t w4 = w[i] << 4;  // byte j: input 2j in its upper nibble, where w has input 2j + 1
#pragma unroll
                for (int j = 0; j < 4; j++) o[i * 4 + j] = hfma2_u32(__byte_perm(w4, w[i], 0x0400 + 0x0101 * j) & 0x00F000F0u, s2, b2);
            }
            return;
        }
        const uint32_t s2 = pack_half2(s, s);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                // byte j of the word holds inputs 2j (low nibble) and 2j + 1: (1024 + q_lo, 1024 + 16 q_hi), brought to
                // (q_lo, q_hi) by one exact fma, then w = fma(q, s, b) rounded once
                const uint32_t t = (__byte_perm(w[i], 0u, 0x4040 + 0x0101 * j) & 0x00F0000Fu) | 0x64006400u;
                o[i * 4 + j] = hfma2_u32(hfma2_u32(t, 0x2C003C00u, 0xD400E400u), s2, b2);
            }
    } else if (FMT == kFmtAffine8) {
        const float s = bf16_bits_to_f32(sc), b = bf16_bits_to_f32(bi);
        const uint32_t s2 = pack_half2(s, s), b2 = pack_half2(b, b);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const uint4 v = lds128(codes + (((unit + q) ^ sw) << 4));
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const uint32_t t = __byte_perm(w[i], 0x64646464u, j ? 0x4342 : 0x4140);  // 1024 + q
                    o[q * 8 + i * 2 + j] = dq_pair(t, s2, b2);
                }
        }
    } else if (FMT == kFmtTernary) {
        // 32 codes of two bits in eight bytes; w = (q - 1) * s with the fp16 scale as it is stored: exact in fp16
        const uint2 v = lds64(codes + ((unit ^ sw) << 4) + 8 * h);
        const uint32_t s2 = (sc & 0xFFFFu) | (sc << 16);
        const uint32_t w[2] = {v.x, v.y};
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) {
                // inputs 2j and 2j + 1 are the bits 4j..4j+1 and 4j+2..4j+3: multiplying by 1 + 2^14 puts the second pair
                // at bit 16; 1024 + q, then (q - 1) * s
                const uint32_t n = (w[i] >> (4 * j)) & 0xFu;
                const uint32_t t = ((n * 0x4001u) & 0x00030003u) | 0x64006400u;
                __half2 q = __hsub2(*reinterpret_cast<const __half2*>(&t), __half2half2(__ushort_as_half(0x6401)));
                o[i * 8 + j] = hmul2_u32(*reinterpret_cast<uint32_t*>(&q), s2);
            }
    } else {
        const uint4 v = lds128(codes + ((unit ^ sw) << 4));
        const DqConst d = make_dq<kFmtMxfp4>(sc);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint32_t q[4];
            cvt_e2m1x8(w[i], q);
#pragma unroll
            for (int j = 0; j < 4; j++) o[i * 4 + j] = hmul2_u32(q[j], d.s2);
        }
    }
}

// The activation of CW token columns of a tile: lanes l and l + 16 hold gate and up of one feature; the lower lane finishes token j, the
// upper token j + 1.
template <int CW>
__device__ __forceinline__ void ta_gated(const TaParams& p, const float (&v)[CW], int mi, float (&g)[CW / 2]) {
    float u[CW / 2];
#pragma unroll
    for (int j = 0; j < CW / 2; j++) {
        const float other = __shfl_xor_sync(0xffffffffu, mi ? v[2 * j] : v[2 * j + 1], 16);
        g[j] = mi ? other : v[2 * j];
        u[j] = mi ? v[2 * j + 1] : other;
    }
    auto act = [&](auto tag) {
#pragma unroll
        for (int j = 0; j < CW / 2; j++) g[j] = glu<decltype(tag)::value>(g[j], u[j], p.limit);
    };
    if (p.act == kActSilu) act(std::integral_constant<int, kActSilu>{});
    else if (p.act == kActSwigluOai) act(std::integral_constant<int, kActSwigluOai>{});
    else if (p.act == kActGelu) act(std::integral_constant<int, kActGelu>{});
    else act(std::integral_constant<int, kActRelu2>{});
}

// What becomes of CW token columns of a tile: v[j] is feature n of token row0 + j (gate/up: ta_gated) with the expert's bias, j < live.
template <int EPI, int CW>
__device__ __forceinline__ void ta_store(const TaParams& p, float (&v)[CW], int row0, int n, bool n_ok, int live, int mi) {
    if (EPI) {
        float g[CW / 2];
        ta_gated(p, v, mi, g);
        if (!n_ok) return;
        __half* yp = reinterpret_cast<__half*>(p.y) + (size_t)(row0 + mi) * p.ldy + n;
        const size_t step = 2 * p.ldy;
        if (live >= CW) {
#pragma unroll
            for (int j = 0; j < CW / 2; j++, yp += step) *yp = __float2half_rn(g[j]);
        } else {
#pragma unroll
            for (int j = 0; j < CW / 2; j++, yp += step)
                if (2 * j + mi < live) *yp = __float2half_rn(g[j]);
        }
    } else {
        if (!n_ok) return;
        const size_t step = p.ldy;
        auto store = [&](auto* y, auto load_f, auto round_f) {
            y += (size_t)row0 * p.ldy + n;
            if (p.accumulate) {  // all loads before the first store
                float old[CW];
                auto* yp = y;
#pragma unroll
                for (int j = 0; j < CW; j++, yp += step) old[j] = j < live ? load_f(*yp) : 0.f;
#pragma unroll
                for (int j = 0; j < CW; j++) v[j] = old[j] + v[j];
            }
            if (live >= CW) {
#pragma unroll
                for (int j = 0; j < CW; j++, y += step) *y = round_f(v[j]);
            } else {
#pragma unroll
                for (int j = 0; j < CW; j++, y += step)
                    if (j < live) *y = round_f(v[j]);
            }
        };
        if (p.y_dtype == kF32) store(reinterpret_cast<float*>(p.y), [](float f) { return f; }, [](float f) { return f; });
        else if (p.y_dtype == kF16) store(reinterpret_cast<__half*>(p.y), [](__half h) { return __half2float(h); }, [](float f) { return __float2half_rn(f); });
        else store(reinterpret_cast<uint16_t*>(p.y), [](uint16_t u) { return bf16_bits_to_f32(u); }, [](float f) { return (uint16_t)f32_to_bf16_bits(f); });
    }
}

// The same with a guard per column instead of stepped pointers, for the low tiles' kernel: it has 64 registers a thread, and few of its
// sets of 16 columns are full.
template <int EPI, int CW>
__device__ __forceinline__ void ta_store_low(const TaParams& p, float (&v)[CW], int row0, int n, bool n_ok, int live, int mi) {
    if (EPI) {
        float g[CW / 2];
        ta_gated(p, v, mi, g);
        __half* yp = reinterpret_cast<__half*>(p.y) + (size_t)(row0 + mi) * p.ldy + n;
#pragma unroll
        for (int j = 0; j < CW / 2; j++)
            if (n_ok && 2 * j + mi < live) yp[(size_t)(2 * j) * p.ldy] = __float2half_rn(g[j]);
    } else {
        const size_t o0 = (size_t)row0 * p.ldy + n;
        auto store = [&](auto* y, auto load_f, auto round_f) {
            if (p.accumulate) {  // all loads before the first store
                float old[CW];
#pragma unroll
                for (int j = 0; j < CW; j++) old[j] = n_ok && j < live ? load_f(y[o0 + (size_t)j * p.ldy]) : 0.f;
#pragma unroll
                for (int j = 0; j < CW; j++) v[j] = old[j] + v[j];
            }
#pragma unroll
            for (int j = 0; j < CW; j++)
                if (n_ok && j < live) y[o0 + (size_t)j * p.ldy] = round_f(v[j]);
        };
        if (p.y_dtype == kF32) store(reinterpret_cast<float*>(p.y), [](float f) { return f; }, [](float f) { return f; });
        else if (p.y_dtype == kF16) store(reinterpret_cast<__half*>(p.y), [](__half h) { return __half2float(h); }, [](float f) { return __float2half_rn(f); });
        else store(reinterpret_cast<uint16_t*>(p.y), [](uint16_t u) { return bf16_bits_to_f32(u); }, [](float f) { return (uint16_t)f32_to_bf16_bits(f); });
    }
}

// EPI: 0 store, 1 gate + up + activation.
// PAIR: a cluster of two CTAs works on tiles of twice the features.
template <int FMT, int EPI, int GROUPS, bool PAIR>
__global__ void __launch_bounds__(ta_threads(GROUPS), GROUPS == kTaGroups ? 1 : 2) qmm_ta_kernel(const __grid_constant__ TaMaps maps, const TaParams p) {
    using F = TaFmt<FMT>;
    constexpr int KPS = F::KPS;
    static_assert(!PAIR || GROUPS == kTaGroups, "a pair has its SMs to itself");
    constexpr uint32_t TCOLS = GROUPS == kTaGroups ? 512 : 256;
    constexpr int CTAS = PAIR ? 2 : 1;
    constexpr int RS = GROUPS == kTaGroups ? 2 : 1;  // A stages per hand-over to the issuer
    constexpr bool SPLIT = GROUPS == kTaGroups;      // (two CTAs per SM: tiles are never divided along K)
    const uint32_t rank = PAIR ? cluster_rank() : 0;  // the even CTA issues the MMAs
    const int unit = (int)blockIdx.x / CTAS, units = (int)gridDim.x / CTAS;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t codes0 = smem_u32(smem), x0 = codes0 + p.nc * kTaCodeStage;  // codes, X, scales
    const uint32_t scales0 = x0 + p.nx * p.x_stage;
    constexpr int SSTAGE = F::STAGE - kTaCodeStage;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)p.nc * F::STAGE + (size_t)p.nx * p.x_stage);
    const uint32_t bar_cfull = smem_u32(bars), bar_cempty = bar_cfull + 8 * kTaMaxStages, bar_xfull = bar_cempty + 8 * kTaMaxStages;
    const uint32_t bar_xempty = bar_xfull + 8 * kTaMaxStages, bar_aready = bar_xempty + 8 * kTaMaxStages;
    const uint32_t bar_aempty = bar_aready + 64, bar_tfull = bar_aempty + 64, bar_tempty = bar_tfull + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4 * kTaMaxStages + 20);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile TaSched* sched = reinterpret_cast<volatile TaSched*>(tmem_slot + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < p.nc; i++) {
            mbar_init(bar_cfull + 8 * i, 1 + 32);  // the codes' copy, the scale producer's lanes
            mbar_init(bar_cempty + 8 * i, 4 * GROUPS);
        }
        for (int i = 0; i < p.nx; i++) {
            mbar_init(bar_xfull + 8 * i, 1);
            mbar_init(bar_xempty + 8 * i, 1);
        }
        for (int i = 0; i < 8; i++) {
            mbar_init(bar_aready + 8 * i, 4 * RS * CTAS);
            mbar_init(bar_aempty + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(bar_tfull + 8 * i, 1);
            mbar_init(bar_tempty + 8 * i, 4 * CTAS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (SPLIT && threadIdx.x == 0) {  // the work list
        if (p.tiles != nullptr && !p.early) pdl_wait();
        constexpr int NROWS = EPI ? 64 : 128;
        const int n_tiles = (p.N + CTAS * NROWS - 1) / (CTAS * NROWS);
        const int m_tiles = p.tiles != nullptr ? (int)(*p.ntiles) : (p.M + p.tile_rows - 1) / p.tile_rows;
        const int total = m_tiles * n_tiles, bid = unit;
        const TaSplit& sp = p.split;
        sched->total = total; sched->n_tiles = n_tiles; sched->m_tiles = m_tiles; sched->split = sp.tiles;
        int np = 0;
        if (bid < sp.ctas) {
            const int all = sp.tiles * sp.units, lo = bid * all / sp.ctas, hi = (bid + 1) * all / sp.ctas;
            for (int t = lo / sp.units; t * sp.units < hi; t++, np++) {  // (two at most)
                const int ua = t * sp.units, ub = ua + sp.units;
                volatile TaSched::Piece& c = sched->piece[np];
                int c0, c1, slot0;
                ta_split_tile(sp, t, c0, c1, slot0);
                c.tile = t; c.ks0 = max(lo - ua, 0) * p.ustep; c.ks1 = min((min(hi, ub) - ua) * p.ustep, p.K / 64);
                c.slot = c1 - c0 == 1 ? -1 : bid == c0 ? slot0 : bid;
            }
        }
        sched->np = np;
    }
    if (warp == 1) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TCOLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TCOLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();  // the other CTA's barriers exist
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // The weights do not depend on the previous kernel of the stream, a tile list, the activations and y do. With dense tiling the
    // weights' producers and the dequantisers start at once. With p.early as well: the tile list is complete then, because the
    // first kernel of the chain (packing, gate/up, down) waited in every thread before it let the next one start. An early kernel
    // of the chain lets its own successor start without having waited; that one may read the list on the strength of the first
    // kernel's wait alone, and nothing else of what its predecessors wrote before its own.
    if (p.tiles == nullptr) pdl_launch_dependents();
    if ((p.tiles != nullptr && !p.early) || !(warp == 2 || warp == 3 || warp >= 8)) pdl_wait();
    if (p.tiles != nullptr) pdl_launch_dependents();

    constexpr int NROWS = EPI ? 64 : 128;  // output features per tile
    const int ksteps = p.K / 64;
    int n_all = 0, m_all = 0;
    if (!SPLIT) {
        n_all = (p.N + NROWS - 1) / NROWS;
        m_all = p.tiles != nullptr ? (int)(*p.ntiles) : (p.M + p.tile_rows - 1) / p.tile_rows;
    }
    const int na = p.dcols == 128 ? 8 : 4;
    const uint32_t tmem_a = tmem + 2 * p.dcols;
    struct Item {
        int ks0, ks1, expert, row0, rows, n0;
    };
    // work items: the pieces and tiles of the schedule, 0 up; without one the tiles themselves
    const int first = SPLIT ? 0 : unit, stride = SPLIT ? 1 : units;
    auto item = [&](int i, Item& t) -> bool {
        int tile;
        const int np = SPLIT ? sched->np : 0, n_tiles = SPLIT ? sched->n_tiles : n_all, m_tiles = SPLIT ? sched->m_tiles : m_all;
        if (!SPLIT) {
            tile = i;
            t.ks0 = 0; t.ks1 = ksteps;
            if (tile >= n_all * m_all) return false;
        } else if (i < np) {
            tile = sched->piece[i].tile; t.ks0 = sched->piece[i].ks0; t.ks1 = sched->piece[i].ks1;
        } else {
            tile = sched->split + unit + (i - np) * units;
            t.ks0 = 0; t.ks1 = ksteps;
            if (tile >= sched->total) return false;
        }
        if (p.tiles != nullptr) {
            const Tile l = p.tiles[tile / n_tiles];
            t.expert = (int)l.expert - p.expert_lo; t.row0 = (int)l.start; t.rows = (int)l.count;
            t.n0 = ((tile % n_tiles) * CTAS + (int)rank) * NROWS;
        } else {
            t.expert = 0; t.row0 = (tile % m_tiles) * p.tile_rows; t.rows = min(p.tile_rows, p.M - t.row0);
            t.n0 = ((tile / m_tiles) * CTAS + (int)rank) * NROWS;
        }
        return true;
    };

    if (warp == 0) {
        // ================= X producer =================
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            Item t;
            for (int i = first; ok && item(i, t); i += stride) {
                const int bi = (t.rows - 1) / p.xbox;
                const CUtensorMap* const map = &maps.x[bi];
                const uint32_t bytes = (uint32_t)(p.xbox * (bi + 1) * p.xk * 128);
                const int xrow = t.row0 + (PAIR ? (int)rank * (((t.rows + 15) & ~15) / 2) : 0);  // a pair's CTAs hold half of the MMA's tokens each
                for (int ks = t.ks0; ks < t.ks1; ks += p.xk) {
                    if (!(ok = mbar_wait(bar_xempty + 8 * s, ph ^ 1, abort_flag))) break;
                    if (rank == 0) mbar_arrive_expect_tx(bar_xfull + 8 * s, bytes);  // (of both halves)
                    if (PAIR) tma_load_3d_pair(x0 + s * p.x_stage, map, bar_xfull + 8 * s, 0, xrow, ks);
                    else tma_load_3d(x0 + s * p.x_stage, map, bar_xfull + 8 * s, 0, xrow, ks);
                    if (++s == p.nx) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 2) {
        // ================= producer of the packed codes =================
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            Item t;
            for (int i = first; ok && item(i, t); i += stride) {
                const int wrow = t.expert * p.N + t.n0;
                for (int ch = t.ks0 / KPS; ch * KPS < t.ks1; ch++) {
                    if (!(ok = mbar_wait(bar_cempty + 8 * s, ph ^ 1, abort_flag))) break;
                    mbar_arrive_expect_tx(bar_cfull + 8 * s, kTaCodeStage);
                    const uint32_t dst = codes0 + s * kTaCodeStage;
                    tma_load_2d(dst, &maps.w[0], bar_cfull + 8 * s, ch * 128, wrow);
                    if (EPI) tma_load_2d(dst + kTaCodeStage / 2, &maps.w[1], bar_cfull + 8 * s, ch * 128, wrow);
                    if (++s == p.nc) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 3) {
        // ================= producer of the scales and biases =================
        // Per stage of codes the SPB scale bytes of each of the 128 rows: lane l takes rows l, l + 32, ... Row pitches that
        // allow it go by asynchronous copies, others (an odd number of groups) by two-byte loads, MXFP4 scales at an odd address
        // (a tensor inside a mapped file) by bytes. Rows beyond the matrix
        // take the last row's: their weights only feed rows of D that are not stored.
        constexpr int SPB = F::SPB, NT = F::BIAS ? 2 : 1;
        const size_t pitch = (size_t)p.K / F::GROUP * F::ES;
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        Item t;
        for (int it = first; ok && item(it, t); it += stride) {
            const char* src[4][NT];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int row = lane + 32 * i, mi = EPI ? i >> 1 : 0, n = min(t.n0 + (EPI ? row & 63 : row), p.N - 1);
                const size_t o = ((size_t)t.expert * p.N + n) * pitch;
                src[i][0] = static_cast<const char*>(p.s[mi]) + o;
                if (NT == 2) src[i][NT - 1] = static_cast<const char*>(p.b[mi]) + o;
            }
            for (int ch = t.ks0 / KPS; ch * KPS < t.ks1; ch++) {
                ok = mbar_wait(bar_cempty + 8 * s, ph ^ 1, abort_flag);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                const uint32_t dst = scales0 + s * SSTAGE;
                const int left = (int)pitch - ch * SPB;  // scale bytes of a row from this stage on
                if (p.vec > 0) {
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int m = 0; m < NT; m++)
                            cp_async_ca<SPB>(dst + m * 128 * SPB + (lane + 32 * i) * SPB, src[i][m] + ch * SPB);
                } else {
                    uint32_t v[4][NT][SPB / 2];
                    auto load = [&](auto bytes) {  // (the choice outside: the loads of a stage go out together)
#pragma unroll
                        for (int i = 0; i < 4; i++)
#pragma unroll
                            for (int m = 0; m < NT; m++)
#pragma unroll
                                for (int e = 0; e < SPB / 2; e++) {
                                    const char* a = src[i][m] + ch * SPB + min(2 * e, left - 2);
                                    v[i][m][e] = decltype(bytes)::value ? ldg_nc_u8(a) | (ldg_nc_u8(a + 1) << 8) : ldg_nc_u16(a);
                                }
                    };
                    if (FMT == kFmtMxfp4 && p.vec < 0) load(std::true_type{});
                    else load(std::false_type{});
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int m = 0; m < NT; m++)
#pragma unroll
                            for (int e = 0; e < SPB / 4; e++)
                                sts32(dst + m * 128 * SPB + (lane + 32 * i) * SPB + 4 * e, v[i][m][2 * e] | (v[i][m][2 * e + 1] << 16));
                }
                // (the copies' arrival orders copies only: plain stores are published by an arrival that releases them)
                if (p.vec > 0) cp_async_arrive_noinc(bar_cfull + 8 * s);
                else mbar_arrive(bar_cfull + 8 * s);
                if (++s == p.nc) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        // The loop's time is its round trips to barriers (100 to 200 cycles each beside the dequantisers), not the MMAs' issue (some 15
        // cycles each). So every barrier is asked one step ahead, behind the MMAs, and with four dequantiser groups two A stages are
        // handed over on one barrier and back on their own: 64 x 14336 x 14336 (MXFP4) 46.7 -> 42.7 us, 192 x 4096 x 4096 19.9 -> 18.3
        // (also handed back together, tiles of 192 rows were 3 % slower; two groups, which hold two such pairs in all, 5 to 10 %).
        if (rank == 0 && elect_one()) {
            auto commit = [&](uint32_t bar) {
                if (PAIR) umma_commit_pair(bar);
                else umma_commit(bar);
            };
            int xs = 0, as = 0, acc = 0;
            uint32_t xph = 0, aph = 0, tph = 0;
            uint32_t a_hint = 0, x_hint = 0;
            const uint32_t xdesc0 = (x0 & 0x3FFFFu) >> 4;
            bool ok = true;
            Item t;
            for (int i = first; ok && item(i, t); i += stride) {
                const uint32_t idesc = ta_idesc((t.rows + 15) & ~15, CTAS);
                if (!(ok = mbar_wait_hint(0, bar_tempty + 8 * acc, tph ^ 1, abort_flag))) break;
                const uint32_t td = tmem + acc * p.dcols;
                const uint32_t kunits = (uint32_t)(p.xbox * ((t.rows - 1) / p.xbox + 1) / CTAS * 8);
                if constexpr (!SPLIT) {
                    // low tiles: the MMAs are over before answers asked behind them would come, so the barriers are asked ahead of them
                    for (int ks0 = 0; ks0 < ksteps && ok; ks0 += p.xk) {
                        if (!(ok = mbar_wait_hint(x_hint, bar_xfull + 8 * xs, xph, abort_flag))) break;
                        const int ks1 = min(ksteps, ks0 + p.xk);
                        uint32_t xdesc = xdesc0 + xs * ((uint32_t)p.x_stage >> 4);
                        const uint32_t xdone = bar_xempty + 8 * xs;
                        if (++xs == p.nx) { xs = 0; xph ^= 1; }
                        for (int ks = ks0; ks < ks1; ks++, xdesc += kunits) {
                            if (!(ok = mbar_wait_hint(a_hint, bar_aready + 8 * as, aph, abort_flag))) break;
                            const uint32_t ta = tmem_a + as * 32, done = bar_aempty + 8 * as;
                            if (++as == na) { as = 0; aph ^= 1; }
                            a_hint = mbar_test(bar_aready + 8 * as, aph);
                            if (ks + 1 == ks1) x_hint = mbar_test(bar_xfull + 8 * xs, xph);
                            tc_fence_after();
#pragma unroll
                            for (int kk = 0; kk < 4; kk++)
                                umma_f16_ta<PAIR>(td, ta + 8 * kk, kTaDescHi | (uint64_t)(xdesc + 2 * kk), idesc, (ks | kk) ? 1u : 0u);
                            commit(done);
                        }
                        commit(xdone);
                    }
                } else {
                    uint32_t more = 0;  // the tile's first MMA starts the sums
                    for (int left = t.ks1 - t.ks0; left > 0 && ok; left -= p.xk) {
                        if (!(ok = mbar_wait_hint(x_hint, bar_xfull + 8 * xs, xph, abort_flag))) break;
                        uint32_t xdesc = xdesc0 + xs * ((uint32_t)p.x_stage >> 4);
                        const uint32_t xdone = bar_xempty + 8 * xs;
                        if (++xs == p.nx) { xs = 0; xph ^= 1; }
                        for (int j = min(left, p.xk); j > 0; j -= 2, xdesc += 2 * kunits) {
                            if (!(ok = mbar_wait_hint(a_hint, bar_aready + 4 * as, aph, abort_flag))) break;
                            const uint32_t ta = tmem_a + as * 32, done = bar_aempty + 8 * as;
                            tc_fence_after();
#pragma unroll
                            for (int kk = 0; kk < 4; kk++) {
                                umma_f16_ta<PAIR>(td, ta + 8 * kk, kTaDescHi | (uint64_t)(xdesc + 2 * kk), idesc, more);
                                more = 1;
                            }
                            commit(done);
                            if (j >= 2) {
#pragma unroll
                                for (int kk = 0; kk < 4; kk++)
                                    umma_f16_ta<PAIR>(td, ta + 32 + 8 * kk, kTaDescHi | (uint64_t)(xdesc + kunits + 2 * kk), idesc, 1u);
                            }
                            commit(done + 8);
                            if (j <= 2) commit(xdone);
                            as += 2;
                            if (as == na) { as = 0; aph ^= 1; }
                            a_hint = mbar_test(bar_aready + 4 * as, aph);
                            if (j <= 2) x_hint = mbar_test(bar_xfull + 8 * xs, xph);
                        }
                    }
                }
                if (ok) commit(bar_tfull + 8 * acc);
                acc ^= 1;
                if (acc == 0) tph ^= 1;
            }
        }
    } else if (warp >= 8) {
        // ================= dequantisers =================
        // Group g converts the steps whose number, counted over all items of the CTA, is g modulo GROUPS, a thread per weight row
        // (never by the step's number in its tile: a group that skips the end of a tile would wait on an A stage more than
        // one round ahead, which a phase bit cannot tell from this round). One warp's step is a chain of latencies
        // (barrier, shared-memory round trip, conversion, tensor-memory store and its completion, about 1000 cycles); four
        // groups keep four of them under way.
        const int grp = (warp - 8) >> 2, q = warp & 3;
        const int row = EPI ? (lane >> 4) * 64 + q * 16 + (lane & 15) : q * 32 + lane;  // row of the stage
        const uint32_t sw = row & 7;
        const uint32_t my_a = tmem_a + ((uint32_t)(32 * q) << 16);
        constexpr int SPB = F::SPB;
        const int nash = na == 8 ? 3 : 2;
        uint32_t it0 = 0;     // steps of the items before
        int cs = 0;           // stage of codes
        uint32_t cph = 0;
        bool ok = true;
        Item t;
        for (int n = first; ok && item(n, t); n += stride) {
            const int steps = t.ks1 - t.ks0;  // (t.ks0 is the first step of a stage)
            for (int ch = 0; ch * KPS < steps; ch++) {
                const int j0 = (grp - (int)it0 - ch * KPS) & (GROUPS - 1);  // this group's first step of the stage
                // Every group waits for every stage and hands it back, also those that hold no step of its own (8-bit codes have
                // two steps per stage, for two of the four groups). A group that passed stages over could ask for the next round
                // of one whose first codes had not arrived yet, which a phase bit answers with yes: with an odd number of
                // stages it then converted a stage in flight and counted as its reader one round early.
                ok = __all_sync(0xffffffffu, mbar_wait(bar_cfull + 8 * cs, cph, abort_flag));
                if (!ok) break;
                if (j0 < KPS) {
                    const uint32_t codes = codes0 + cs * kTaCodeStage + row * 128, scales = scales0 + cs * SSTAGE + row * SPB;
#pragma unroll
                    for (int i = 0; i < (KPS + GROUPS - 1) / GROUPS; i++) {
                        const int j = j0 + GROUPS * i;
                        const int ks = ch * KPS + j;
                        if (ks >= steps) break;
                        const uint32_t it = it0 + ks, as = it & (na - 1), aph = (it >> nash) & 1;
                        const uint32_t a_hint = mbar_test(bar_aempty + 8 * as, aph ^ 1);
                        uint32_t sc, bi = 0;
                        if (FMT == kFmtAffine4G32) {
                            sc = lds32(scales + 4 * j);
                            bi = lds32(scales + 128 * SPB + 4 * j);
                        } else {
                            sc = lds_u16(scales + 2 * (FMT == kFmtTernary ? j >> 1 : j));
                            if (F::BIAS) bi = lds_u16(scales + 128 * SPB + 2 * j);
                        }
                        bool small = false;
                        if (FMT == kFmtAffine4) small = __all_sync(0xffffffffu, (sc & 0x7FFFu) < 0x3D80u);
                        if (FMT == kFmtAffine4G32) small = __all_sync(0xffffffffu, (sc & 0x7FFFu) < 0x3D80u && (sc & 0x7FFF0000u) < 0x3D800000u);
                        auto convert = [&](int h, uint32_t (&o)[16]) {
                            // groups of 32 (g32: 16 bits each; mxfp4: 8 bits each) have a scale per half
                            const uint32_t sch = FMT == kFmtAffine4G32 ? sc & 0xFFFFu : (FMT == kFmtMxfp4 ? sc & 0xFFu : sc);
                            ta_dequant32<FMT>(codes, (uint32_t)(j * (F::BPS / 16) + (FMT == kFmtTernary ? 0 : h * (F::BPS / 32))), h, sw, sch,
                                              FMT == kFmtAffine4G32 ? bi & 0xFFFFu : bi, small, o);
                            if (FMT == kFmtAffine4G32) { sc >>= 16; bi >>= 16; }
                            if (FMT == kFmtMxfp4) sc >>= 8;
                        };
                        // Converted before the wait where the registers allow it (not with 64): a stage's turn-around is then a store, not a
                        // conversion
                        uint32_t early[SPLIT ? 2 : 1][16];
                        if constexpr (SPLIT) { convert(0, early[0]); convert(1, early[1]); }
                        ok = __all_sync(0xffffffffu, a_hint || mbar_wait(bar_aempty + 8 * as, aph ^ 1, abort_flag));
                        if (!ok) break;
                        tc_fence_after();
                        if constexpr (SPLIT) {
                            tmem_st16(my_a + as * 32, early[0]);
                            tmem_st16(my_a + as * 32 + 16, early[1]);
                        } else {
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                uint32_t o[16];
                                convert(h, o);
                                tmem_st16(my_a + as * 32 + h * 16, o);
                            }
                        }
                        tmem_st_wait();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            if (PAIR && rank != 0) mbar_arrive_remote_done(bar_aready + 8 * (as / RS), 0);
                            else mbar_arrive(bar_aready + 8 * (as / RS));
                        }
                    }
                    if (!ok) break;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_cempty + 8 * cs);
                if (++cs == p.nc) { cs = 0; cph ^= 1; }
            }
            if (RS == 2 && (steps & 1)) {  // an odd number of steps: the second of the last two A stages holds nothing, but its group reports it
                const uint32_t it = it0 + steps, as = it & (na - 1), aph = (it >> nash) & 1;
                if (ok && (int)(it & (GROUPS - 1)) == grp) {
                    ok = __all_sync(0xffffffffu, mbar_wait(bar_aempty + 8 * as, aph ^ 1, abort_flag));
                    if (ok && lane == 0) {
                        if (PAIR && rank != 0) mbar_arrive_remote_done(bar_aready + 8 * (as / RS), 0);
                        else mbar_arrive(bar_aready + 8 * (as / RS));
                    }
                }
            }
            it0 += (steps + RS - 1) & ~(RS - 1);
        }
    } else {
        // ================= epilogue (warps 4-7) =================
        const int q = warp & 3;
        const int mi = EPI ? lane >> 4 : 0;
        const int nl = EPI ? q * 16 + (lane & 15) : q * 32 + lane;
        int acc = 0;
        uint32_t tph = 0;
        Item t;
        for (int i = first; item(i, t); i += stride) {
            const int rows = t.rows, n = t.n0 + nl;
            const bool n_ok = n < p.N;
            const float* eb = mi ? p.ebias[1] : p.ebias[0];
            const float bias = eb != nullptr && n_ok ? eb[(size_t)t.expert * p.N + n] : 0.f;
            if (!__all_sync(0xffffffffu, mbar_wait(bar_tfull + 8 * acc, tph, abort_flag))) break;
            tc_fence_after();
            const uint32_t td = tmem + acc * p.dcols + ((uint32_t)(32 * q) << 16);
            constexpr int CW = 16;  // token columns at a time
            const int slot = SPLIT && i < sched->np ? sched->piece[i].slot : -1;
            float4* const part = reinterpret_cast<float4*>(p.part) + ((size_t)slot * CTAS + rank) * (ta_slot(p.tile_rows) / 4) + q * (ta_slot(p.tile_rows) / 16) + lane;
            for (int c0 = 0; c0 < rows; c0 += CW) {
                uint32_t r[CW];
                tmem_ld16(td + c0, r);
                tmem_ld_wait();
                if (SPLIT && slot >= 0) {  // a piece: [warp][four columns][lane], 16 bytes each
#pragma unroll
                    for (int j = 0; j < CW / 4; j++)
                        part[(c0 / 4 + j) * 32] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                              __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
                    continue;
                }
                float v[CW];
#pragma unroll
                for (int j = 0; j < CW; j++) v[j] = __uint_as_float(r[j]) + bias;
                if (SPLIT) ta_store<EPI, CW>(p, v, t.row0 + c0, n, n_ok, rows - c0, mi);
                else ta_store_low<EPI, CW>(p, v, t.row0 + c0, n, n_ok, rows - c0, mi);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR && rank != 0) mbar_arrive_remote(bar_tempty + 8 * acc, 0);
                else mbar_arrive(bar_tempty + 8 * acc);
            }
            acc ^= 1;
            if (acc == 0) tph ^= 1;
        }
    }

    __syncwarp();
    // ---- teardown ---------------------------------------------------------------------------------------------------
    if (*abort_flag && (warp == 0 || warp == 2)) {  // copies in flight land before the shared memory is given back
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();  // (the other CTA's MMAs read this one's memory, its arrivals go to this one's barriers)
    if (*abort_flag && threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, kErrTimeout);
    if (warp == 1) {
        tc_fence_after();
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS) : "memory");
    }
}

// Sums of the pieces of the split tiles, behind the GEMM: a warp takes a quarter of a tile's rows and four token columns, 16
// bytes per lane and piece.
template <int EPI>
__global__ void __launch_bounds__(256) ta_sum_kernel(const TaParams p) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int NROWS = EPI ? 64 : 128;
    const int m_tiles = (p.M + p.tile_rows - 1) / p.tile_rows;
    const TaSplit& sp = p.split;
    const int cols = (p.tile_rows + 3) / 4, lane = threadIdx.x & 31;
    const int slot4 = ta_slot(p.tile_rows) / 4;
    const int ctas = p.pair ? 2 : 1, quarters = 4 * ctas;
    for (int w = blockIdx.x * 8 + (threadIdx.x >> 5); w < sp.tiles * cols * quarters; w += gridDim.x * 8) {
        const int q = w & 3, rank = (w % quarters) >> 2, c4 = w / quarters % cols, t = w / quarters / cols;
        const int row0 = (t % m_tiles) * p.tile_rows, rows = min(p.tile_rows, p.M - row0), n0 = ((t / m_tiles) * ctas + rank) * NROWS;
        int a, b, slot0;
        ta_split_tile(sp, t, a, b, slot0);
        if (b - a == 1 || 4 * c4 >= rows) continue;
        const int mi = EPI ? lane >> 4 : 0, n = n0 + (EPI ? q * 16 + (lane & 15) : q * 32 + lane);
        const bool n_ok = n < p.N;
        const float* eb = mi ? p.ebias[1] : p.ebias[0];
        const float bias = eb != nullptr && n_ok ? eb[n] : 0.f;
        const float4* s = reinterpret_cast<const float4*>(p.part) + rank * slot4 + q * (slot4 / 4) + c4 * 32 + lane;
        float4 f[kTaSplitPieces + 2];  // (a run that starts inside the tile's neighbour makes one piece more)
#pragma unroll
        for (int k = 0; k < kTaSplitPieces + 2; k++)
            if (a + k < b) f[k] = s[(size_t)(k == 0 ? slot0 : a + k) * ctas * slot4];
        float v[4] = {f[0].x, f[0].y, f[0].z, f[0].w};
#pragma unroll
        for (int k = 1; k < kTaSplitPieces + 2; k++)
            if (a + k < b) { v[0] += f[k].x; v[1] += f[k].y; v[2] += f[k].z; v[3] += f[k].w; }
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] += bias;
        ta_store<EPI, 4>(p, v, row0 + 4 * c4, n, n_ok, rows - 4 * c4, mi);
    }
}

}  // namespace iq
