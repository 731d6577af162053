// What decode kernels on tcgen05 integers share: the MMA with the codes as bytes in tensor memory, its descriptors,
// tensor-memory loads and stores, the columns of the activation rows.
#pragma once

#include "ptx.cuh"

namespace iq {

constexpr int kQtCodes = 128 * 128;  // bytes of a stage of codes: 128 bytes of 128 weight rows

// Column of token m among its digit's T columns: the pairs of tokens are dealt to the two groups of warps that finish them
__host__ __device__ constexpr int qt_col(int t, int m) { return ((m >> 1) & 1) * (t / 2) + (m >> 2) * 2 + (m & 1); }

// D[128, N] (s32) (+)= A[128, 32] (u8, tensor memory: lane = row, four inputs per column) * B[N, 32]^T (s8, shared memory)
__device__ __forceinline__ void umma_i8_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n}\n"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void qt_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void qt_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void qt_ld(uint32_t taddr, int (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void qt_ld(uint32_t taddr, int (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
// (the registers pass through the wait, so that no use of them moves above it)
__device__ __forceinline__ void qt_ld_wait(int (&a)[8], int (&b)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]), "+r"(b[0]), "+r"(b[1]),
                   "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7])
                 :
                 : "memory");
}
__device__ __forceinline__ void qt_ld_wait(int (&a)[4], int (&b)[4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3])
                 :
                 : "memory");
}

// K-major operand with the 128-byte swizzle: eight rows of 128 bytes, 1024 bytes from eight to eight
constexpr uint64_t kQtDescHi = ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
// s32 sums, u8 x s8, M = 128
constexpr uint32_t qt_idesc(int n) { return (2u << 4) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (8u << 24); }

}  // namespace iq
