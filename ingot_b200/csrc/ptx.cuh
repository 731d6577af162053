// PTX wrappers shared by the TMA / mbarrier / tcgen05 kernels (sm_100a).
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace iq {

constexpr uint64_t kWaitCycles = 4000000000ull;  // bound of every device-side wait: about two seconds

// One lane of a converged warp. Tensor copies and tcgen05 instructions take their operands from uniform registers: under
// `if (lane == 0)` the compiler cannot know that one lane is active and wraps every one of them in a loop over the active
// lanes (125 cycles per tcgen05.mma measured, whatever its size); under this predicate it issues them directly (30).
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
    return r != 0;
}

// ---- PTX wrappers ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait. Returns false when the wait gave up or another role already did.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if ((unsigned long long)(clock64() - t0) > kWaitCycles) {
            *abort_flag = 1;
            return false;
        }
    }
}
// A look at a barrier without waiting, for software pipelining: asked early, its latency (about 100 cycles) passes under the
// instructions that follow, and mbar_wait_hint only waits when the answer was no. The wait spins on test_wait: a try_wait
// that finds the phase open sleeps in steps of about 250 cycles.
__device__ __forceinline__ uint32_t mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}
__device__ __forceinline__ bool mbar_wait_hint(uint32_t hint, uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (hint) return true;
    const long long t0 = clock64();
    while (true) {
        if (mbar_test(bar, parity)) return true;
        if (*abort_flag) return false;
        if ((unsigned long long)(clock64() - t0) > kWaitCycles) {
            *abort_flag = 1;
            return false;
        }
    }
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
// D[128, N] (s32) (+)= A[128, 32] * B[N, 32]^T on signed 8-bit operands
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
        "%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }


// Shared-memory loads by 32-bit shared address.
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 r;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(a));
    return r;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 r;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(a));
    return r;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t r;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(a));
    return r;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
    unsigned short r;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(r) : "r"(a));
    return r;
}
__device__ __forceinline__ uint32_t lds_u8(uint32_t a) {
    uint32_t r;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(r) : "r"(a));
    return r;
}

// Two fp32 operations per instruction, each rounded as fmaf and a product are (the grouped int8 kernel, where its registers allow it; no
// effect in the dense GEMVs): {a0, a1} += {v0, v1} * ({s0, s1} * {x0, x1}), and then
// += {b0, b1} * {y0, y1}.
__device__ __forceinline__ void scaled_add2(float& a0, float& a1, float v0, float v1, float s0, float s1, float x0, float x1) {
    asm("{\n.reg .b64 a, v, s, x;\nmov.b64 a, {%0, %1};\nmov.b64 v, {%2, %3};\nmov.b64 s, {%4, %5};\nmov.b64 x, {%6, %7};\n"
        "mul.rn.f32x2 s, s, x;\nfma.rn.f32x2 a, v, s, a;\nmov.b64 {%0, %1}, a;\n}\n"
        : "+f"(a0), "+f"(a1)
        : "f"(v0), "f"(v1), "f"(s0), "f"(s1), "f"(x0), "f"(x1));
}
// {a0, a1} = {v0, v1} * (s * {x0, x1}), rounded as scaled_add2 on zeros
__device__ __forceinline__ void scaled_mul2(float& a0, float& a1, float v0, float v1, float s, float x0, float x1) {
    asm("{\n.reg .b64 a, v, s, x;\nmov.b64 v, {%2, %3};\nmov.b64 s, {%4, %4};\nmov.b64 x, {%5, %6};\nmul.rn.f32x2 s, s, x;\nmul.rn.f32x2 a, v, s;\nmov.b64 {%0, %1}, a;\n}\n"
        : "=f"(a0), "=f"(a1)
        : "f"(v0), "f"(v1), "f"(s), "f"(x0), "f"(x1));
}
// ... and {l0, l1} += {w0, w1} * that product, for a lower digit
__device__ __forceinline__ void scaled_add2_low(float& a0, float& a1, float& l0, float& l1, float v0, float v1, float w0, float w1, float s, float x0, float x1) {
    asm("{\n.reg .b64 a, l, v, w, s, x;\nmov.b64 a, {%0, %1};\nmov.b64 l, {%2, %3};\nmov.b64 v, {%4, %5};\nmov.b64 w, {%6, %7};\nmov.b64 s, {%8, %8};\n"
        "mov.b64 x, {%9, %10};\nmul.rn.f32x2 s, s, x;\nfma.rn.f32x2 a, v, s, a;\nfma.rn.f32x2 l, w, s, l;\nmov.b64 {%0, %1}, a;\nmov.b64 {%2, %3}, l;\n}\n"
        : "+f"(a0), "+f"(a1), "+f"(l0), "+f"(l1)
        : "f"(v0), "f"(v1), "f"(w0), "f"(w1), "f"(s), "f"(x0), "f"(x1));
}
__device__ __forceinline__ void fma2(float& a0, float& a1, float b0, float b1, float y0, float y1) {
    asm("{\n.reg .b64 a, b, y;\nmov.b64 a, {%0, %1};\nmov.b64 b, {%2, %3};\nmov.b64 y, {%4, %5};\nfma.rn.f32x2 a, b, y, a;\nmov.b64 {%0, %1}, a;\n}\n"
        : "+f"(a0), "+f"(a1)
        : "f"(b0), "f"(b1), "f"(y0), "f"(y1));
}

// 1-D bulk copy global -> shared memory, completion counted in bytes on an mbarrier (no multicast).
// Both addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// Asynchronous copy of 4, 8 or 16 bytes global -> shared memory through L1 (neighbouring pieces of the line follow), and the
// arrival that an mbarrier receives once all of this thread's copies issued so far have landed (.noinc: it counts as one
// of the barrier's expected arrivals).
template <int BYTES>
__device__ __forceinline__ void cp_async_ca(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_cg16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// four bytes of which the first n are copied, the others zero
__device__ __forceinline__ void cp_async4_zfill(uint32_t dst, const void* src, int n) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_arrive_noinc(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// Programmatic dependent launch: let the next kernel in the stream start its independent prologue, and wait for the
// previous kernel's results before touching anything it may have written. Both are no-ops without the launch attribute.
// A kernel may let its successor start before it has waited for its own predecessor, and the successor may then read what neither
// of the two writes: weights (codes, scales, biases) are read ahead of the wait by the GEMVs and the dense GEMM. So a kernel that writes
// weights lets nothing start early (of this library's, the W8A8 conversions; anybody else's copy or kernel without the trigger is as good:
// the first kernel behind it starts when it has ended, and all later ones after that).
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- pairs of CTAs (tcgen05 with cta_group::2): the even CTA of a cluster of two issues for both -------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// arrival on the barrier at the same shared-memory offset of the cluster's CTA `cta`
__device__ __forceinline__ void mbar_arrive_remote(uint32_t bar, uint32_t cta) {
    asm volatile("{\n.reg .b32 r;\nmapa.shared::cluster.u32 r, %0, %1;\nmbarrier.arrive.release.cluster.shared::cluster.b64 _, [r];\n}\n" ::"r"(bar), "r"(cta)
                 : "memory");
}
// Tensor copy into this CTA's shared memory whose bytes count on the barrier at this offset of the pair's even CTA
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
    asm volatile(
        "{\n.reg .b32 r;\nmapa.shared::cluster.u32 r, %2, 0;\n"
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [r];\n}\n"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
// ... without the ordering of memory at cluster scope, which makes the thread wait for all it has under way: for what is complete
// already (tensor memory behind tcgen05.wait)
__device__ __forceinline__ void mbar_arrive_remote_done(uint32_t bar, uint32_t cta) {
    asm volatile("{\n.reg .b32 r;\nmapa.shared::cluster.u32 r, %0, %1;\nmbarrier.arrive.shared::cluster.b64 _, [r];\n}\n" ::"r"(bar), "r"(cta) : "memory");
}
// completion of all tcgen05.mma issued so far, to the barrier at this offset in both CTAs
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3)
                 : "memory");
}

// ---- thread-block clusters ------------------------------------------------------------------------------------------
// barrier over all threads of the cluster, with release/acquire ordering of shared-memory writes
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// float64 at the same shared-memory offset as `p` in the block with rank `cta` of this cluster
__device__ __forceinline__ double ld_dsmem_f64(const double* p, uint32_t cta) {
    const uint32_t local = static_cast<uint32_t>(__cvta_generic_to_shared(p));
    uint32_t remote;
    double v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(cta));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote) : "memory");
    return v;
}

// a word stored at the same shared-memory offset as `p` in the block with rank `cta` of this cluster
__device__ __forceinline__ void st_dsmem_u32(uint32_t* p, uint32_t cta, uint32_t v) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(cta));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(v) : "memory");
}

__device__ __forceinline__ void st_dsmem_u64(unsigned long long* p, uint32_t cta, unsigned long long v) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(cta));
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote), "l"(v) : "memory");
}

}  // namespace iq
