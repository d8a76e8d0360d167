// mbarriers, bulk copies, the 5th-generation tensor core and pairs of halves in PTX: what mm_id.cu, mv_dense.cu and route_filter.cu share.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace {

constexpr int MM_WAIT_HINT_NS = 1000, MM_WAIT_TRIES = 1 << 22;

__device__ __forceinline__ uint32_t s32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mb_init(uint64_t *b, uint32_t c) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(b)), "r"(c));
}
__device__ __forceinline__ void mb_arrive(uint64_t *b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(b)) : "memory");
}
__device__ __forceinline__ void mb_expect_tx(uint64_t *b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(b)), "r"(bytes) : "memory");
}
// Bounded wait.  The loop is one piece of assembly: no branch that the compiler sees separates the values a warp has
// computed from the store that follows the wait.  Each try waits inside the hardware for up to the hint before it answers
// (without one a waiting warp asks again every few dozen cycles and takes issue slots from the converting ones), so the
// limit is a few seconds.  Returns false when it runs out; mm_timeout() records that.
__device__ __forceinline__ bool mb_wait(uint64_t *b, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p, q;\n\t.reg .b32 n;\n\tmov.b32 n, 0;\n"
                 "W%=:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t@p bra D%=;\n\t"
                 "add.u32 n, n, 1;\n\tsetp.lt.u32 q, n, %4;\n\t@q bra W%=;\n"
                 "D%=:\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(s32(b)), "r"(parity), "n"(MM_WAIT_HINT_NS), "n"(MM_WAIT_TRIES) : "memory");
    return ok != 0;
}
// Whether that phase is over, without waiting.
__device__ __forceinline__ bool mb_test(uint64_t *b, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(s32(b)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(s32(dst)),
                 "l"(src), "r"(bytes), "r"(s32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Arrives, once the multiplies issued so far are done, at the barrier at this place in both CTAs of the pair.
template <int CG>
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    if (CG == 1) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(bar)) : "memory");
    else asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(s32(bar)),
                 "h"((uint16_t)3) : "memory");
}
// 16 columns of the warp's 32 tensor-memory lanes; the registers hold the values after tc_wait_ld()
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tc_ld4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// One lane of a converged warp, chosen by the hardware: code under this predicate is known to be single-lane.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(p));
    return p != 0;
}

// K-major, 128-byte-swizzled operand tile: rows of 64 f16 (128 B); groups of 8 rows are 1024 B apart; the 16-byte
// chunk c of row r sits at chunk position c ^ (r % 8).
// Shared-memory matrix descriptor of such a tile (start address advanced by 32 B per K=16 step).
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    const uint64_t lo = (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16);           // LBO (unused) = 16 B
    const uint64_t hi = (uint64_t)(1024 >> 4) | ((uint64_t)1 << 14) | ((uint64_t)2 << 29);   // SBO 1024 B, version 1, SWIZZLE_128B
    return lo | (hi << 32);
}

// (v & mask) | magic in one instruction, which it is not when written in C
__device__ __forceinline__ uint32_t and_or(uint32_t v, uint32_t mask, uint32_t magic) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(v), "r"(mask), "r"(magic));
    return r;
}
// f16 pairs
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}

} // namespace
