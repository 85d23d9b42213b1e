// Fifth-generation tensor core (tcgen05) and asynchronous-copy building blocks of the token-row kernels: shared-memory descriptors,
// commits and fences, reads of tensor memory as packed pairs, packed float arithmetic, 16-byte copies that arrive on an mbarrier,
// bounded waits.
#pragma once
#include "brrr_dev.cuh"
#include "brrr_tma.cuh"

namespace brrr {

// shared-memory matrix descriptor: K-major, no swizzle; core matrix = 8 rows x 16 bytes, `sbo` bytes apart along M/N (stride byte
// offset), `lbo` bytes apart along K (leading byte offset)
__device__ __forceinline__ uint64_t tl_smem_desc(const void *p, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_u32(p) >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;                      // descriptor version of this architecture
    return d;
}
// The barrier's phase completes with the products that the lanes with issue != 0 have issued so far.  A predicate: an issuing warp whose instructions carry its elected lane's predicate, instead of standing in a one-lane branch,
// keeps a uniform loop and its descriptors and addresses in uniform registers, where these instructions want them.
__device__ __forceinline__ void tl_commit_if(uint32_t issue, uint64_t *bar) {
    asm volatile("{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %1, 0;\n\t@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)), "r"(issue) : "memory");
}
__device__ __forceinline__ void tl_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tl_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// packed pairs of floats
typedef unsigned long long f32x2;
// Two runs of consecutive columns (32-bit floats) of this warp's 32 lanes of tensor memory as pairs, one wait.  Loads, wait and
// packing are one statement, so nothing can use a register before the wait.
__device__ __forceinline__ void tl_ld16x2(uint32_t ta, uint32_t tb, f32x2 (&v)[8], f32x2 (&w)[8]) {
    asm volatile("{\n\t.reg .b32 r<16>;\n\t.reg .b32 s<16>;\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x16.b32 {r0,r1,r2,r3,r4,r5,r6,r7,r8,r9,r10,r11,r12,r13,r14,r15}, [%16];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x16.b32 {s0,s1,s2,s3,s4,s5,s6,s7,s8,s9,s10,s11,s12,s13,s14,s15}, [%17];\n\t"
                 "tcgen05.wait::ld.sync.aligned;\n\t"
                 "mov.b64 %0, {r0,r1};\n\tmov.b64 %1, {r2,r3};\n\tmov.b64 %2, {r4,r5};\n\tmov.b64 %3, {r6,r7};\n\t"
                 "mov.b64 %4, {r8,r9};\n\tmov.b64 %5, {r10,r11};\n\tmov.b64 %6, {r12,r13};\n\tmov.b64 %7, {r14,r15};\n\t"
                 "mov.b64 %8, {s0,s1};\n\tmov.b64 %9, {s2,s3};\n\tmov.b64 %10, {s4,s5};\n\tmov.b64 %11, {s6,s7};\n\t"
                 "mov.b64 %12, {s8,s9};\n\tmov.b64 %13, {s10,s11};\n\tmov.b64 %14, {s12,s13};\n\tmov.b64 %15, {s14,s15};\n\t"
                 "}"
                 : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]), "=l"(v[4]), "=l"(v[5]), "=l"(v[6]), "=l"(v[7]), "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3]), "=l"(w[4]), "=l"(w[5]), "=l"(w[6]), "=l"(w[7])
                 : "r"(ta), "r"(tb)
                 : "memory");
}
__device__ __forceinline__ void tl_ld8x2(uint32_t ta, uint32_t tb, f32x2 (&v)[4], f32x2 (&w)[4]) {
    asm volatile("{\n\t.reg .b32 r<8>;\n\t.reg .b32 s<8>;\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {r0,r1,r2,r3,r4,r5,r6,r7}, [%8];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {s0,s1,s2,s3,s4,s5,s6,s7}, [%9];\n\t"
                 "tcgen05.wait::ld.sync.aligned;\n\t"
                 "mov.b64 %0, {r0,r1};\n\tmov.b64 %1, {r2,r3};\n\tmov.b64 %2, {r4,r5};\n\tmov.b64 %3, {r6,r7};\n\t"
                 "mov.b64 %4, {s0,s1};\n\tmov.b64 %5, {s2,s3};\n\tmov.b64 %6, {s4,s5};\n\tmov.b64 %7, {s6,s7};\n\t"
                 "}"
                 : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]), "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                 : "r"(ta), "r"(tb)
                 : "memory");
}
// four chains (`step` columns apart) x two blocks (8 apart): the first two or four columns of each, v[2 chain + block]
__device__ __forceinline__ void tl_ld_blocks(uint32_t ta, uint32_t step, f32x2 (&v)[8][1]) {
    asm volatile("{\n\t.reg .b32 r0_<2>;\n\t.reg .b32 r1_<2>;\n\t.reg .b32 r2_<2>;\n\t.reg .b32 r3_<2>;\n\t.reg .b32 r4_<2>;\n\t.reg .b32 r5_<2>;\n\t.reg .b32 r6_<2>;\n\t.reg .b32 r7_<2>;\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x2.b32 {r0_0,r0_1}, [%8];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x2.b32 {r1_0,r1_1}, [%9];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x2.b32 {r2_0,r2_1}, [%10];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x2.b32 {r3_0,r3_1}, [%11];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x2.b32 {r4_0,r4_1}, [%12];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x2.b32 {r5_0,r5_1}, [%13];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x2.b32 {r6_0,r6_1}, [%14];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x2.b32 {r7_0,r7_1}, [%15];\n\t"
                 "tcgen05.wait::ld.sync.aligned;\n\t"
                 "mov.b64 %0, {r0_0,r0_1};\n\tmov.b64 %1, {r1_0,r1_1};\n\tmov.b64 %2, {r2_0,r2_1};\n\tmov.b64 %3, {r3_0,r3_1};\n\tmov.b64 %4, {r4_0,r4_1};\n\tmov.b64 %5, {r5_0,r5_1};\n\tmov.b64 %6, {r6_0,r6_1};\n\tmov.b64 %7, {r7_0,r7_1};\n\t"
                 "}"
                 : "=l"(v[0][0]), "=l"(v[1][0]), "=l"(v[2][0]), "=l"(v[3][0]), "=l"(v[4][0]), "=l"(v[5][0]), "=l"(v[6][0]), "=l"(v[7][0])
                 : "r"(ta + 0 * step + 0), "r"(ta + 0 * step + 8), "r"(ta + 1 * step + 0), "r"(ta + 1 * step + 8), "r"(ta + 2 * step + 0), "r"(ta + 2 * step + 8), "r"(ta + 3 * step + 0), "r"(ta + 3 * step + 8)
                 : "memory");
}
__device__ __forceinline__ void tl_ld_blocks(uint32_t ta, uint32_t step, f32x2 (&v)[8][2]) {
    asm volatile("{\n\t.reg .b32 r0_<4>;\n\t.reg .b32 r1_<4>;\n\t.reg .b32 r2_<4>;\n\t.reg .b32 r3_<4>;\n\t.reg .b32 r4_<4>;\n\t.reg .b32 r5_<4>;\n\t.reg .b32 r6_<4>;\n\t.reg .b32 r7_<4>;\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r0_0,r0_1,r0_2,r0_3}, [%16];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r1_0,r1_1,r1_2,r1_3}, [%17];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r2_0,r2_1,r2_2,r2_3}, [%18];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r3_0,r3_1,r3_2,r3_3}, [%19];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r4_0,r4_1,r4_2,r4_3}, [%20];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r5_0,r5_1,r5_2,r5_3}, [%21];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r6_0,r6_1,r6_2,r6_3}, [%22];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r7_0,r7_1,r7_2,r7_3}, [%23];\n\t"
                 "tcgen05.wait::ld.sync.aligned;\n\t"
                 "mov.b64 %0, {r0_0,r0_1};\n\tmov.b64 %1, {r0_2,r0_3};\n\tmov.b64 %2, {r1_0,r1_1};\n\tmov.b64 %3, {r1_2,r1_3};\n\tmov.b64 %4, {r2_0,r2_1};\n\tmov.b64 %5, {r2_2,r2_3};\n\tmov.b64 %6, {r3_0,r3_1};\n\tmov.b64 %7, {r3_2,r3_3};\n\tmov.b64 %8, {r4_0,r4_1};\n\tmov.b64 %9, {r4_2,r4_3};\n\tmov.b64 %10, {r5_0,r5_1};\n\tmov.b64 %11, {r5_2,r5_3};\n\tmov.b64 %12, {r6_0,r6_1};\n\tmov.b64 %13, {r6_2,r6_3};\n\tmov.b64 %14, {r7_0,r7_1};\n\tmov.b64 %15, {r7_2,r7_3};\n\t"
                 "}"
                 : "=l"(v[0][0]), "=l"(v[0][1]), "=l"(v[1][0]), "=l"(v[1][1]), "=l"(v[2][0]), "=l"(v[2][1]), "=l"(v[3][0]), "=l"(v[3][1]), "=l"(v[4][0]), "=l"(v[4][1]), "=l"(v[5][0]), "=l"(v[5][1]), "=l"(v[6][0]), "=l"(v[6][1]), "=l"(v[7][0]), "=l"(v[7][1])
                 : "r"(ta + 0 * step + 0), "r"(ta + 0 * step + 8), "r"(ta + 1 * step + 0), "r"(ta + 1 * step + 8), "r"(ta + 2 * step + 0), "r"(ta + 2 * step + 8), "r"(ta + 3 * step + 0), "r"(ta + 3 * step + 8)
                 : "memory");
}
__device__ __forceinline__ f32x2 tl_pack2(uint32_t lo, uint32_t hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ void tl_unpack2(f32x2 v, float &lo, float &hi) {
    uint32_t a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v));
    lo = __uint_as_float(a); hi = __uint_as_float(b);
}
__device__ __forceinline__ f32x2 tl_fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 tl_mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 tl_add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void lds_pairs(uint32_t addr, f32x2 &a, f32x2 &b) { asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr)); }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Waits of the pipeline loops: a probe that suspends in hardware, a bounded number of times (far above any copy or product, well
// under a second); when it runs out the error word is set and this thread does not wait again.  No call and no clock: a function
// call in the loop would force every accumulator through the calling convention's registers (80 moves per pair and warp).
constexpr int TL_WAIT_TRIES = 1 << 17;
struct TlWaiter {
    uint32_t *err;
    bool dead;
    __device__ __forceinline__ void operator()(uint64_t *bar, uint32_t parity) {
        if (dead || mbar_test_wait(bar, parity)) return;
        for (int i = 0; !mbar_try_wait_hint(bar, parity, 20000u);)
            if (++i == TL_WAIT_TRIES) {
                dead = true;
                if (err) atomicCAS(err, (uint32_t)DEV_ERR_NONE, (uint32_t)DEV_ERR_COPY_TIMEOUT);
                break;
            }
    }
};

}  // namespace brrr
