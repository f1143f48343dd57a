// Float32 operands on the tensor cores: numbers as sums of three bfloat16 numbers, and what their kernels (gemm_f32_tc.cu,
// attention_f32_tc.cu) need of barriers, tensor memory and tcgen05.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace ps {
namespace f32tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return done != 0;
}
__device__ __forceinline__ uint64_t global_timer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
constexpr uint64_t WAIT_LIMIT_NS = 200ull * 1000 * 1000;         // 0.2 s: far beyond any legitimate wait here
// false: the wait ran out, or another thread of this CTA gave up (abort flag set)
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t start = global_timer_ns();
    while (true) {
#pragma unroll 1
        for (int spin = 0; spin < 64; ++spin)
            if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (global_timer_ns() - start > WAIT_LIMIT_NS) { *abort_flag = 1; return false; }
    }
}
__device__ __forceinline__ bool elect_one() {
    uint32_t chosen;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(chosen));
    return chosen != 0;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
// K-major operand tile with 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
    uint64_t desc = (uint64_t)((smem_addr >> 4) & 0x3FFF);
    desc |= (uint64_t)1 << 16;                     // leading byte offset (unused with swizzle), 16-byte units
    desc |= (uint64_t)(1024 >> 4) << 32;           // stride byte offset between 8-row groups
    desc |= (uint64_t)1 << 46;                     // descriptor version of sm_100
    desc |= (uint64_t)2 << 61;                     // SWIZZLE_128B
    return desc;
}
// first operand from tensor memory: a row per lane, two neighbouring k's per column
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Two numbers as three pairs of bfloat16 numbers that add up to them: exactly from 2^-110 on; of a smaller one the third piece loses what is
// below 2^-133, the smallest bfloat16 number.  The first pieces are cut off, not rounded (a number near the largest float would round to an
// infinity); what is left has 16 bits, the second pieces are rounded to 8 of them, with what is left then of 8 bits and either sign: the terms
// that the products leave out have no sign in common.  A second piece is at most 2^-7 of its number's power of two, a third one 2^-16, so
// that those terms (second by third and third by third) are below 2^-22 of a product (the worst found is 3.9 * 2^-24).
__device__ __forceinline__ void split(float x, float y, uint32_t& first, uint32_t& second, uint32_t& third) {
    const unsigned long long minus = pair_of(-1.f, -1.f);
    const uint32_t ux = __float_as_uint(x), uy = __float_as_uint(y);
    first = __byte_perm(ux, uy, 0x7632);
    unsigned long long rest = pair_fma(pair_of(__uint_as_float(ux & 0xffff0000u), __uint_as_float(uy & 0xffff0000u)), minus, pair_of(x, y));
    pair_split(rest, x, y);
    const __nv_bfloat162 rounded = __floats2bfloat162_rn(x, y);
    second = *reinterpret_cast<const uint32_t*>(&rounded);
    rest = pair_fma(pair_of(__uint_as_float(second << 16), __uint_as_float(second & 0xffff0000u)), minus, rest);
    pair_split(rest, x, y);
    third = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
}

// Whether a result has to be formed again term by term: one that is not finite (an infinity or a NaN among the operands, or an overflow), and one
// so small that the third pieces behind it may have lost bits (products of numbers below 2^-110 by ones up to 2^19, sums of up to 2^11 of them;
// on their own such sums were up to 1.4e-4 off at 2^-122, and from 2^-114 down further than multiply-adds).
__device__ __forceinline__ bool doubtful(float v) {
    const float size = fabsf(v);
    return !(size <= 3.402823466e38f) || (size < 8.2718061e-25f /* 2^-80 */ && size > 0.f);
}

}  // namespace f32tc
}  // namespace ps
