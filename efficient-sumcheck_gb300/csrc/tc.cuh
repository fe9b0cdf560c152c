// tc.cuh -- what the tensor-core passes share: tcgen05 instructions, operand
// descriptors, and exact integer products from 8-bit floats.
//
// A 64-bit word is sixteen 4-bit digits.  As the low bits of an e4m3 byte a
// digit n in 0..15 is the number n 2^-9 (0..7 subnormal, 8..15 normal with the
// smallest exponent), so splitting a word takes a mask and a shift, no
// conversion.  A product of two digits is below 225 in units of 2^-18, and a
// float accumulator of such sums is exact below 2^24 of them: 74565 terms.
// A chunk is a word's sixteen digit bytes: the low digits of bytes 0..7, then
// the high digits (digit e < 8 weighs 16^(2 e), digit 8 + b 16^(2 b + 1)).
#pragma once
#include "round_common.cuh"

namespace effsc {

__device__ __forceinline__ uint4 digits_of(u64 v) {
    const u32 w0 = (u32)v, w1 = (u32)(v >> 32), m = 0x0F0F0F0Fu;
    return make_uint4(w0 & m, w1 & m, (w0 >> 4) & m, (w1 >> 4) & m);
}
// 128-byte rows with the 128-byte swizzle: chunk c of row r.
__device__ __forceinline__ u32 swz128(u32 row, u32 chunk) { return row * 128 + ((chunk ^ (row & 7)) << 4); }

// Shared-memory matrix descriptor: start address, both strides (bytes between
// 8-row groups / between 128-byte wide atoms; the operands here are one atom
// wide, so only one is used), 128-byte swizzle.
__device__ __forceinline__ u64 tc_desc(u32 addr, u32 stride) {
    const u64 s = stride >> 4;
    return (u64)((addr & 0x3FFFF) >> 4) | (s << 16) | (s << 32) | (1ULL << 46) | (2ULL << 61);
}
// Instruction descriptor of kind::f8f6f4, e4m3 x e4m3 -> f32 (mn: both
// operands stored with the M / N index contiguous, else K).
__host__ __device__ constexpr u32 tc_idesc(u32 m, u32 n, bool mn) {
    return (1u << 4) | (mn ? (1u << 15) | (1u << 16) : 0u) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
__device__ __forceinline__ void tc_mma_f8(u32 d, u64 a, u64 b, u32 idesc, u32 accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrive on `bar` when every MMA issued so far by this thread has finished.
__device__ __forceinline__ void tc_commit(u64* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Tensor memory, by one whole warp.
__device__ __forceinline__ void tc_alloc(u32* slot, u32 cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(u32 addr, u32 cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 16 columns of this warp's 32 tensor-memory lanes.
__device__ __forceinline__ void tc_ld16(float (&f)[16], u32 addr) {
    u32 r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
#pragma unroll
    for (int i = 0; i < 16; i++) f[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(u64* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

}  // namespace effsc
