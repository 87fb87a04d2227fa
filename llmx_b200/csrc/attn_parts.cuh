// Pieces of the attention kernels whose 32-bit factors meet the tensor cores as three bfloat16 parts.
//
// Their softmax weights are exp2f of a score's distance from the row's maximum (within two units in the last place, like the expf
// of the general forms), subnormal weights among them: the instruction that flushes those gave 0 where the general forms
// give 2^-126 and less (a value of 2^120 makes the difference visible), and was 8 % faster over [key ; value] rows.
#pragma once
#include "attn_common.cuh"

namespace attn {

// Shared-memory operand, MN-major, 128-byte swizzle: 64 elements of the MN dimension contiguous, the next 64 `block` bytes on.
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t addr, uint32_t block) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(block >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Three 8-bit pieces of a float's significand, cut off (not rounded) so that each remainder is exact: a pair of numbers
// becomes three pairs of bfloat16, the first number in the low half.
__device__ __forceinline__ void split3_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
    hi = __byte_perm(ua, ub, 0x7632);
    const float ra = a - __uint_as_float(ua & 0xffff0000u), rb = b - __uint_as_float(ub & 0xffff0000u);
    const uint32_t va = __float_as_uint(ra), vb = __float_as_uint(rb);
    mid = __byte_perm(va, vb, 0x7632);
    lo = __byte_perm(__float_as_uint(ra - __uint_as_float(va & 0xffff0000u)), __float_as_uint(rb - __uint_as_float(vb & 0xffff0000u)), 0x7632);
}

}  // namespace attn

// Host: whether a kernel of `threads` threads a block was given at least `total` registers for 128 threads' worth of them each
// (setmaxnreg hands the block's own registers around: asked for more than it was launched with, it would wait for good).
template <typename K>
static inline bool registers_reach(K kernel, int threads, int total) {
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, kernel) == cudaSuccess && threads / 128 * a.numRegs >= total;
}
