// A float32 in three bfloat16 for products on the tensor cores (gemm_f32_tc.cuh, chunk_mma.cuh):
//
//   a = a0 + a1 + a2,   a0 = a rounded to 8 bits, a1 = the rest rounded to 8 bits, a2 = what is left (7 bits),
//
// and the product of two is the sum of six products of parts, a0 b0, a0 b1, a1 b0, a1 b1, a0 b2, a2 b0.  The three left out, a1 b2,
// a2 b1 and a2 b2, are at most 2^-24 of a b (|a1| <= 2^-8 |a|, |a2| <= 2^-17 |a|), half of the last bit that float32 keeps of it; over
// normally distributed operands their root mean square is 2^-27.4.  (With a0 cut off instead of rounded 2^-22 and 2^-25.4.)
//
// The sum of the parts is a exactly for 2^-110 <= |a|; below, the third and then the second part fall under bfloat16's smallest
// values, and what is lost is at most 2^-134 (the tensor cores take subnormal operands as they are): sums of 512 products with values
// around 2^-110 are off by 0.9e-7 of their norm, 2^-112 1.7e-7, 2^-116 2.2e-6, 2^-120 3.5e-5, where multiply-adds are by 1.2e-7.  Beyond bfloat16's largest value a0 is that value, and a0 b0 may overflow where a b is within 2^-7 of
// float32's largest value.  The parts of infinities and NaN sum up to NaN.
#pragma once
#include "common.cuh"

// The pairs of parts of two values, a in the lower half of each.
__device__ __forceinline__ void bf16_parts(float a, float b, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    auto pack = [](float x, float y) -> uint32_t {
        const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
        return *reinterpret_cast<const uint32_t*>(&v);
    };
    auto below = [](float x) -> float {   // x, or bfloat16's largest value with x's sign
        float r;
        asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(__uint_as_float(0x7f7f0000u)));
        return r;
    };
    p0 = pack(below(a), below(b));
    const float ra = a - __uint_as_float(p0 << 16), rb = b - __uint_as_float(p0 & 0xffff0000u);   // exact: 16 bits
    p1 = pack(ra, rb);
    p2 = pack(ra - __uint_as_float(p1 << 16), rb - __uint_as_float(p1 & 0xffff0000u));            // exact: 7 bits
}
