// fp32 values as three bf16 values that add up to them, for products of fp32 accuracy on bf16 tensor cores.
#pragma once
#include "common.cuh"

// Two consecutive values, times SPLIT_SCALE, as one word of each part: x1 nearest to x, x2 the leading 8 bits of x - x1, x3 the rest, 24 bits of
// significand in all.  The first part, here minus it, comes of a multiplication by 2^16 + 1 and two differences (Dekker's and Veltkamp's splitting: a nearest value of 8
// bits; past 2^111, here 2^87, not finite), in pairs on the FMA pipe: conversions to bf16 are a sixteenth of its rate.  (As fused operations: a
// product and the difference behind it would be fused by the compiler, and the first part not be one.)  The second part is cut off and
// not rounded: behind a nearest first part the signs of the rest are random, and what is cut off is the third part whole.
// The scale costs nothing: the operations apply it, and the first part comes negated instead (a multiplication ahead of them was 2 to 3 % of the
// narrow products, 20000 x 30 x 3000 109.4 -> 111.5 us).  It keeps the third part of every fp32 value, subnormal ones among them, a normal bf16 value (from 2^-125 on), and the small
// products of results that fp32 holds above the accumulators' subnormal range; a sum past 2^79 is not finite.
constexpr float SPLIT_SCALE = 16777216.f, SPLIT_UNSCALE = 1.f / (SPLIT_SCALE * SPLIT_SCALE);   // of an operand; of a sum of products
__device__ __forceinline__ uint64_t split_pair(float a, float b) { return (uint64_t)__float_as_uint(a) | (uint64_t)__float_as_uint(b) << 32; }
__device__ __forceinline__ uint64_t split_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t split_sub2(uint64_t a, uint64_t b) { return split_fma2(b, 0xbf800000bf800000ull, a); }   // a - b
__device__ __forceinline__ uint32_t split_upper(uint64_t v) { return __byte_perm((uint32_t)v, (uint32_t)(v >> 32), 0x7632); }
__device__ __forceinline__ void split2(float a, float b, uint32_t& w1, uint32_t& w2, uint32_t& w3) {
  constexpr float S = SPLIT_SCALE;
  const uint64_t x = split_pair(a, b), t = split_fma2(x, split_pair(65537.f * S, 65537.f * S), 0ull);
  const uint64_t n1 = split_sub2(split_fma2(x, split_pair(-S, -S), t), t), r = split_fma2(x, split_pair(S, S), n1);   // -x1, x - x1
  w1 = split_upper(n1);
  w2 = split_upper(r);
  w3 = split_upper(split_sub2(r, r & 0xffff0000ffff0000ull));
}

// The products that are formed, part of the one operand by part of the other, smallest first.  A second part is up to 2^-8 of its value and a third up to
// 2^-16, so what is left out is below 2^-23 of a product (both at 1 + 2^-8 - 2^-23: 2^-23.03), and 2^-26 of it in the root mean square over random
// values, whose signs are random as well: in sums it grows with the root of their number, as long as the values are no such constants.
constexpr int SPLIT_PRODUCTS = 6;
__host__ __device__ constexpr int split_a(int p) { return p == 0 ? 2 : (p == 2 || p == 3 ? 1 : 0); }   // 2 0 1 1 0 0
__host__ __device__ constexpr int split_b(int p) { return p == 1 ? 2 : (p == 2 || p == 4 ? 1 : 0); }   // 0 2 1 0 1 0
// The first parts come negated: the instruction takes the sign out of a product with one of them (bit 13 of its descriptor: minus A).
__host__ __device__ constexpr uint32_t split_sign(int p) { return (split_a(p) == 0) != (split_b(p) == 0) ? 1u << 13 : 0u; }
