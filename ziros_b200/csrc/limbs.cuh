// limbs.cuh — field words from the accumulators of 8-bit integer products (tcgen05.cuh): accumulator l of
// an output has weight 2^(8 l).
#pragma once
#include "field.cuh"

namespace zkb {
namespace limbs {

// Largest half of a BabyBear output's accumulators that `babybear` takes.
constexpr uint64_t BABYBEAR_MAX_HALF = (uint64_t)BabyBear::P * 97 / 100;
#ifdef __CUDACC__
// BabyBear: a word congruent to a0 + a1 2^8 + a2 2^16 + a3 2^24 mod p, in [-p, 1.04 p], for u = a0 + a1 2^8 and
// v = a2 + a3 2^8 of at most BABYBEAR_MAX_HALF: q = floor(v * 139810 / 2^32) is at most the true quotient of
// v 2^16 by p (2^32 * 2^16 / p = 139810.13) and less than 1.07 below it, so v 2^16 - (q + 1) p lies in
// [-p, 0.07 p].
__device__ __forceinline__ int babybear(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
  const uint32_t u = a0 + (a1 << 8), v = a2 + (a3 << 8);
  const uint32_t q = __umulhi(v, 139810u) + 1;
  return (int)(u + (v << 16) - q * BabyBear::P);
}

// Goldilocks: e + f 2^32 for e, f < 2^56, some 64-bit representative: f = f0 + f1 2^32 adds
// (f0 + f1) 2^32 - f1.
__device__ __forceinline__ uint64_t goldilocks_join(uint64_t e, uint64_t f) {
  uint32_t l, h;
  asm("{\n\t.reg .u32 x, k;\n\t"
      "add.u32 x, %3, %5;\n\t"
      "sub.cc.u32 %0, %2, %5;\n\tsubc.u32 x, x, 0;\n\t"
      "add.cc.u32 %1, x, %4;\n\taddc.u32 k, 0, 0;\n\t"
      "sub.cc.u32 %0, %0, k;\n\tsubc.u32 %1, %1, 0;\n\tadd.u32 %1, %1, k;\n\t}"
      : "=&r"(l), "=&r"(h)
      : "r"((uint32_t)e), "r"((uint32_t)(e >> 32)), "r"((uint32_t)f), "r"((uint32_t)(f >> 32)));
  return ((uint64_t)h << 32) | l;
}
#endif
// The column of Goldilocks accumulator l among its eight: pairs (0, 2), (1, 3), (4, 6), (5, 7).
__host__ __device__ constexpr int goldilocks_col(int l) {
  return (l & 4) | ((l & 3) == 1 ? 2 : (l & 3) == 2 ? 1 : (l & 3));
}
// Largest sum of a column's operand bytes for which a0 + a1 2^8 stays below 2^32.
constexpr uint32_t MAX_COLUMN = 65500;  // 65500 * 255 * 257 < 2^32
#ifdef __CUDACC__
// The word of eight accumulators in column order.
__device__ __forceinline__ uint64_t goldilocks(const uint32_t *a) {
  const uint32_t u0 = a[0] + (a[2] << 8), v0 = a[1] + (a[3] << 8), u1 = a[4] + (a[6] << 8), v1 = a[5] + (a[7] << 8);
  return goldilocks_join(u0 + ((uint64_t)v0 << 16), u1 + ((uint64_t)v1 << 16));
}
#endif

}  // namespace limbs
}  // namespace zkb
