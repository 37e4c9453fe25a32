// Products of matrices of scaled 56-bit integers (fix64.cuh: whole56) on the
// tensor cores, by splitting them into exact products of short numbers (Ozaki, Ogita,
// Oishi, Rump, Numerical Algorithms 59, 2012): an integer is seven signed 8-bit
// digits, each exact in FP16, and of the 49 products of digits those 28 with
// i + j >= 6 are formed.  The products of one weight i + j above 6, summed over up to
// 128 terms, stay within 2^24: FP32 accumulators hold them exactly, whatever the
// order.  Those of weight 6, of which a 256th goes into the result, reach 1.13 2^24
// where all digits are at their limits, and may be rounded to even numbers there.
// What is left out of a term is below 2^-55 of the two scales' product, and 2^-58 of
// it root mean square.  28 FP16 multiply-adds take the place of three 32x32+64-bit
// ones, of which an SM does 25 a clock.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "fix64.cuh"

namespace abx {
namespace dg {

constexpr int MD = fx::DIGITS;
constexpr int MAX_TERMS = 128;  // terms of an exact sum

// Two digits as FP16: 1536 + a as bits, less 1536.
__device__ __forceinline__ __half2 pair(int a, int b) {
  const uint32_t bits = (uint32_t)(0x6600 + a) | (uint32_t)(0x6600 + b) << 16;
  return __hsub2(*reinterpret_cast<const __half2 *>(&bits), __half2half2(__float2half(1536.f)));
}

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                        uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Sums of a warp's 16 x 16 entries by weight (acc[w]: weight MD - 1 + w) with
// digit d of the right operand (two 8-column fragments) for 16 terms.
__device__ __forceinline__ void multiply(float (&acc)[MD][2][4], const uint32_t (&a)[MD][4],
                                         const uint32_t (&b)[4], int d) {
#pragma unroll
  for (int i = 0; i < MD; ++i) {
    if (i + d < MD - 1) continue;
    mma_f16(acc[i + d - (MD - 1)][0], a[i], b[0], b[1]);
    mma_f16(acc[i + d - (MD - 1)][1], a[i], b[2], b[3]);
  }
}
// An entry's sum in units of 2^56: weights 7 to 12, and 6 rounded.
__device__ __forceinline__ long long sum(const float (&acc)[MD][2][4], int c, int q) {
  long long s = (long long)__float2int_rn(acc[MD - 1][c][q]);
#pragma unroll
  for (int w = MD - 2; w > 0; --w) s = s * 256 + __float2int_rn(acc[w][c][q]);
  return s + ((__float2int_rn(acc[0][c][q]) + 128) >> 8);
}

}  // namespace dg
}  // namespace abx
