// Floats as sums of bfloat16 terms, for products of 32-bit operands on the tensor cores.
//
// A float has 24 significant bits, a bfloat16 eight and the same range of exponents: the nearest
// bfloat16, the nearest one to what is left and what is left then are three bfloat16 numbers whose
// sum is the float, as long as its last bit is no smaller than bfloat16's smallest (2^-133).  Floats of less
// than 2^-110 have smaller ones (of 1e-36 the terms keep some 14 bits); multiplied by 2^24 first, every
// float up to 2^104 is the sum of its terms, and these are normal numbers.
//
// A product of two floats is then nine products of terms, each exact in float; the three smallest
// (together up to 2^-24 of the product) are left out.  Taking floats apart into bfloat16 terms for
// matrix hardware: Henry, Tang, Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For
// Higher-Precision Computations", ARITH 2019.
#pragma once
#include "common.cuh"
#include "umma_utils.cuh"

namespace {

constexpr float SPLIT_UP = 16777216.f, SPLIT_DOWN = 1.f / 16777216.f;      // 2^24

__device__ __forceinline__ void split_up(float& a, float& b) {
  asm("{\n\t.reg .b64 u, v;\n\t"
      "mov.b64 u, {%0, %1};\n\t"
      "mov.b64 v, {%2, %2};\n\t"
      "mul.rn.f32x2 u, u, v;\n\t"
      "mov.b64 {%0, %1}, u;\n\t}"
      : "+f"(a), "+f"(b)
      : "f"(SPLIT_UP));
}
// (a, b) -> the terms of a in the low halves, those of b in the high halves: hi, mid, lo.
__device__ __forceinline__ uint32_t split_pack(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ void sub2f(float& x, float& y, float a, float b, uint32_t terms) {
  asm("{\n\t.reg .b64 u, v;\n\t"
      "mov.b64 u, {%2, %3};\n\t"
      "mov.b64 v, {%4, %5};\n\t"
      "sub.rn.f32x2 u, u, v;\n\t"
      "mov.b64 {%0, %1}, u;\n\t}"
      : "=f"(x), "=f"(y)
      : "f"(a), "f"(b), "f"(__uint_as_float(terms << 16)), "f"(__uint_as_float(terms & 0xffff0000u)));
}
__device__ __forceinline__ void split3(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  float x, y;
  hi = split_pack(a, b);
  sub2f(x, y, a, b, hi);
  mid = split_pack(x, y);
  sub2f(x, y, x, y, mid);
  lo = split_pack(x, y);
}
// left: gets what is left behind the first terms added up, which is finite exactly where both
// floats have terms.  (Infinities, NaN and the floats above the largest bfloat16 have none: inf - inf.)
__device__ __forceinline__ void split3(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo,
                                       float2& left) {
  float x, y;
  hi = split_pack(a, b);
  sub2f(x, y, a, b, hi);
  add2f(left.x, left.y, x, y);
  mid = split_pack(x, y);
  sub2f(x, y, x, y, mid);
  lo = split_pack(x, y);
}

// K-major operand tile in rows of 64 bytes (32 bfloat16) with the 64-byte swizzle: 8-row groups
// 512 bytes apart.  A row's 16-byte piece p lies at piece p ^ (row / 2 % 4).
__device__ __forceinline__ uint64_t umma_desc_k_sw64(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;                            // leading byte offset (unused here)
  d |= (uint64_t)(512 >> 4) << 32;                   // stride byte offset: 8 rows
  d |= (uint64_t)1 << 46;                            // descriptor version of sm_100
  d |= (uint64_t)4 << 61;                            // SWIZZLE_64B
  return d;
}

}  // namespace
