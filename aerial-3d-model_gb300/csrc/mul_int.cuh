// Exact FP64 products in integer instructions.
//
// On this GPU an FP64 warp instruction occupies its SM sub-partition's FP64
// pipe for about 64 cycles, in which the same sub-partition issues 64 integer
// instructions.  A kernel bound by that pipe takes part of its products off
// it: the product of two normal doubles, rounded to nearest, ties to even, is
// the 106-bit product of the significands (four 32 x 32 -> 64-bit
// multiplications), normalised and rounded, some 35 instructions.  The result
// is the one of __dmul_rn, bit for bit, whenever both factors are in
// mul_safe's range, where neither they nor the product can be zero,
// subnormal, infinite or NaN.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define BA_MUL_FN __host__ __device__ __forceinline__
#else
#define BA_MUL_FN inline  // (also compiled by the host's compiler for its test)
#endif

namespace ba {

// Exponent field 512 .. 1532: the product's is 1 .. 2042.
BA_MUL_FN bool mul_safe_hi(uint32_t hi) {
  return hi * 2u - (512u << 21) < (1021u << 21);
}

// A factor: its significand in the upper 53 of 64 bits, and sign and exponent
// as two of them add up to those of the product's high word, less the leading
// bit that the significand adds there (the exponent less 512).
struct MulOp {
  uint32_t m1, m0, e;
};
BA_MUL_FN MulOp mul_op_bits(uint32_t hi, uint32_t lo) {
  return MulOp{0x80000000u | (hi << 11) | (lo >> 21), lo << 11,
               (hi & 0xfff00000u) - (512u << 20)};
}

// The bits of the product a * b.
BA_MUL_FN uint64_t mul_bits(const MulOp& a, const MulOp& b) {
  const uint64_t w = (uint64_t)a.m0 * b.m0;
  const uint64_t x = (uint64_t)a.m1 * b.m0 + (w >> 32);
  const uint64_t y = (uint64_t)a.m0 * b.m1 + (uint32_t)x;
  const uint64_t z = (uint64_t)a.m1 * b.m1 + (x >> 32) + (y >> 32);
  const uint32_t z1 = (uint32_t)(z >> 32), z0 = (uint32_t)z;
  const uint32_t n = z1 >> 31;  // the significands' product is 2 or more
  const uint32_t sticky = ((uint32_t)y | (uint32_t)w) != 0u ? 1u : 0u;
  const uint32_t rest = (z0 << (22 - n)) | sticky;  // what is cut off, over 2^32
  const uint64_t m = z >> (10 + n);                 // 53 bits, the leading one included
  const uint32_t up = rest + ((uint32_t)m & 1u) > 0x80000000u ? 1u : 0u;
  const uint32_t head = a.e + b.e + (n << 20);
  return m + up + ((uint64_t)head << 32);
}

#ifdef __CUDACC__
__device__ __forceinline__ bool mul_safe(double x) {
  return mul_safe_hi((uint32_t)__double2hiint(x));
}
__device__ __forceinline__ MulOp mul_op(double x) {
  return mul_op_bits((uint32_t)__double2hiint(x), (uint32_t)__double2loint(x));
}
__device__ __forceinline__ double mul_int(const MulOp& a, const MulOp& b) {
  return __longlong_as_double((long long)mul_bits(a, b));
}
// The rounded product of any two doubles, in integers where they allow it.
__device__ __forceinline__ double mul_any(double a, double b) {
  if (mul_safe(a) && mul_safe(b)) return mul_int(mul_op(a), mul_op(b));
  return __dmul_rn(a, b);
}
// a b + c d as the compiler fuses it: the second product is rounded.
__device__ __forceinline__ double sum2(double a, double b, double c, double d) {
  return fma(a, b, mul_any(c, d));
}
#endif

}  // namespace ba
