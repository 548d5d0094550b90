// Intrinsics::undistort (geometry.rs:35-44) for the device passes: pixel to
// normalised coordinates by eight fixed-point steps x <- q / d(x).
//
// The steps are FP64 operations one after the other, ~64 cycles of the SM
// sub-partition each, and a division is nine of them; the two of a step share
// their divisor.  So a step takes one reciprocal (two) and two residual
// corrections (three each): 13 operations instead of 23 with the polynomial,
// of which the four plain products are made in integers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mul_int.cuh"

namespace ba {

static __device__ __noinline__ double quotient_slow(double x, double d) { return x / d; }

// 1 / d to 2^-45 of it: the FP32 reciprocal of d's leading 24 bits and one
// Newton step, two FP64 operations (the moves between the formats are integer
// ones).
__device__ __forceinline__ double reciprocal_near(double d) {
  const uint32_t hi = (uint32_t)__double2hiint(d), lo = (uint32_t)__double2loint(d);
  const uint32_t mag = hi & 0x7fffffffu, sign = hi & 0x80000000u;
  if (mag - (960u << 20) >= (126u << 20)) return __drcp_rn(d);  // not in 2^-63 .. 2^63
  const float f = __uint_as_float(((mag - (896u << 20)) << 3) | (lo >> 29));
  const uint32_t u = __float_as_uint(__frcp_rn(f));
  const double r = __hiloint2double((int)(((u >> 3) + (896u << 20)) | sign), (int)(u << 29));
  return fma(r, fma(-d, r, 1.0), r);
}

// x / d with r = 1 / d to 2^-45 or better: q = x r and one residual
// correction (Markstein, IBM J. Res. Dev. 34, 1990).  q is off by up to 2^8
// last places, so the residual x - q d has some 60 bits and is rounded to 53:
// an error of 2^-45 of a last place of q; r adds 2^8 times 2^-45 of one.  The
// result is x / d rounded but for 2^-36 of a last place (with r rounded to
// nearest q is off by one and the residual exact).  For q or r outside of
// 2^-900 .. 2^900 (and zero, infinite or NaN values) the division; an x below
// 2^-960, whose residual would be subnormal, is divided to its own spacing.
__device__ __forceinline__ double quotient_by(double x, double d, double r) {
  const double q = mul_any(x, r);
  const uint32_t eq = ((uint32_t)__double2hiint(q) >> 20) & 0x7ffu;
  const uint32_t er = ((uint32_t)__double2hiint(r) >> 20) & 0x7ffu;
  if (eq - 123u > 1800u || er - 123u > 1800u) return quotient_slow(x, d);
  return fma(fma(-q, d, x), r, q);
}

// K = {f, cx, cy, k1, k2}; rf = 1 / f rounded to nearest.
__device__ __forceinline__ void undistort(const double* K, double rf, double u, double v,
                                          double* p) {
  const double f = K[0], k1 = K[3], k2 = K[4];
  const double qx = quotient_by(u - K[1], f, rf), qy = quotient_by(v - K[2], f, rf);
  double px = qx, py = qy;
#pragma unroll 1
  for (int i = 0; i < 8; ++i) {
    const double r2 = sum2(px, px, py, py);
    const double d = fma(mul_any(k2, r2), r2, fma(k1, r2, 1.0));
    const double r = reciprocal_near(d);
    px = quotient_by(qx, d, r);
    py = quotient_by(qy, d, r);
  }
  p[0] = px, p[1] = py;
}

}  // namespace ba
