// Order statistics of FP64 values within a CTA.
#pragma once

#include "ba_common.cuh"

namespace ba {

// f64 bits -> u64 whose unsigned order is f64::total_cmp's order.
__device__ __forceinline__ uint64_t total_order_key(double z) {
  const uint64_t b = (uint64_t)__double_as_longlong(z);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double from_total_order_key(uint64_t k) {
  const uint64_t b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)b);
}

// The key of rank k (0-based) among key[0..n): byte by byte from the top, the
// CTA counts the bytes of the keys that share the bytes found so far.  Lanes
// with the same byte count once (the top bytes hold a dozen exponents).  hist
// (256) and found (3) are shared; every thread of the CTA calls, and gets it.
template <int kThreads>
__device__ uint64_t select_key(const uint64_t* key, uint32_t n, uint32_t k, uint32_t* hist,
                               uint32_t* found) {
  const int lane = threadIdx.x & 31;
  uint64_t prefix = 0;
  for (int shift = 56; shift >= 0; shift -= 8) {
    for (int i = threadIdx.x; i < 256; i += kThreads) hist[i] = 0;
    __syncthreads();
    for (uint32_t i0 = 0; i0 < n; i0 += kThreads) {
      const uint32_t i = i0 + threadIdx.x;
      uint32_t d = 256;
      if (i < n) {
        const uint64_t v = key[i];
        if (shift == 56 || (v >> (shift + 8)) == prefix) d = (uint32_t)(v >> shift) & 255u;
      }
      const unsigned same = __match_any_sync(kFull, d);
      if (d < 256u && lane == __ffs(same) - 1) atomicAdd(&hist[d], (uint32_t)__popc(same));
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // the byte at which the running count passes k
      uint32_t c[8], sum = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) c[j] = hist[8 * lane + j], sum += c[j];
      uint32_t incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
      }
      uint32_t run = incl - sum;
      if (run <= k && k < incl) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (run <= k && k < run + c[j]) found[0] = 8 * lane + j, found[1] = k - run, found[2] = c[j];
          run += c[j];
        }
      }
    }
    __syncthreads();
    prefix = (prefix << 8) | found[0];
    k = found[1];
    const bool alone = found[2] == 1;
    __syncthreads();
    if (alone && shift > 0) {  // one key left: it has this prefix
      for (uint32_t i = threadIdx.x; i < n; i += kThreads) {
        const uint64_t v = key[i];
        if ((v >> shift) == prefix) found[0] = (uint32_t)v, found[1] = (uint32_t)(v >> 32);
      }
      __syncthreads();
      return ((uint64_t)found[1] << 32) | found[0];
    }
  }
  return prefix;
}

}  // namespace ba
