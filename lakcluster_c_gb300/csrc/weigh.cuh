// RN(D c) in integers, for a positive normal D and a count c.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace lakgb {

// D = dm 2^(ed - 1075) with dm in [2^52, 2^53), 0 < c < 2^11: dm c < 2^64 is
// exact and is rounded to 53 bits, ties to even.  (An FP64 multiply holds its
// sub-partition's FP64 pipe for 80 cycles per warp.)
__device__ __forceinline__ double weigh(unsigned long long dm, int ed, uint32_t c) {
  const unsigned long long x = dm * c;
  const int sh = 11 - __clzll((long long)x);  // bits past 53
  const unsigned long long r = (x + ((1ull << sh) >> 1) - (sh > 0) + ((x >> sh) & (sh > 0 ? 1ull : 0ull))) >> sh;
  return __longlong_as_double((long long)(((unsigned long long)(ed + sh - 1) << 52) + r));
}

// (Out of line: an FP64 instruction that the compiler predicates holds the pipe all
// the same.)
static __device__ __noinline__ double times_count_fp64(double d, uint32_t c) { return __dmul_rn(d, (double)c); }

// RN(d c), 0 <= c < 2^11, for any d: in integers where |d| is a normal number
// far from overflow.
__device__ __forceinline__ double times_count(double d, uint32_t c) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(d);
  const int ed = (int)(bits >> 52) & 0x7ff;
  if (ed == 0 || ed >= 2000) return times_count_fp64(d, c);
  const unsigned long long sign = bits & 0x8000000000000000ull;
  if (c == 0) return __longlong_as_double((long long)sign);
  return __longlong_as_double(__double_as_longlong(weigh((bits & 0x000fffffffffffffull) | 0x0010000000000000ull, ed, c)) |
                              (long long)sign);
}

}  // namespace lakgb
