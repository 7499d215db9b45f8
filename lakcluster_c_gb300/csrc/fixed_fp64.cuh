// FP64 sums of a few values of like size in 64-bit integers: a warp's FP64
// instruction holds its sub-partition's FP64 pipe for 80 cycles, an integer
// one an ALU for 2, so a rounded add of about 20 integer instructions takes
// half the time and leaves the pipe to others.
//
// With emax the largest biased exponent of the values, a fixed-point number is
// a multiple of 2^(emax - 1082): the largest value has 60 bits, so sums and
// differences of up to eight stay below 2^63.  A value is representable if it
// has no bits below that unit (any value down to 2^-7 of the largest, smaller
// ones if their low bits are clear); the others take the FP64 operations.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define LAKGB_HD __host__ __device__ __forceinline__
#else
#define LAKGB_HD inline
#endif

namespace lakgb {
namespace fixed {

constexpr int kBelow = 7;  // binades below the largest

LAKGB_HD int clz32(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}
LAKGB_HD int clz64(unsigned long long x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}

// Exponents for which every result is a normal number.
LAKGB_HD bool in_range(int emax) { return emax >= 100 && emax <= 2040; }

// x (its bits; exponent <= emax) as a fixed-point number; false: not
// representable (also -0, subnormal, infinite or not a number).
LAKGB_HD bool from_bits(unsigned long long x, int emax, long long *out) {
  *out = 0;
  if (x == 0ull) return true;
  const int e = (int)((x >> 52) & 0x7FF);
  if (e == 0 || e == 0x7FF) return false;
  unsigned long long m = (x & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
  const int sh = e - emax + kBelow;
  if (sh >= 0) {
    m <<= sh;
  } else {
    if (sh < -52 || (m & ((1ull << -sh) - 1ull))) return false;
    m >>= -sh;
  }
  *out = (x >> 63) ? -(long long)m : (long long)m;
  return true;
}

// s rounded to 53 significant bits, ties to even: adding just under half a
// unit (half of one where the last kept bit is odd) and clearing the k bits
// below, which rounds negative numbers alike.  k comes from the length of
// |s| - 1 for those: one less only for a power of two, which is exact anyway.
LAKGB_HD long long round53(long long s) {
  const int hi = (int)(s >> 32);
  const int k = 11 - clz32((uint32_t)(hi ^ (hi >> 31)));
  const uint32_t mask = (1u << (k > 0 ? k : 0)) - 1u, lo = (uint32_t)s;
  s += (mask >> 1) + ((lo >> (k > 0 ? k : 0)) & mask & 1u);
  return s & ~(long long)mask;
}

// The bits of s rounded to the nearest double, ties to even.
LAKGB_HD unsigned long long to_bits(long long s, int emax) {
  if (s == 0) return 0ull;
  const unsigned long long sign = (unsigned long long)s & 0x8000000000000000ull;
  unsigned long long n = sign ? 0ull - (unsigned long long)s : (unsigned long long)s;
  const int z = clz64(n);
  n <<= z;
  const unsigned long long b = n >> 11;
  const uint32_t up = (((uint32_t)n & 0x7FFu) + 0x3FFu + ((uint32_t)b & 1u)) >> 11;
  return sign | ((((unsigned long long)(emax + 10 - kBelow - z)) << 52) + b + up);
}

// 2 x on the bits, as the FP64 multiply rounds it: one more in the exponent,
// a shift for subnormal numbers, infinity past the largest.
LAKGB_HD unsigned long long twice_bits(unsigned long long x) {
  const unsigned long long sign = x & 0x8000000000000000ull, mag = x ^ sign;
  const int e = (int)(mag >> 52);
  if (e >= 1 && e <= 2045) return x + (1ull << 52);
  if (e == 0) return sign | (mag << 1);
  return e == 2046 ? sign | 0x7FF0000000000000ull : x;
}

}  // namespace fixed
}  // namespace lakgb
