// 32 x 32 bit-matrix transpose in registers, one row per lane.
#pragma once

#include <cstdint>

namespace lakgb {

// Element (i, c) at bit 31 - c of lane i's word; afterwards lane r holds row
// r of the transpose.  Each step swaps the off-diagonal blocks of every
// 2j x 2j diagonal block (lanes j apart, bit groups j apart).
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
  const uint32_t masks[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int j = 16 >> k;
    const uint32_t m = masks[k];
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? ((x & m) | ((y << j) & ~m)) : ((x & ~m) | ((y >> j) & m));
  }
  return x;
}

// The same transpose with the lane's masks and rotations kept in registers,
// for kernels that transpose many words: per step one shuffle, one byte
// permute or rotation and one select of bits (the steps above: two shifts,
// two selects of bits and a select between them).
struct Transpose32 {
  uint32_t keep[3];
  uint32_t perm16, perm8, rot4, rot2, rot1;
  __device__ explicit Transpose32(int lane) {
    const uint32_t masks[3] = {0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int k = 0; k < 3; ++k) keep[k] = (lane & (4 >> k)) ? masks[k] : ~masks[k];
    // x and the shuffled y as bytes 0-3 and 4-7
    perm16 = (lane & 16) ? 0x5410u : 0x3276u;
    perm8 = (lane & 8) ? 0x6240u : 0x3715u;
    rot4 = (lane & 4) ? 4u : 28u;  // rotate left
    rot2 = (lane & 2) ? 2u : 30u;
    rot1 = (lane & 1) ? 1u : 31u;
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), perm16);
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), perm8);
    uint32_t y = __shfl_xor_sync(0xffffffffu, x, 4);
    x = (x & keep[0]) | (__funnelshift_l(y, y, rot4) & ~keep[0]);
    y = __shfl_xor_sync(0xffffffffu, x, 2);
    x = (x & keep[1]) | (__funnelshift_l(y, y, rot2) & ~keep[1]);
    y = __shfl_xor_sync(0xffffffffu, x, 1);
    return (x & keep[2]) | (__funnelshift_l(y, y, rot1) & ~keep[2]);
  }
};

}  // namespace lakgb
