// Tensor-core bit-pair counts for small Grams and the SNP x SNP product
// (tc_counts.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace lakgb {

struct GramParams;

constexpr int kCountsM = 128, kCountsN = 64;  // tile rows of A and Z
constexpr int kCountsMaxRows = 65535 * kCountsM;

// The Gram p as per-block counts (cnt: P x nZ x nA 16-bit integers of scratch)
// and a fold over the blocks in order.  P <= 65535.
void launch_gram_tc_split(const GramParams &p, uint16_t *cnt, cudaStream_t s);

// The counts alone, per span of blocks: cnt (spans x nZ x nA 16-bit integers:
// popcount(A & Z & mask)) and zcnt (spans x nZ: popcount(Z & mask)), with
// ceil(P / span) spans of and_counts_span(...) blocks; nA <= kCountsMaxRows.
int and_counts_span(long long nA, long long nZ, int P);
void launch_and_counts_tc(const GramParams &p, int span, uint16_t *cnt, uint16_t *zcnt, cudaStream_t s);

// AtTYn_vv and, with `symmetric`, AtTAn_vv.
struct AtTYnParams {
  const uint8_t *At; const uint32_t *a_rowb; int nA; long long a_row_bytes;
  const uint8_t *Yt; const uint32_t *y_rowb; int nY; long long y_row_bytes;
  const uint8_t *Tt; const uint32_t *t_rowb; long long t_row_bytes;
  const uint8_t *mask; int P; long long cpop;
  const double *hhAy;   // [t][na]
  const double *hhaY;   // [t][ny]
  const double *hhay;   // [t]
  const double *aA; const double *aY;
  const unsigned long long *out_a; const unsigned long long *out_y; const unsigned long long *out_t;
  double *out;
  // AtTAn (Yt = At): pairs na <= ny only, each also stored at
  // out_a2[ny] + out_y2[na] (the transposed position).
  int symmetric;
  const unsigned long long *out_a2; const unsigned long long *out_y2;
};
void launch_attyn_tc(const AtTYnParams &p, int nT, cudaStream_t s);

}  // namespace lakgb
