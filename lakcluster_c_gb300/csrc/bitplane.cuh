// Parameters of the bit-plane loop product At_T_YnWt_S_Zn_ww shared by its
// CUDA-core kernel (bitplane.cu) and its tensor-core kernel (bitplane_tc.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "scratch_limits.h"

namespace lakgb {

struct BitplaneParams {
  // At / Tt / planes share the row length `kbytes` (patients, a-space bits).
  const uint8_t *At; const uint32_t *at_rowb;   // per pair: At row (b index)
  long long at_row_bytes;
  const uint8_t *Tt; long long tt_row_bytes; const uint32_t *tt_rowb;  // per t
  const uint8_t *planes; long long plane_bytes;
  const uint8_t *mask;                          // M_At->mc_j
  int P;                                        // 1920-bit blocks per row
  int npairs;
  const uint8_t *Zt; const uint32_t *zt_rowb; long long zt_row_bytes;
  const uint32_t *mw_a;                         // a-index of each Wn row (j order)
  int nW; int B; int ncols_per; int nT;
  const int8_t *vS;                             // [t][mw] +/-1
  const double *aA; const double *aZ;           // per pair
  const int *ycnt;                              // per plane row: popcount(y & mask)
  const double *T_base; const double *T_tmp;    // [t], [t][mw]
  double min_d, mlt_d;
  const unsigned long long *out_off;            // per pair: row index in the output
  const unsigned long long *t_off;              // per t: column offset (index * row_stride)
  double *out;
  // tensor-core form
  int chunks;                                   // 128-bit chunks that hold patients
  const uint32_t *a_blk;                        // per pair: 1920-SNP block of the At row
  const double *aBlk; int nblk;                 // a of every block
  double inv_mlt;                               // RN(1 / mlt); 0: divide by mlt itself
  const double *At_base;                        // [t][pair]
  const double2 *zz;                            // per pair: 1 - aZ, -1 - aZ
  const long long *ysum;                        // per Wn row: sum_k 2^k popcount(plane_k & mask)
  const double *q2;                             // [t][block][mw]: (a T_base + a T_tmp) / mlt
};

// The tensor-core form (bitplane_tc.cu), in place of bitplane_main_kernel;
// requires B in {8, 16, 32}.  A segment is a range of Wn rows of one (call,
// covariate column); its terms, one per (pair, Wn row), go to a scratch array
// and are then added up in order.  A batch is what one pair of launches
// computes: as many segments as the scratch holds.
struct BitplaneSeg {
  int call, t, w0, w1;
  int unit0;      // first (pair tile, N tile) unit of the segment in its batch
  int block0;     // first block of the segment in the batch's adding launch
  long long y0;   // its terms in the scratch: [w - w0][pair]
};
struct BitplaneBatch { int seg0, nseg, units, blocks; };
// Segments and batches of calls (host parameters) of the same B; returns the
// scratch's size in doubles.
size_t bitplane_tc_plan(int B, const std::vector<BitplaneParams> &ps, std::vector<BitplaneSeg> *segs,
                        std::vector<BitplaneBatch> *batches);
void launch_bitplane_tc(int B, const BitplaneParams *d_ps, const BitplaneSeg *d_segs,
                        const std::vector<BitplaneBatch> &batches, double *scratch, cudaStream_t s);
// Most doubles of scratch that the terms of a batch take; one step of Wn rows of
// one column always fits.
constexpr size_t kBitplaneScratch = kBitplaneScratchBytes / sizeof(double);

}  // namespace lakgb
