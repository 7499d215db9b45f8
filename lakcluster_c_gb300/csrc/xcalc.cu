// Quantisation of an FP64 matrix into bit planes: get_xcalc / wrap_xcalc
// (dir_c/xcalc.c:5-263).
//
// Given YnWt (rows: the Yn rows selected by mr_b & mr_j; columns: the Wn rows
// selected by mc_b & mc_j), the planes M_X hold, for each retained column
// nc_j, ncols_per = b_mlt + 1 rows of bits over the Yn rows (a-space):
//   plane ncols_per*nc_j + ncols_per-1-nb = bit nb of
//       cz = crop((unsigned long long)(mlt*(x - min)), 1, D_MLT-1)
// and plane 0 additionally marks the rows set in mr_j.  min, max and mlt come
// from the masked extremes (xcalc_setmaxmin, xcalc.c:5-39):
//   min = min_x - (max_x-min_x)/16,  max = max_x + (max_x-min_x)/16,
//   mlt = D_MLT / (max - min).
// The products that read the planes (At_T_YnWt_S_Zn_ww, An_ZtSn_ww) undo the
// scaling exactly as the reference does, so the planes must match bit for bit:
// the conversion is one IEEE subtract, one multiply and a truncation, computed
// here with the same rounding.
//
// Device side: the masked min / max is a grid reduction (exact, order-free)
// whose last block forms min, max and mlt; the planes are built by warps that
// each take 256 rows, quantise in 64-bit fixed point and transpose 32 x 32
// bits in registers.  The planes stay resident on the device for the products
// that follow, and are copied into M_X->wX for callers that read them on the
// host.
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>
#include <optional>

#include "abi_common.cuh"
#include "bit_transpose.cuh"
#include "bcc_model.h"
#include "lmirror.cuh"

namespace lakgb {

namespace {

// GLOBAL_D_MLT (default lakcluster_ver18.c:83), per host thread: concurrent
// solves may use different B_MLT.
thread_local long long g_d_mlt = 4294967296LL;

// min, max and mlt of one matrix, and the constants of the fixed-point
// quantisation (quantise_fixed below): frac = -1 when the FP64 operations are
// used for every value.
struct XcalcScalars {
  double lo, hi, mlt;
  unsigned long long K;       // mlt in fixed point
  unsigned long long neglo;   // -lo in fixed point
  unsigned long long span;    // largest value - lo in fixed point
  int shift0, frac;
};

struct XcalcParams {
  const double *lf;
  const long long *row_off;  // per a-row of Yn (nrows_a): element offset, -1 = not retained
  int nrows_a;
  const long long *col_off;  // per retained column nc_j
  int ncols_j;
  unsigned long long dmax;   // D_MLT - 1
  int ncols_per;
  long long brows;           // bytes per plane row
  uint8_t *planes;
  const uint8_t *row0;       // first plane's bytes (null: zeros)
  long long row_max;         // largest row offset
  unsigned long long lf_n, planes_n;  // elements of lf, bytes of planes (bounds checks)
  // set when an index would leave its buffer (access skipped); null: the
  // caller's offsets, negative ones among them, are taken as they are
  int *bad;
  const XcalcScalars *sc;
};

// The masked min / max compare order keys instead of doubles: GB300's FP64
// pipe issues about two compares per clock per SM, which held a min/max scan
// to a quarter of HBM bandwidth, while the integer pipe compares 64-bit keys
// at memory speed.  The key of x is its bit pattern with the sign bit flipped
// for x >= 0 and every bit flipped for x < 0, so unsigned key order is the
// order of the values, with -0 below +0.  The reference keeps the first of
// equal extremes (xcalc.c:25), so a min or max of zero may differ from it in
// sign only; min, max and mlt (xcalc.c:130) come out the same either way:
// a zero extreme enters them only through differences with the other extreme
// or, when both are zero, through min_data + 1 (xcalc.c:34).
__device__ __forceinline__ unsigned long long order_key(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

__device__ __forceinline__ double key_value(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
}

// |x| < 2^e in units of 2^(e-62), truncated towards zero, negated for x < 0;
// shift0 = e + 1024.  *ok is false outside that range (and for inf and NaN).
__device__ __forceinline__ unsigned long long to_fixed(double x, int shift0, bool *ok) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const int r = shift0 - (int)((hi >> 20) & 0x7ffu);
  *ok = r >= 2;
  // the significand with its leading bit at bit 63, shifted down (by 64 and
  // more: zero, as PTX defines the shift)
  const unsigned long long m = ((unsigned long long)((hi << 11) | (lo >> 21) | 0x80000000u) << 32) | (lo << 11);
  unsigned long long v;
  asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"(r));
  const unsigned long long sgn = (unsigned long long)((long long)((unsigned long long)hi << 32) >> 63);
  return (v ^ sgn) - sgn;
}

// min, max and mlt from the extremes' keys with the reference's operations
// (xcalc.c:34, :130), and the fixed-point constants: with w = max - min in
// [2^(e-1), 2^e), values are taken in units of 2^(e-62), and
// K = mlt 2^(e + 2 + frac) <= 2^63 turns them into quantised values with
// `frac` fraction bits: T = x_fixed K / 2^64 = mlt (x - min) 2^frac.
__device__ void make_scalars(unsigned long long kmn, unsigned long long kmx, bool nan_first, long long d_mlt,
                             XcalcScalars *out) {
  double mn = 0.0, mx = 0.0;
  if (kmn <= kmx) { mn = key_value(kmn); mx = key_value(kmx); }
  if (nan_first) mn = mx = __longlong_as_double(0x7ff8000000000000ll);
  const double top = mx;
  if (mn >= mx) mx = __dadd_rn(mn, 1.0);
  const double range = __dsub_rn(mx, mn);
  XcalcScalars r;
  r.lo = __dsub_rn(mn, __dmul_rn(0.0625, range));
  r.hi = __dadd_rn(mx, __dmul_rn(0.0625, range));
  const double w = __dsub_rn(r.hi, r.lo);
  r.mlt = __ddiv_rn((double)d_mlt, w);
  const int E = (int)(((unsigned long long)__double_as_longlong(w) >> 52) & 0x7ff);
  const int bits = 64 - __clzll(d_mlt - 1);  // d_mlt <= 2^bits
  const int e = E - 1022;
  r.frac = 60 - bits;
  r.shift0 = e + 1024;
  r.K = r.neglo = r.span = 0ull;
  bool ok_lo, ok_top;
  r.neglo = 0ull - to_fixed(r.lo, r.shift0, &ok_lo);
  r.span = to_fixed(top, r.shift0, &ok_top) + r.neglo;
  if (d_mlt < 64 || bits > 38 || E < 200 || E > 1800 || !(w > 0.0) || !(r.mlt > 0.0) || !ok_lo || !ok_top) {
    r.frac = -1;
  } else {
    const unsigned long long mb = (unsigned long long)__double_as_longlong(r.mlt);
    const int s = (int)(mb >> 52) - 1075 + e + 2 + r.frac;  // 9 <= s <= 11: 2^61 < K <= 2^63
    r.K = ((mb & 0x000fffffffffffffull) | 0x0010000000000000ull) << s;
  }
  *out = r;
}

// Grid: blockIdx.x * blockDim.x + threadIdx.x strides the retained rows, each
// thread holding kMinMaxRows row offsets in registers for all its columns;
// blockIdx.y strides the retained columns, kMinMaxCols per pass, so that
// kMinMaxRows * kMinMaxCols loads are in flight per thread.  One partial
// (min key, max key) per block; the last block to finish reduces them and
// forms the scalars, so the planes kernel follows with no launch between.
// SKIP_NAN: a NaN is left out of the extremes unless it is the first retained
// value, which then gives NaN (the comparisons of xcalc.c:25 in order).
constexpr int kMinMaxRows = 4, kMinMaxCols = 2, kMinMaxThreads = 256;
constexpr int kMinMaxBlocks = 152 * 8;  // most blocks of a launch

template <bool SKIP_NAN>
__global__ void __launch_bounds__(kMinMaxThreads, 5)
    xcalc_minmax_kernel(const double *lf, const long long *rows_j, int nr, const long long *cols_j, int nc,
                        ulonglong2 *part, unsigned *ticket, long long d_mlt, XcalcScalars *out) {
  release_next();
  unsigned long long kmn = ~0ull, kmx = 0ull;  // empty: kmn > kmx
  const int stride = gridDim.x * blockDim.x;
  for (int rb = blockIdx.x * blockDim.x + threadIdx.x; rb < nr; rb += kMinMaxRows * stride) {
    long long ro[kMinMaxRows];
    bool rok[kMinMaxRows];
#pragma unroll
    for (int u = 0; u < kMinMaxRows; ++u) {
      const int r = rb + u * stride;
      rok[u] = r < nr;
      ro[u] = rok[u] ? rows_j[r] : 0;
    }
    for (int c = blockIdx.y; c < nc; c += kMinMaxCols * gridDim.y) {
      double x[kMinMaxCols][kMinMaxRows];
      bool cok[kMinMaxCols];
#pragma unroll
      for (int k = 0; k < kMinMaxCols; ++k) {
        const int ck = c + k * gridDim.y;
        cok[k] = ck < nc;
        const long long co = cok[k] ? cols_j[ck] : 0;
#pragma unroll
        for (int u = 0; u < kMinMaxRows; ++u) x[k][u] = (cok[k] && rok[u]) ? __ldg(lf + ro[u] + co) : 0.0;
      }
#pragma unroll
      for (int k = 0; k < kMinMaxCols; ++k)
#pragma unroll
        for (int u = 0; u < kMinMaxRows; ++u) {
          const unsigned long long b = (unsigned long long)__double_as_longlong(x[k][u]);
          if (cok[k] && rok[u] && !(SKIP_NAN && (b << 1) > 0xffe0000000000000ull)) {
            const unsigned long long q = order_key(x[k][u]);
            kmn = q < kmn ? q : kmn;
            kmx = q > kmx ? q : kmx;
          }
        }
    }
  }
  __shared__ unsigned long long smn[kMinMaxThreads / 32], smx[kMinMaxThreads / 32];
  __shared__ bool last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto block_reduce = [&]() {  // result in thread 0
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long omn = __shfl_xor_sync(0xffffffffu, kmn, o);
      const unsigned long long omx = __shfl_xor_sync(0xffffffffu, kmx, o);
      kmn = omn < kmn ? omn : kmn;
      kmx = omx > kmx ? omx : kmx;
    }
    if (lane == 0) { smn[warp] = kmn; smx[warp] = kmx; }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 1; w < kMinMaxThreads / 32; ++w) {
        kmn = smn[w] < kmn ? smn[w] : kmn;
        kmx = smx[w] > kmx ? smx[w] : kmx;
      }
  };
  block_reduce();
  const int blocks = gridDim.x * gridDim.y;
  if (threadIdx.x == 0) {
    part[blockIdx.x + gridDim.x * blockIdx.y] = make_ulonglong2(kmn, kmx);
    __threadfence();
    last = atomicAdd(ticket, 1u) == (unsigned)blocks - 1u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  kmn = ~0ull;
  kmx = 0ull;
  for (int i = threadIdx.x; i < blocks; i += kMinMaxThreads) {
    const ulonglong2 q = __ldcg(part + i);
    kmn = q.x < kmn ? q.x : kmn;
    kmx = q.y > kmx ? q.y : kmx;
  }
  block_reduce();
  if (threadIdx.x == 0) {
    bool nan_first = false;
    if (SKIP_NAN && nr > 0 && nc > 0) nan_first = isnan(lf[rows_j[0] + cols_j[0]]);
    make_scalars(kmn, kmx, nan_first, d_mlt, out);
    *ticket = 0u;  // ready for the next launch
  }
}

// floor(mlt * (x - min)) cropped to [1, dmax], as the FP64 operations of
// xcalc.c:150 give it.
__device__ __forceinline__ unsigned long long quantise_fp64(double x, const XcalcScalars &s, unsigned long long dmax) {
  unsigned long long v = __double2ull_rz(__dmul_rn(s.mlt, __dsub_rn(x, s.lo)));
  if (v < 1ull) v = 1ull;
  return v > dmax ? dmax : v;
}

// The same in 64-bit integers: GB300's FP64 pipe takes 80 cycles per warp
// instruction, and the subtract, the multiply and the conversion are three.
// T = mlt (x - min) 2^frac is within 5 of the exact product (two truncations
// to the unit, the product's low words left out, K <= 2^63), and the two FP64
// roundings move that by at most 2^-52 of 2^60, 2^8.  Only where a multiple
// of 2^frac lies within kMargin of T could the integer part differ: for those
// values (about one in 2^17 at 32 bits) and for values above the largest one,
// below min or not finite, *ok is false and the FP64 operations decide.  A
// value up to the largest one stays below 17 d_mlt / 18 and so needs no
// cropping from above (frac is -1 for d_mlt < 64).
constexpr unsigned kMargin = 1u << 10;
__device__ __forceinline__ unsigned long long quantise_fixed(double x, const XcalcScalars &s, bool *ok) {
  bool in;
  const unsigned long long d = to_fixed(x, s.shift0, &in) + s.neglo;
  const uint32_t dh = (uint32_t)(d >> 32), kh = (uint32_t)(s.K >> 32);
  const unsigned long long t =
      (unsigned long long)dh * kh + __umulhi(dh, (uint32_t)s.K) + __umulhi((uint32_t)d, kh);
  // frac is 22 to 54; its low 22 bits or more lie in the low word
  const uint32_t low = (uint32_t)t + kMargin;
  bool clear = (low & ((1u << min(s.frac, 31)) - 1u)) >= 2u * kMargin;
  *ok = in && d <= s.span && clear;
  const unsigned long long v = t >> s.frac;
  return v < 1ull ? 1ull : v;
}

__device__ __forceinline__ void note_bad(int *bad, int code) {
  if (bad) atomicCAS(bad, 0, code);
}

// Warp per 256-row group (32 bytes of every plane row), for the columns
// c, c + step, ...: the row offsets stay in registers, lane l quantises rows
// 256g + 32k + l, k = 0..7 (eight independent coalesced loads).  Per k, the
// 32 x 32 bit matrix (row l = bits nb0 .. nb0+31 of lane l's value) is
// transposed in registers, so lane j holds the word of bit nb0+j; lane j then
// writes its plane's 32 bytes.  Every byte of the column's plane rows is
// written, the first plane and (by the last group's warp) the padding past the
// rows included, so the planes need no zero-fill before.  WIDE: plane rows and the array are 16-byte
// aligned (16-byte stores); otherwise 4-byte ones.  T: holds b_mlt bits.
// Bound: the integer pipe (71 % active at 8192 x 8192; about 100 operations per value,
// 30 of them the transpose), then load latency.  4096 x 4001 values to 32 bits
// through lakgb_xcalc_noalloc: 1463 us a call before (a warp per 32 rows, FP64
// operations, 4-byte stores, one thread folding the columns' extremes), 130 us
// now; this kernel 76 us, the extremes 37 us.
constexpr int kPlaneRows = 256, kPlaneThreads = 256, kPlaneBlocks = 3;
template <bool WIDE, typename T>
__global__ void __launch_bounds__(kPlaneThreads, kPlaneBlocks) xcalc_planes_kernel(XcalcParams p, int cstep) {
  constexpr int R = kPlaneRows / 32;
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  const int ngroups = max(1, (p.nrows_a + kPlaneRows - 1) / kPlaneRows);
  const int g = warp % ngroups;
  await_previous();
  if (warp / ngroups >= cstep) return;
  const long long pad0 = g == ngroups - 1 ? 32ll * ngroups : p.brows;  // padding this warp clears
  const XcalcScalars s = *p.sc;
  const Transpose32 tr(lane);
  long long ro[R];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int r = g * kPlaneRows + 32 * k + lane;
    ro[k] = r < p.nrows_a ? p.row_off[r] : -1;
  }
  const int nbits = p.ncols_per - 1;
  const long long byte0 = 32ll * g;
  for (int c = warp / ngroups; c < p.ncols_j; c += cstep) {
    const long long co = p.col_off[c];
    const bool inside = !p.bad || (unsigned long long)(p.row_max + co) < p.lf_n;
    if (!inside) note_bad(p.bad, 1);
    double x[R];
    unsigned live = 0u;
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const bool l = inside && ro[k] >= 0;
      live |= (unsigned)l << k;
      x[k] = l ? __ldg(p.lf + ro[k] + co) : 0.0;
    }
    T cz[R];
    unsigned fp64 = live;
    if (s.frac >= 0) {
      fp64 = 0u;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        bool ok;
        cz[k] = (T)quantise_fixed(x[k], s, &ok);
        if (!ok) fp64 |= 1u << k;
      }
      fp64 &= live;
    }
    // one branch for the warp and the eight rows, its values read again: FP64
    // instructions that the compiler predicates, or hoists above the branch,
    // cost their 80 cycles for every value
    if (__any_sync(0xffffffffu, fp64 != 0u)) {
#pragma unroll
      for (int k = 0; k < R; ++k)
        if ((fp64 >> k) & 1u) cz[k] = (T)quantise_fp64(__ldcv(p.lf + ro[k] + co), s, p.dmax);
    }
#pragma unroll
    for (int k = 0; k < R; ++k)
      if (!((live >> k) & 1u)) cz[k] = 0;
    const long long first = (long long)p.ncols_per * c;
    for (int nb0 = 0; nb0 < nbits; nb0 += 32) {
      // lane j's word has row i at bit 31-i; memory wants row 8m+q at byte m, bit 7-q.
      uint32_t o[R];
#pragma unroll
      for (int k = 0; k < R; ++k) o[k] = __byte_perm(tr(__brev((uint32_t)(cz[k] >> nb0))), 0u, 0x0123);
      if (lane < nbits - nb0) {
        const unsigned long long off = (unsigned long long)((first + nbits - (nb0 + lane)) * p.brows + byte0);
        if (WIDE) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (byte0 + 16 * h < p.brows) {
              if (off + 16 * h + 16 > p.planes_n) note_bad(p.bad, 2);
              else *reinterpret_cast<uint4 *>(p.planes + off + 16 * h) =
                  make_uint4(o[4 * h], o[4 * h + 1], o[4 * h + 2], o[4 * h + 3]);
            }
          for (long long b = pad0; b < p.brows; b += 16)
            if (off - byte0 + b + 16 <= p.planes_n)
              *reinterpret_cast<uint4 *>(p.planes + off - byte0 + b) = make_uint4(0u, 0u, 0u, 0u);
        } else {
#pragma unroll
          for (int k = 0; k < R; ++k)
            if (byte0 + 4 * k < p.brows) {
              if (off + 4 * k + 4 > p.planes_n) note_bad(p.bad, 2);
              else *reinterpret_cast<uint32_t *>(p.planes + off + 4 * k) = o[k];
            }
          for (long long b = pad0; b < p.brows; b += 4)
            if (off - byte0 + b + 4 <= p.planes_n) *reinterpret_cast<uint32_t *>(p.planes + off - byte0 + b) = 0u;
        }
      }
      if (sizeof(T) == 4) break;
    }
    // the column's mask plane: row0 before the first column, zero elsewhere
    const long long mask_end = pad0 < p.brows ? p.brows : min(p.brows, byte0 + 32);
    for (long long b = byte0 + lane; b < mask_end; b += 32) {
      const unsigned long long off = (unsigned long long)(first * p.brows + b);
      if (off >= p.planes_n) note_bad(p.bad, 2);
      else p.planes[off] = (c == 0 && p.row0) ? p.row0[b] : (uint8_t)0;
    }
  }
}

// One resident wave of warps (kPlaneBlocks blocks per SM) over the row groups
// and as many column steps.
void launch_planes(const XcalcParams &p, cudaStream_t s) {
  if (p.brows <= 0) return;
  const long long ngroups = std::max(1, (p.nrows_a + kPlaneRows - 1) / kPlaneRows);
  const long long resident = 152ll * kPlaneBlocks * (kPlaneThreads / 32);
  const int cstep = (int)std::max(1ll, std::min<long long>(p.ncols_j, resident / ngroups));
  const unsigned blocks = (unsigned)((ngroups * cstep * 32 + kPlaneThreads - 1) / kPlaneThreads);
  const bool wide = (p.brows & 15) == 0 && (reinterpret_cast<uintptr_t>(p.planes) & 15) == 0;
  const bool narrow = p.ncols_per - 1 <= 32 && p.dmax <= 0xffffffffull;
  if (wide && narrow)
    launch_after(xcalc_planes_kernel<true, uint32_t>, blocks, kPlaneThreads, 0, s, p, cstep);
  else if (wide)
    launch_after(xcalc_planes_kernel<true, unsigned long long>, blocks, kPlaneThreads, 0, s, p, cstep);
  else
    launch_after(xcalc_planes_kernel<false, unsigned long long>, blocks, kPlaneThreads, 0, s, p, cstep);
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
}

// Rows across blockIdx.x (kMinMaxRows per thread), columns across blockIdx.y.
dim3 minmax_grid(int nr, int nc) {
  const int gx = std::max(1, std::min((nr + kMinMaxRows * kMinMaxThreads - 1) / (kMinMaxRows * kMinMaxThreads),
                                      kMinMaxBlocks));
  return dim3(gx, std::max(1, std::min(nc, kMinMaxBlocks / gx)));
}

// --- allocation-free variant ---------------------------------------------
//
// lakgb_xcalc_noalloc runs the same kernels on caller-owned device buffers
// for callers that cannot allocate device memory.  Its only scratch is this
// file-scope array: the blocks' partial extremes, the scalars and the ticket of
// the last block.  Every entry a call reads is written earlier in the same call;
// the array is shared by every call on a device, so calls whose kernels overlap
// on the GPU race.  (The scratch does not grow with the columns any more; their
// limit is one of the interface.)
constexpr int kNoAllocMaxCols = LAKGB_XCALC_NOALLOC_MAX_COLS;
constexpr int kScratchScalars = 2 * kMinMaxBlocks;       // doubles from the start
constexpr int kScratchTicket = kScratchScalars + (int)(sizeof(XcalcScalars) / sizeof(double));
static __device__ __align__(256) double g_xcalc_noalloc_scratch[kScratchTicket + 1];
static_assert(sizeof(ulonglong2) == 2 * sizeof(double) && sizeof(XcalcScalars) % sizeof(double) == 0, "whole doubles");

std::mutex g_noalloc_mu;
void *g_noalloc_scratch[64] = {nullptr};

// Device address of the scratch array on the current device, looked up once
// per device (the lookup is a runtime call that must not run inside a stream
// capture, so callers make their first call before any capture).
double *noalloc_scratch() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_scratch[dev]) {
    void *ptr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&ptr, g_xcalc_noalloc_scratch);
    if (e != cudaSuccess) {
      set_error(1000 + (int)e, "lakgb_xcalc_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      return nullptr;
    }
    g_noalloc_scratch[dev] = ptr;
  }
  return static_cast<double *>(g_noalloc_scratch[dev]);
}

}  // namespace

}  // namespace lakgb

using namespace lakgb;

extern "C" void lakgb_set_d_mlt(long long d_mlt) { g_d_mlt = d_mlt; }

namespace lakgb {
namespace {
// The flag of the planes kernel's bounds checks and the ticket of the extremes
// kernel's last block (its launches follow one another on the thread's stream;
// zero between launches), per host thread.
int *bad_flag() { return thread_word(kXcalcBad); }
unsigned *minmax_ticket() { return reinterpret_cast<unsigned *>(thread_word(kXcalcTicket)); }

// Calls inside a deferral scope: their scalars stay on the device (one
// XcalcScalars per call, in chunks of kSlots calls) until the scope ends;
// then M_X's fields are set from them.
constexpr int kSlots = 256;
struct XcalcDeferred { M_handle *M_X; int slot; };
thread_local std::vector<DBuf> t_xs_chunks;
thread_local int t_xs_used = 0;
thread_local std::vector<XcalcDeferred> t_xs;

XcalcScalars *xcalc_slot(int &slot) {
  if (t_xs_used == (int)t_xs_chunks.size() * kSlots) t_xs_chunks.emplace_back((size_t)kSlots * sizeof(XcalcScalars));
  slot = t_xs_used++;
  return t_xs_chunks[slot / kSlots].as<XcalcScalars>() + slot % kSlots;
}

void xcalc_deferred_enqueue() {}

// After the scope's wait: the scalars into M_X (xcalc.c:240), the planes
// kernels' bounds flag checked once.
void xcalc_deferred_finish() {
  std::vector<XcalcScalars> h((size_t)t_xs_used);
  for (size_t c = 0; c < t_xs_chunks.size(); ++c) {
    const int n = std::min(kSlots, t_xs_used - (int)c * kSlots);
    if (n > 0)
      LAKGB_CUDA(cudaMemcpyAsync(h.data() + c * kSlots, t_xs_chunks[c].p, (size_t)n * sizeof(XcalcScalars),
                                 cudaMemcpyDeviceToHost, stream()));
  }
  int hbad = 0;
  LAKGB_CUDA(cudaMemcpyAsync(&hbad, bad_flag(), sizeof(int), cudaMemcpyDeviceToHost, stream()));
  LAKGB_CUDA(cudaStreamSynchronize(stream()));
  for (const XcalcDeferred &d : t_xs) {
    const XcalcScalars &v = h[(size_t)d.slot];
    d.M_X->min_d = v.lo; d.M_X->max_d = v.hi; d.M_X->mlt_d = v.mlt;
    if (!isfinite(d.M_X->mlt_d) || d.M_X->mlt_d <= 0) d.M_X->mlt_d = 1;
  }
  if (hbad) {
    printf(" %% Warning! wrap_xcalc: a call skipped an out-of-range index (code %d)\n", hbad);
    set_error(5, "wrap_xcalc: a call skipped an out-of-range index (code %d)", hbad);
    LAKGB_CUDA(cudaMemsetAsync(bad_flag(), 0, sizeof(int), stream()));
  }
  t_xs.clear();
  t_xs_chunks.clear();
  t_xs_used = 0;
}
}  // namespace
}  // namespace lakgb

extern "C" void wrap_xcalc(int *tidx, void **vpra, pthread_t *thread_in, unsigned char *mr_j,
                           unsigned char *mr_b, unsigned char *mc_j, unsigned char *mc_b,
                           L_handle *lf_YnWt, double *YnWt, int *Yn_nrows_p, int *Wn_nrows_p,
                           M_handle **M_X_p, int *b_mlt_p, int trm_flag) {
  LAKGB_PROFILE_CALL("wrap_xcalc");
  (void)tidx; (void)vpra; (void)thread_in;
  const int Yn_nrows = *Yn_nrows_p, Wn_nrows = *Wn_nrows_p, b_mlt = *b_mlt_p;
  if (!M_X_p || !*M_X_p) {
    set_error(3, "wrap_xcalc: *M_X_p must be pre-allocated");
    return;
  }
  if (!mr_j || !mr_b || !mc_j || !mc_b) printf(" %% Warning! null mask in get_xcalc\n");
  M_handle *M_X = *M_X_p;
  const long ylen = lakbcc::bsize(Yn_nrows), wlen = lakbcc::bsize(Wn_nrows);
  const int rpop_j = popcount_bytes(mr_j, ylen), rpop_b = popcount_bytes(mr_b, ylen);
  const int cpop_j = popcount_bytes(mc_j, wlen);
  const long long length = (long long)Yn_nrows * Wn_nrows;
  const int ncols_per = b_mlt + 1;
  if (ncols_per > 63) printf(" %% Warning! overflow in get_xcalc!\n");

  // Retained rows / columns and their element offsets (L2_lf_get, L_init.c:188-200).
  const int sr = lf_YnWt ? lf_YnWt->spacing_row : 0, sc = lf_YnWt ? lf_YnWt->spacing_col : 0;
  const unsigned long long rs = lf_YnWt ? lf_YnWt->row_stride : 0;
  std::vector<long long> row_off_a((size_t)(Yn_nrows > 0 ? Yn_nrows : 1), -1), rows_j, cols_j;
  {
    std::vector<unsigned> ia, ib;
    // the retained elements' offsets in one dimension of lf
    auto offsets = [&](int n, const unsigned char *mb, const unsigned char *mj, int spacing, unsigned long long stride,
                       std::vector<long long> &out) {
      ia.resize((size_t)(n > 0 ? n : 0));
      ib.resize(ia.size());
      const long cnt = lakbcc::mask_lists(n, mb, mj, ia.data(), ib.data());
      out.resize((size_t)cnt);
      const unsigned *from = spacing == LAKGB_SPACING_b ? ib.data() : spacing == LAKGB_SPACING_j ? nullptr : ia.data();
      for (long i = 0; i < cnt; ++i) out[i] = (long long)((from ? from[i] : (unsigned long long)i) * stride);
    };
    offsets(Yn_nrows, mr_b, mr_j, trm_flag ? sc : sr, trm_flag ? rs : 1, rows_j);
    for (size_t i = 0; i < rows_j.size(); ++i) row_off_a[ia[i]] = rows_j[i];
    offsets(Wn_nrows, mc_b, mc_j, trm_flag ? sr : sc, trm_flag ? 1 : rs, cols_j);
  }
  long long max_off = 0;
  for (long long o : rows_j) max_off = o > max_off ? o : max_off;
  long long max_coff = 0;
  for (long long o : cols_j) max_coff = o > max_coff ? o : max_coff;
  const size_t lf_elems = (size_t)(max_off + max_coff + 1);

  std::optional<Stager> st;
  DBuf d_lf, d_rows, d_cols, d_roff_all, d_row0, d_part, d_sc;
  const int nr = (int)rows_j.size(), nc = (int)cols_j.size();
  // A mirrored matrix (lmirror.cu) is read in place.
  Mirror *mlf = (lf_YnWt && YnWt == lf_YnWt->lf) ? find_mirror(lf_YnWt) : nullptr;
  const double *plf = nullptr;
  // Inside a deferral scope (and when no host copy of the planes is wanted)
  // min, max and mlt stay on the device: the planes kernel reads them there
  // and M_X's fields are set when the scope ends, so the call does not wait.
  const bool deferred = defer_active() && !host_planes_wanted();
  const bool values = nr > 0 && nc > 0 && YnWt;
  XcalcScalars *dev_sc = nullptr;
  int slot = -1;
  // Plane 0: the rows set in mr_j (xcalc.c:141).
  std::vector<unsigned char> row0((size_t)lakbcc::bsize(Yn_nrows), 0);
  memcpy(row0.data(), mr_j, (size_t)(Yn_nrows + 7) / 8);
  if (Yn_nrows % 8) row0[Yn_nrows / 8] &= (unsigned char)(0xFF00 >> (Yn_nrows % 8));
  // no values: min 0, max 1 before the margins (xcalc.c:34)
  double min = 0.0 - 0.0625, max = 1.0 + 0.0625, mlt = (double)g_d_mlt / (max - min);
  if (values) {
    if (mlf && lf_elems <= mlf->n) {
      plf = mlf->d;
    } else {
      d_lf = DBuf(lf_elems * sizeof(double));
      d_lf.upload(YnWt, lf_elems * sizeof(double));
      plf = d_lf.as<double>();
    }
    // The Stager lives to the end of the call: arrays of 1 MB or more go to
    // buffers it owns, which must outlive the kernels below.
    st.emplace();
    d_rows = upload_vec(rows_j);
    d_cols = upload_vec(cols_j);
    d_roff_all = upload_vec(row_off_a);
    d_row0 = upload_vec(row0);
    st->flush();
    const dim3 grid = minmax_grid(nr, nc);
    d_part = DBuf((size_t)grid.x * grid.y * sizeof(ulonglong2));
    if (deferred) {
      dev_sc = xcalc_slot(slot);
    } else {
      d_sc = DBuf(sizeof(XcalcScalars));
      dev_sc = d_sc.as<XcalcScalars>();
    }
    xcalc_minmax_kernel<false><<<grid, kMinMaxThreads, 0, stream()>>>(plf, d_rows.as<long long>(), nr,
                                                                      d_cols.as<long long>(), nc,
                                                                      d_part.as<ulonglong2>(), minmax_ticket(),
                                                                      g_d_mlt, dev_sc);
    LAKGB_CUDA(cudaGetLastError());
    count_launch();
  }

  int ncols_bZ = 0, nrows_bZ = 0;
  long long brows = 0;
  if (length > 0 && lf_YnWt != nullptr) {
    ncols_bZ = ncols_per * cpop_j;
    nrows_bZ = Yn_nrows;
    brows = lakbcc::bsize(nrows_bZ);
    const size_t nbytes = (size_t)ncols_bZ * (size_t)brows;
    if (!M_X->Ara) {
      M_X->Ara = (unsigned char *)calloc(nbytes + kBlockBytes, 1);
      if (!M_X->Ara) { set_error(2, "wrap_xcalc: out of host memory"); return; }
    }
    DBuf planes(nbytes);
    if (values) {
      XcalcParams p{};
      p.lf = plf;
      p.row_off = d_roff_all.as<long long>(); p.nrows_a = Yn_nrows;
      p.col_off = d_cols.as<long long>(); p.ncols_j = nc;
      p.dmax = (unsigned long long)(g_d_mlt - 1);
      p.sc = dev_sc;
      p.row0 = d_row0.as<uint8_t>();
      p.ncols_per = ncols_per; p.brows = brows; p.planes = planes.as<uint8_t>();
      p.row_max = max_off;
      p.lf_n = (plf == d_lf.p) ? (unsigned long long)lf_elems : (unsigned long long)mlf->n;
      p.planes_n = (unsigned long long)nbytes;
      p.bad = bad_flag();
      launch_planes(p, stream());
    } else {
      planes.zero();
      if (nbytes) planes.upload(row0.data(), (size_t)brows);
    }
    if (host_planes_wanted()) {
      if (nbytes) LAKGB_CUDA(cudaMemcpyAsync(M_X->Ara, planes.p, nbytes, cudaMemcpyDeviceToHost, stream()));
      LAKGB_CUDA(cudaStreamSynchronize(stream()));
    }
    resident_put(M_X->Ara, nbytes, std::move(planes));
  }
  if (values && !deferred) {
    XcalcScalars h;
    int hbad = 0;  // this call or an earlier one met an index outside its buffers
    LAKGB_CUDA(cudaMemcpyAsync(&hbad, bad_flag(), sizeof(int), cudaMemcpyDeviceToHost, stream()));
    LAKGB_CUDA(cudaMemcpyAsync(&h, dev_sc, sizeof h, cudaMemcpyDeviceToHost, stream()));
    LAKGB_CUDA(cudaStreamSynchronize(stream()));
    if (hbad) {
      printf(" %% Warning! wrap_xcalc: a call skipped an out-of-range index (code %d)\n", hbad);
      set_error(5, "wrap_xcalc: a call skipped an out-of-range index (code %d)", hbad);
      LAKGB_CUDA(cudaMemsetAsync(bad_flag(), 0, sizeof(int), stream()));
    }
    min = h.lo; max = h.hi; mlt = h.mlt;
  }
  // M_X fields (xcalc.c:231-241).
  M_X->nrows = ncols_bZ; M_X->ncols = nrows_bZ;
  M_X->nrows_extend = (lakbcc::BITJ - (M_X->nrows % lakbcc::BITJ)) % lakbcc::BITJ;
  M_X->mr_length = lakbcc::bsize(M_X->nrows);
  M_X->ncols_extend = (lakbcc::BITJ - (M_X->ncols % lakbcc::BITJ)) % lakbcc::BITJ;
  M_X->mc_length = lakbcc::bsize(M_X->ncols);
  memset(M_X->mr_b, 0xFF, (size_t)(ncols_bZ / 8));
  memset(M_X->mr_j, 0xFF, (size_t)(ncols_bZ / 8));
  for (int j = ncols_bZ / 8 * 8; j < ncols_bZ; ++j) { lakbcc::bset_on(M_X->mr_b, j); lakbcc::bset_on(M_X->mr_j, j); }
  M_X->rpop_b = ncols_bZ; M_X->rpop_j = ncols_bZ;
  memcpy(M_X->mc_b, mr_b, M_X->mc_length);
  memcpy(M_X->mc_j, mr_j, M_X->mc_length);
  M_X->cpop_b = rpop_b; M_X->cpop_j = rpop_j;
  M_X->wX = M_X->Ara;
  M_X->ncols_per_z = ncols_per;
  if (values && deferred) {
    t_xs.push_back(XcalcDeferred{M_X, slot});
    defer_register(xcalc_deferred_enqueue, xcalc_deferred_finish);
  } else {
    M_X->max_d = max; M_X->min_d = min; M_X->mlt_d = mlt;
    if (!isfinite(M_X->mlt_d) || M_X->mlt_d <= 0) M_X->mlt_d = 1;
  }
  lakbcc::mhandle_mxget(M_X);
}

extern "C" int lakgb_xcalc_noalloc(const struct lakgb_xcalc_noalloc_args *a) {
  if (!a || !a->planes || !a->min_max_mlt || (a->n_rows_j > 0 && a->n_cols_j > 0 && (!a->lf || !a->rows_j ||
      !a->cols_j || !a->row_off_a))) {
    set_error(2, "lakgb_xcalc_noalloc: null argument");
    return 2;
  }
  if (a->n_cols_j < 0 || a->n_rows_j < 0 || a->nrows_a < 0) {
    set_error(2, "lakgb_xcalc_noalloc: negative count (nrows_a %d, n_rows_j %d, n_cols_j %d)", a->nrows_a,
              a->n_rows_j, a->n_cols_j);
    return 2;
  }
  if (a->n_cols_j > kNoAllocMaxCols) {
    set_error(2, "lakgb_xcalc_noalloc: %d retained columns exceed the scratch limit of %d", a->n_cols_j,
              kNoAllocMaxCols);
    return 2;
  }
  if (a->b_mlt < 1 || a->b_mlt > 62 || a->d_mlt < 2) {
    set_error(2, "lakgb_xcalc_noalloc: b_mlt %d outside [1, 62] or d_mlt %lld below 2", a->b_mlt, a->d_mlt);
    return 2;
  }
  // The plane kernel stores whole 4-byte words at planes + plane * brows + 4 * w.
  if (a->brows < (long long)((a->nrows_a + 31) / 32) * 4 || (a->brows & 3) ||
      (reinterpret_cast<uintptr_t>(a->planes) & 3)) {
    set_error(2, "lakgb_xcalc_noalloc: plane rows of %lld bytes too short or not a multiple of 4, or planes "
              "not 4-byte aligned", a->brows);
    return 2;
  }
  double *scratch = noalloc_scratch();
  if (!scratch) return 3;
  cudaStream_t s = static_cast<cudaStream_t>(a->stream);
  const int ncols_per = a->b_mlt + 1;
  const size_t nbytes = (size_t)ncols_per * (size_t)a->n_cols_j * (size_t)a->brows;
  const bool values = a->n_rows_j > 0 && a->n_cols_j > 0;
  if (!values && nbytes) {
    LAKGB_CUDA(cudaMemsetAsync(a->planes, 0, nbytes, s));
    if (a->row0) LAKGB_CUDA(cudaMemcpyAsync(a->planes, a->row0, (size_t)a->brows, cudaMemcpyDeviceToDevice, s));
  }
  XcalcScalars *sc = reinterpret_cast<XcalcScalars *>(scratch + kScratchScalars);
  unsigned *ticket = reinterpret_cast<unsigned *>(scratch + kScratchTicket);
  // zeroed here, whatever calls that raced on the scratch may have left in it
  LAKGB_CUDA(cudaMemsetAsync(ticket, 0, sizeof(unsigned), s));
  const dim3 grid = minmax_grid(values ? a->n_rows_j : 0, values ? a->n_cols_j : 0);
  xcalc_minmax_kernel<true><<<grid, kMinMaxThreads, 0, s>>>(a->lf, a->rows_j, values ? a->n_rows_j : 0, a->cols_j,
                                                            values ? a->n_cols_j : 0,
                                                            reinterpret_cast<ulonglong2 *>(scratch), ticket,
                                                            (long long)a->d_mlt, sc);
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
  if (values) {
    XcalcParams p{};
    p.lf = a->lf; p.row_off = a->row_off_a; p.nrows_a = a->nrows_a;
    p.col_off = a->cols_j; p.ncols_j = a->n_cols_j;
    p.dmax = (unsigned long long)(a->d_mlt - 1); p.ncols_per = ncols_per; p.brows = a->brows;
    p.planes = a->planes; p.row0 = a->row0;
    p.sc = sc;
    p.planes_n = (unsigned long long)nbytes;
    launch_planes(p, s);
  }
  XcalcScalars h;
  LAKGB_CUDA(cudaMemcpyAsync(&h, sc, sizeof(h), cudaMemcpyDeviceToHost, s));
  LAKGB_CUDA(cudaStreamSynchronize(s));
  a->min_max_mlt[0] = h.lo;
  a->min_max_mlt[1] = h.hi;
  a->min_max_mlt[2] = (!isfinite(h.mlt) || h.mlt <= 0) ? 1.0 : h.mlt;  // the value wrap_xcalc stores
  return 0;
}
