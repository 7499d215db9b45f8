// Bit-plane loop product At_T_YnWt_S_Zn_ww (dir_c/At_T_YnWt_S_Zn_ww.c:5-190)
// with its integer part on the tensor cores.
//
// Same outputs as bitplane_main_kernel (bitplane.cu), bit for bit.  The
// integer part is the count
//   cnt[na][q] = popcount(a'_na & plane_q)  over all patient bits,
//   a' = ~(At_na ^ Tt_t) & mask,
// for every value plane q = (Wn row mw, bit k): a GEMM over bits, M = SNP
// pairs, N = planes, K = patients.  Bits become e2m1 values (kind::mxf4, unit
// scale factors), so the fp32 accumulator in TMEM holds cnt exactly
// (cnt <= patients < 2^22).  The fold then forms
//   At_tmp = sum_k 2^k (2 cnt[k] - popcount(plane_k & mask))   (int64)
// and the term of (pair, Wn row),
//   ((At_base + At_tmp) / mlt - (a T_base + a T_tmp) / mlt) * vS * (vZ - aZ),
// with the reference's operations.  Only the sum of the terms over the Wn rows
// has an order: the terms of a batch go to a scratch array ([Wn row][pair], so
// both kernels' accesses coalesce) and a second kernel adds them in order, a
// thread per (pair, t).  So the tensor kernel's work splits into units of
// 128 pairs x 224 planes that any CTA may take: one CTA per 128 pairs, walking
// the Wn rows with its sums in registers, left most SMs idle below 19456 pairs
// (4096 SNPs x 1000 controls x 1024 cases, 32 bits: 32 CTAs, 1.9 ms; the whole
// call takes 466 us, with one e4m3 byte per bit, rows read by their own threads
// and an adding loop with a test per term 556 us).
//
// Persistent CTAs, one per SM.  20 warps:
//   warps 0-10  producers, one tile row per thread (128 rows a', then 224
//               planes): per step of 384 patients, read the row's 48 bytes
//               from the raw slot, expand to three 64-byte rows of e2m1 in one
//               of two stages (K-major, 64-byte swizzle).  Each warp brings
//               its rows' next steps into its own raw slots by cp.async, a
//               fixed (row, 16 bytes) per lane and copy (16 bytes of its own
//               row per thread took 32 wavefronts per warp load).  Steps past
//               the last patient are skipped.
//   warp 11     owns TMEM (2 x 224 count columns and the scale factors); lane 0
//               issues the MMAs (M=128, N=224, K=64), a whole unit into one
//               count buffer.
//   warps 12-19 fold: thread = SNP pair = TMEM lane; two warps share a lane
//               quadrant, each with every other Wn row of the unit.  What a
//               term needs beside its counts is read before the unit's counts
//               are waited for.
// The calls' parameters and the segments are copied to shared memory first
// where they fit: finding a unit reads them in a chain.
// What bounds a unit: the fold's FP64 operations (9 per term, 80 cycles each
// per warp: 5000 cycles) up to about 30 steps, then the MMAs.
// Every wait is bounded (tc_ptx.cuh); a pipeline error is recorded in the
// tensor-core status word read by lakgb_device_status.
#include <algorithm>
#include <mutex>

#include "bitplane.cuh"
#include "gram.cuh"
#include "lakgb_runtime.cuh"
#include "tc_ptx.cuh"

namespace lakgb {

namespace {

constexpr int kM = 128, kN = 224;
constexpr int kStages = 2;
constexpr int kChunk = 3;                  // 128-patient chunks per step
constexpr int kRawRow = 16 * kChunk;       // bytes of one row of a step
constexpr int kAhead = 3;                  // steps fetched ahead
constexpr int kRawBytes = (kM + kN) * kRawRow;
constexpr int kTileA = kM * 64, kTileB = kN * 64, kChunkBytes = kTileA + kTileB;
constexpr int kStageBytes = kChunk * kChunkBytes;
constexpr int kSBO = 512;                  // bytes between 8-row swizzle atoms
constexpr int kProducers = kM + kN;        // warps 0-10
constexpr int kMmaWarp = kProducers / 32;  // 11
constexpr int kFold = 256;                 // warps 12-19
constexpr int kThreads = kProducers + 32 + kFold;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kSfCol = 2 * kN;        // 16 columns of ones
constexpr int kParamsCached = 48, kSegsCached = 128;  // in shared memory
constexpr size_t kCacheBytes = kParamsCached * sizeof(BitplaneParams) + kSegsCached * sizeof(BitplaneSeg);
constexpr size_t kSmemBytes =
    (size_t)kStages * kStageBytes + (kAhead + 1) * kRawBytes + kCacheBytes + 1024;
static_assert(kSmemBytes <= 227 * 1024 - 256, "one CTA per SM");
static_assert(kProducers % 32 == 0 && kSfCol + 16 <= kTmemCols, "whole warps, TMEM layout");

struct Smem {
  uint64_t full[kStages], empty[kStages];
  uint64_t acc_full[2], acc_empty[2], done;
  uint32_t tmem_base;
  int abort;
};

// sum_k 2^k cnt[k] of the B counts of one Wn row: each count in the low bits
// of a float (0x4B400000 + n for n < 2^22), up to ten of them added with their
// weights in 32 bits (n 2^10 < 2^32), the floats' bits taken off at the end.
template <int B>
__device__ __forceinline__ long long weigh_counts(const uint32_t (&cnt)[B]) {
  long long v = 0;
#pragma unroll
  for (int k0 = 0; k0 < B; k0 += 10) {
    uint32_t s = 0;
#pragma unroll
    for (int k = k0; k < (k0 + 10 < B ? k0 + 10 : B); ++k)
      s += (uint32_t)__float_as_int(__fadd_rn(__uint_as_float(cnt[k]), 12582912.0f)) << (k - k0);
    s -= 0x4B400000u * ((1u << ((k0 + 10 < B ? k0 + 10 : B) - k0)) - 1u);
    v += (long long)((unsigned long long)s << k0);
  }
  return v;
}

// n / mlt, correctly rounded, from y = RN(1 / mlt): q0 = RN(n y) is within two
// units, one correction with the exact remainder makes it faithful and a
// second one gives the rounded quotient (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990, theorem
// on the final correction).  Five FP64 operations in place of the general
// division's; the caller has checked that nothing over- or underflows.
__device__ __forceinline__ double div_mlt(double n, double mlt, double y) {
  if (y == 0.0) return __ddiv_rn(n, mlt);
  double q = __dmul_rn(n, y);
  q = __fma_rn(__fma_rn(-mlt, q, n), y, q);
  return __fma_rn(__fma_rn(-mlt, q, n), y, q);
}

__device__ __forceinline__ int plane_row(int mw, int k, int ncols_per) {
  return mw * ncols_per + ncols_per - 1 - k;
}

// The unit u of a batch: its segment, pair tile and first Wn row.
struct Unit {
  const BitplaneParams *p;
  const BitplaneSeg *s;
  int pair0, w0, w1;  // Wn rows [w0, w1), at most kN / B
};
template <int CW>
__device__ __forceinline__ Unit find_unit(const BitplaneParams *ps, const BitplaneSeg *segs, int nseg, int u) {
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (segs[mid].unit0 <= u) lo = mid; else hi = mid - 1;
  }
  Unit r;
  r.s = segs + lo;
  r.p = ps + r.s->call;
  const int ptiles = (r.p->npairs + kM - 1) / kM, j = u - r.s->unit0;
  r.pair0 = (j % ptiles) * kM;
  r.w0 = r.s->w0 + (j / ptiles) * CW;
  r.w1 = min(r.w0 + CW, r.s->w1);
  return r;
}

template <int B>
__global__ void __launch_bounds__(kThreads, 1)
    bitplane_tc_kernel(const BitplaneParams *g_ps, const BitplaneSeg *g_segs, int nseg, int units,
                       double *__restrict__ Y, int *status) {
  constexpr int CW = kN / B;  // Wn rows per unit
  extern __shared__ __align__(128) uint8_t dsm[];
  __shared__ Smem sm;
  uint8_t *stages = dsm + ((1024 - (tc::smem_u32(dsm) & 1023)) & 1023);
  uint8_t *raw = stages + (size_t)kStages * kStageBytes;
  BitplaneParams *c_ps = reinterpret_cast<BitplaneParams *>(raw + (kAhead + 1) * kRawBytes);
  BitplaneSeg *c_segs = reinterpret_cast<BitplaneSeg *>(c_ps + kParamsCached);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int *abort = &sm.abort;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(&sm.full[s], kProducers / 32);  // one arrival per warp
      tc::mbar_init(&sm.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&sm.acc_full[b], 1);
      tc::mbar_init(&sm.acc_empty[b], kFold / 32);
    }
    tc::mbar_init(&sm.done, 1);
    sm.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) tc::tmem_alloc(&sm.tmem_base, kTmemCols);
  await_previous();
  const BitplaneParams *ps = g_ps;
  const BitplaneSeg *segs = g_segs;
  const int call0 = g_segs[0].call, ncalls = g_segs[nseg - 1].call - call0 + 1;
  if (nseg <= kSegsCached && ncalls <= kParamsCached) {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(g_ps + call0);
    for (int i = tid; i < ncalls * (int)(sizeof(BitplaneParams) / 4); i += kThreads)
      reinterpret_cast<uint32_t *>(c_ps)[i] = src[i];
    src = reinterpret_cast<const uint32_t *>(g_segs);
    for (int i = tid; i < nseg * (int)(sizeof(BitplaneSeg) / 4); i += kThreads)
      reinterpret_cast<uint32_t *>(c_segs)[i] = src[i];
    ps = c_ps - call0;
    segs = c_segs;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = sm.tmem_base;
  if (warp > kMmaWarp && warp <= kMmaWarp + 4) {  // unit scale factors, one warp per lane quadrant
    uint32_t ones[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) ones[i] = tc::kScaleOnes;
    tc::tmem_st16(tmem + kSfCol + ((uint32_t)(32 * (warp & 3)) << 16), ones);
    tc::tmem_wait_st();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();

  if (tid < kProducers) {
    // ---------------- producers ----------------
    const bool is_a = tid < kM;
    const int rr = is_a ? tid : tid - kM;
    const uint32_t my_row = tc::smem_u32(stages) + (is_a ? 0 : kTileA) + (uint32_t)(rr * 64);
    const uint32_t my_sw = (uint32_t)((rr >> 1) & 3);
    const uint32_t my_raw = tc::smem_u32(raw) + (uint32_t)(tid * kRawRow);
    uint8_t *my_dst = raw + (size_t)(tid & ~31) * kRawRow + 16 * lane;  // copy j: + 512 j
    // The fetching position, kAhead steps ahead of the one that is expanded:
    // its unit, the step in it and this lane's kChunk pieces of a step (copy
    // j: piece i % 3 of the warp's row i / 3, i = lane + 32 j; null: no row).
    const uint8_t *piece[kChunk];
    int fu = blockIdx.x, fstep = 0, fsteps = 0;
    auto fetch_unit = [&]() {  // the first unit from fu on that has steps
      for (fsteps = 0; fu < units; fu += gridDim.x) {
        const Unit un = find_unit<CW>(ps, segs, nseg, fu);
        const BitplaneParams &p = *un.p;
        fsteps = (p.chunks + kChunk - 1) / kChunk;
        if (!fsteps) continue;
#pragma unroll
        for (int j = 0; j < kChunk; ++j) {
          const int i = lane + 32 * j, r = (rr & ~31) + i / kChunk;
          piece[j] = nullptr;
          if (is_a) {
            const int pr = un.pair0 + r;
            if (pr < p.npairs) piece[j] = p.At + (long long)p.at_rowb[pr] * p.at_row_bytes + 16 * (i % kChunk);
          } else {
            const int mw = un.w0 + r / B;
            if (mw < un.w1)
              piece[j] = p.planes + (long long)plane_row(mw, r % B, p.ncols_per) * p.plane_bytes + 16 * (i % kChunk);
          }
        }
        return;
      }
    };
    fetch_unit();
    auto fetch = [&](int slot) {
      if (fu < units) {
#pragma unroll
        for (int j = 0; j < kChunk; ++j)
          if (piece[j]) tc::cp_async16(my_dst + (size_t)slot * kRawBytes + 512 * j, piece[j] + (long long)fstep * kRawRow);
        if (++fstep == fsteps) {
          fstep = 0;
          fu += gridDim.x;
          fetch_unit();
        }
      }
      tc::cp_async_commit();
    };
    for (int j = 0; j < kAhead; ++j) fetch(j);
    bool ok = true;
    int s = 0, wrap = 0, slot = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
      const Unit un = find_unit<CW>(ps, segs, nseg, u);
      const BitplaneParams &p = *un.p;
      const int steps = (p.chunks + kChunk - 1) / kChunk;
      const bool live = is_a ? un.pair0 + rr < p.npairs : un.w0 + rr / B < un.w1;
      const uint4 *mk = reinterpret_cast<const uint4 *>(p.mask);
      const uint4 *tk = reinterpret_cast<const uint4 *>(p.Tt + (long long)p.tt_rowb[un.s->t] * p.tt_row_bytes);
      for (int st = 0; st < steps; ++st) {
        // into the slot read before this step
        fetch(slot ? slot - 1 : kAhead);
        uint4 x[kChunk], m[kChunk], tt[kChunk];
#pragma unroll
        for (int v = 0; v < kChunk; ++v) {
          if (is_a) {
            m[v] = __ldg(mk + st * kChunk + v);
            tt[v] = __ldg(tk + st * kChunk + v);
          }
        }
        tc::cp_async_wait<kAhead>();
        __syncwarp();
#pragma unroll
        for (int v = 0; v < kChunk; ++v) x[v] = tc::ld_shared_v4(my_raw + slot * kRawBytes + 16 * v);
        if (wrap > 0 && ok) ok = tc::mbar_wait(&sm.empty[s], (uint32_t)((wrap - 1) & 1), abort, status, 11);
        if (ok) {
          const uint32_t dst = my_row + s * kStageBytes;
#pragma unroll
          for (int v = 0; v < kChunk; ++v) {
            // a missing row's slot holds no data: zeros
            if (!live) x[v] = make_uint4(0u, 0u, 0u, 0u);
            if (is_a) {  // a' = ~(At ^ Tt) & mask
              if (live)
                x[v] = make_uint4(~(x[v].x ^ tt[v].x) & m[v].x, ~(x[v].y ^ tt[v].y) & m[v].y,
                                  ~(x[v].z ^ tt[v].z) & m[v].z, ~(x[v].w ^ tt[v].w) & m[v].w);
              tc::expand_e2m1<0>(dst + v * kChunkBytes, my_sw, x[v]);
            } else {
              tc::expand_e2m1<1>(dst + v * kChunkBytes, my_sw, x[v]);
            }
          }
          tc::fence_proxy_async();
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&sm.full[s]);
        if (++s == kStages) {
          s = 0;
          ++wrap;
        }
        if (++slot == kAhead + 1) slot = 0;
      }
    }
    tc::cp_async_wait<0>();
  } else if (warp == kMmaWarp) {
    // ---------------- MMA issue ----------------
    if (lane == 0) {
      constexpr uint32_t idesc = tc::idesc_mxf4_f32(kM, kN);
      const uint32_t st0 = tc::smem_u32(stages);
      bool ok = true;
      int s = 0, wrap = 0, nt = 0;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x, ++nt) {
        const int steps = (find_unit<CW>(ps, segs, nseg, u).p->chunks + kChunk - 1) / kChunk;
        const int b = nt & 1;
        if (nt >= 2) ok = tc::mbar_wait(&sm.acc_empty[b], (uint32_t)(((nt >> 1) - 1) & 1), abort, status, 13);
        tc::fence_after_sync();
        for (int g = 0; g < steps && ok; ++g) {
          const int cs = s;
          ok = tc::mbar_wait(&sm.full[cs], (uint32_t)(wrap & 1), abort, status, 14);
          if (++s == kStages) {
            s = 0;
            ++wrap;
          }
          if (!ok) break;
          tc::fence_after_sync();
#pragma unroll
          for (int v = 0; v < kChunk; ++v) {
            const uint32_t sa = st0 + cs * kStageBytes + v * kChunkBytes, sb = sa + kTileA;
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
              tc::mma_mxf4(tmem + b * kN, tc::smem_desc_sw64(sa + kk * 32, kSBO), tc::smem_desc_sw64(sb + kk * 32, kSBO),
                           idesc, tmem + kSfCol, tmem + kSfCol + 4, (g | v | kk) != 0);
          }
          tc::mma_commit(&sm.empty[cs]);
        }
        if (ok) tc::mma_commit(&sm.acc_full[b]);
      }
      tc::mma_commit(&sm.done);
      const unsigned long long t0 = tc::globaltimer();
      while (!tc::mbar_try(&sm.done, 0)) {
        if (tc::globaltimer() - t0 > tc::g_wait_ns) {
          atomicCAS(status, 0, 15);
          break;
        }
      }
    }
  } else {
    // ---------------- fold: thread = SNP pair ----------------
    constexpr int kBatch = 4;  // Wn rows whose scalars are read together
    const int q = warp & 3, half = (warp - kMmaWarp - 1) >> 2;
    const int row = 32 * q + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16);
    bool ok = true;
    int nt = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++nt) {
      const Unit un = find_unit<CW>(ps, segs, nseg, u);
      const BitplaneParams &p = *un.p;
      const int t = un.s->t, b = nt & 1;
      const bool live = un.pair0 + row < p.npairs;
      const int pr = live ? un.pair0 + row : p.npairs - 1;
      const double mlt = p.mlt_d, inv_mlt = p.inv_mlt;
      const double At_base = __ldg(p.At_base + (long long)t * p.npairs + pr);
      const double2 zz = __ldg(p.zz + pr);
      const double *q2 = p.q2 + ((long long)t * p.nblk + __ldg(p.a_blk + pr)) * p.nW;
      const uint8_t *z = p.Zt + (long long)__ldg(p.zt_rowb + pr) * p.zt_row_bytes;
      const int8_t *vS = p.vS + (long long)t * p.nW;
      const long long *ysum = p.ysum;
      const uint32_t *mw_a = p.mw_a;
      const long long n = p.npairs;
      const bool counts = p.chunks > 0;
      double *y = Y + un.s->y0 + pr;
      const int w_seg = un.s->w0;
      bool waited = false;
#pragma unroll 1
      for (int i0 = half; i0 < CW; i0 += 2 * kBatch) {
        long long ys[kBatch];
        double sub[kBatch], f[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const int mw = min(un.w0 + i0 + 2 * i, un.w1 - 1);
          ys[i] = __ldg(ysum + mw);
          sub[i] = __ldg(q2 + mw);
          const int mwa = (int)__ldg(mw_a + mw);
          const bool zset = (__ldg(z + (mwa >> 3)) >> (7 - (mwa & 7))) & 1;
          // (X vS) (vZ - aZ) = X (vS (vZ - aZ)): the sign is exact
          const double zf = zset ? zz.x : zz.y;
          f[i] = __ldg(vS + mw) < 0 ? -zf : zf;
        }
        if (!waited) {
          const bool w = ok && tc::mbar_wait(&sm.acc_full[b], (uint32_t)((nt >> 1) & 1), abort, status, 16);
          ok = __all_sync(0xffffffffu, w);
          tc::fence_after_sync();
          waited = true;
        }
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const int mwl = i0 + 2 * i, mw = un.w0 + mwl;
          if (mwl >= CW) break;
          uint32_t cnt[B];
          if (!counts) {  // no patients: no MMA has written the buffer
#pragma unroll
            for (int k = 0; k < B; ++k) cnt[k] = 0u;
          } else if (ok) {
            const uint32_t col = lane_base + b * kN + mwl * B;
            if constexpr (B == 32) {
              tc::tmem_ld32(col, cnt);
            } else if constexpr (B == 16) {
              tc::tmem_ld16(col, cnt);
            } else {
              tc::tmem_ld8(col, cnt);
            }
            tc::tmem_wait_ld();
            tc::reg_fence(cnt);
          }
          if (!(ok && live && mw < un.w1)) continue;
          const long long v = 2 * weigh_counts<B>(cnt) - ys[i];
          const double X = __dsub_rn(div_mlt(__dadd_rn(At_base, (double)v), mlt, inv_mlt), sub[i]);
          y[(long long)(mw - w_seg) * n] = __dmul_rn(X, f[i]);
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&sm.acc_empty[b]);
    }
  }

  tc::fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) {
    __syncwarp();
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, kTmemCols);
  }
}

// The terms of every (pair, t) of a batch added in Wn order, thread per pair,
// carrying the sum on from the output where the segment does not start at the
// first Wn row.  A chain of one FP64 add (80 cycles) per term: small blocks
// put the few warps of a small call on as many SMs.
// Not started while the tensor kernel runs: its blocks were then packed onto the
// first SMs that fall free, many to an FP64 pipe (the 4096 x 1000 x 1024 product
// took 240 us longer).
constexpr int kAddThreads = 32, kAddAhead = 16;
__global__ void __launch_bounds__(kAddThreads)
    bitplane_add_kernel(const BitplaneParams *__restrict__ ps, const BitplaneSeg *__restrict__ segs, int nseg,
                        const double *__restrict__ Y) {
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (segs[mid].block0 <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const BitplaneSeg &s = segs[lo];
  const BitplaneParams &p = ps[s.call];
  const int pr = ((int)blockIdx.x - s.block0) * kAddThreads + threadIdx.x;
  if (pr >= p.npairs) return;
  double *out = p.out + p.out_off[pr] + p.t_off[s.t];
  double acc = s.w0 ? *out : 0.0;
  const double *y = Y + s.y0 + pr;
  const long long n = p.npairs;
  const int nw = s.w1 - s.w0;
  double a[kAddAhead];
  int w = 0;
  if (nw >= kAddAhead) {
#pragma unroll
    for (int j = 0; j < kAddAhead; ++j) a[j] = __ldcs(y + j * n);
    for (; w + 2 * kAddAhead <= nw; w += kAddAhead) {
      const double *next = y + (long long)(w + kAddAhead) * n;
#pragma unroll
      for (int j = 0; j < kAddAhead; ++j) {
        acc = __dadd_rn(acc, a[j]);
        a[j] = __ldcs(next + j * n);
      }
    }
#pragma unroll
    for (int j = 0; j < kAddAhead; ++j) acc = __dadd_rn(acc, a[j]);
    w += kAddAhead;
  }
  for (; w < nw; ++w) acc = __dadd_rn(acc, __ldcs(y + (long long)w * n));
  *out = acc;
}

template <int B>
void launch_b(const BitplaneParams *ps, const BitplaneSeg *segs, const BitplaneBatch &bt, double *Y, cudaStream_t s) {
  static std::once_flag configured;
  std::call_once(configured, [] {
    LAKGB_CUDA(cudaFuncSetAttribute(bitplane_tc_kernel<B>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kSmemBytes));
  });
  launch_after(bitplane_tc_kernel<B>, std::min(bt.units, 152), kThreads, kSmemBytes, s, ps, segs + bt.seg0, bt.nseg,
               bt.units, Y, tc_status_device_ptr());
  LAKGB_CUDA(cudaGetLastError());
  bitplane_add_kernel<<<bt.blocks, kAddThreads, 0, s>>>(ps, segs + bt.seg0, bt.nseg, Y);
  LAKGB_CUDA(cudaGetLastError());
  count_launch(2);
}

}  // namespace

size_t bitplane_tc_plan(int B, const std::vector<BitplaneParams> &ps, std::vector<BitplaneSeg> *segs,
                        std::vector<BitplaneBatch> *batches) {
  const int CW = kN / B;
  size_t used = 0, most = 0;
  BitplaneBatch bt{};
  auto close = [&] {
    most = std::max(most, used);
    if (bt.nseg) batches->push_back(bt);
    bt = BitplaneBatch{};
    bt.seg0 = (int)segs->size();
    used = 0;
  };
  for (int c = 0; c < (int)ps.size(); ++c) {
    const BitplaneParams &p = ps[c];
    const int ptiles = (p.npairs + kM - 1) / kM;
    const size_t step = (size_t)p.npairs * CW;  // terms of one N tile of Wn rows
    for (int t = 0; t < p.nT; ++t)
      for (int w0 = 0; w0 < p.nW;) {
        const int tiles_left = (p.nW - w0 + CW - 1) / CW;
        size_t fit = used < kBitplaneScratch ? (kBitplaneScratch - used) / step : 0;
        // a segment that carries another one's sums on is in a later batch;
        // an empty batch takes at least one step
        if (w0 && bt.nseg) fit = 0;
        if (!fit) {
          if (bt.nseg) {
            close();
            continue;
          }
          fit = 1;
        }
        const int tiles = (int)std::min<size_t>(fit, tiles_left);
        const int w1 = std::min(p.nW, w0 + tiles * CW);
        segs->push_back(BitplaneSeg{c, t, w0, w1, bt.units, bt.blocks, (long long)used});
        ++bt.nseg;
        bt.units += ptiles * tiles;
        bt.blocks += (p.npairs + kAddThreads - 1) / kAddThreads;
        used += step * tiles;
        w0 = w1;
      }
  }
  close();
  return most;
}

void launch_bitplane_tc(int B, const BitplaneParams *d_ps, const BitplaneSeg *d_segs,
                        const std::vector<BitplaneBatch> &batches, double *scratch, cudaStream_t s) {
  for (const BitplaneBatch &bt : batches) {
    if (B == 32)
      launch_b<32>(d_ps, d_segs, bt, scratch, s);
    else if (B == 16)
      launch_b<16>(d_ps, d_segs, bt, scratch, s);
    else
      launch_b<8>(d_ps, d_segs, bt, scratch, s);
  }
}

}  // namespace lakgb
