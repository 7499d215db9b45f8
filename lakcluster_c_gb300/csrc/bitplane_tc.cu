// Bit-plane loop product At_T_YnWt_S_Zn_ww (dir_c/At_T_YnWt_S_Zn_ww.c:5-190)
// with its integer part on the tensor cores.
//
// Same outputs as bitplane_main_kernel (bitplane.cu), bit for bit.  The
// integer part is the count
//   cnt[na][q] = popcount(a'_na & plane_q)  over all patient bits,
//   a' = ~(At_na ^ Tt_t) & mask,
// for every value plane q = (Wn row mw, bit k): a GEMM over bits, M = SNP
// pairs, N = planes, K = patients.  Bits become e4m3 bytes (0x08 = 2^-6 for a
// set bit, 0 otherwise), so the fp32 accumulator in TMEM holds cnt * 2^-12
// exactly (cnt <= patients < 2^22).  The fold then forms
//   At_tmp = sum_k 2^k (2 cnt[k] - popcount(plane_k & mask))   (int64)
// and the term of (pair, Wn row),
//   ((At_base + At_tmp) / mlt - (a T_base + a T_tmp) / mlt) * vS * (vZ - aZ),
// with the reference's operations.  Only the sum of the terms over the Wn rows
// has an order: the terms of a batch go to a scratch array ([Wn row][pair], so
// both kernels' accesses coalesce) and a second kernel adds them in order, a
// thread per (pair, t).  So the tensor kernel's work splits into units of
// 128 pairs x 256 planes that any CTA may take: one CTA per 128 pairs, walking
// the Wn rows with its sums in registers, left most SMs idle below 19456 pairs
// (4096 SNPs x 1000 controls x 1024 cases, 32 bits: 32 CTAs, 1.9 ms).
//
// Persistent CTAs, one per SM.  21 warps:
//   warps 0-11  producers: per 128-patient chunk, 128 rows a' and 256 plane
//               rows, expanded to e4m3 in a 4-stage ring of 128-byte-swizzled
//               K-major tiles (16 KB + 32 KB a stage).  Chunks past the last
//               patient are skipped.
//   warp 12     owns TMEM (2 x 256 count columns); lane 0 issues the MMAs
//               (M=128, N=256, K=32), a whole unit into one count buffer.
//   warps 13-20 fold: thread = SNP pair = TMEM lane; two warps share a lane
//               quadrant, each with half of the unit's Wn rows.
// What bounds a unit: the MMAs (536 cycles a chunk) from about 10 chunks, the
// fold's FP64 operations (9 per term, 80 cycles each per warp) below.
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

constexpr int kM = 128, kN = 256;
constexpr int kStages = 4;
constexpr int kPrefetch = 3;               // producer loads in flight
constexpr int kStageA = kM * 128, kStageB = kN * 128, kStageBytes = kStageA + kStageB;
constexpr int kSBO = 1024;                 // bytes between 8-row swizzle atoms
constexpr int kProducers = kM + kN;        // warps 0-11
constexpr int kMmaWarp = kProducers / 32;  // 12
constexpr int kFold = 256;                 // warps 13-20
constexpr int kThreads = kProducers + 32 + kFold;
constexpr uint32_t kTmemCols = 512;
constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + 1024;

struct Smem {
  uint64_t full[kStages], empty[kStages];
  uint64_t acc_full[2], acc_empty[2], done;
  uint32_t tmem_base;
  int abort;
};

__device__ __forceinline__ void expand_row(uint32_t row_base, uint32_t sw, uint4 x) {
  const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t v = w[q];
    tc::st_shared_v4(row_base + (((2 * q) ^ sw) << 4), (v << 3) & 0x08080808u, (v << 2) & 0x08080808u,
                     (v << 1) & 0x08080808u, v & 0x08080808u);
    tc::st_shared_v4(row_base + (((2 * q + 1) ^ sw) << 4), (v >> 1) & 0x08080808u, (v >> 2) & 0x08080808u,
                     (v >> 3) & 0x08080808u, (v >> 4) & 0x08080808u);
  }
}

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
      s += (uint32_t)__float_as_int(__fmaf_rn(__uint_as_float(cnt[k]), 4096.0f, 12582912.0f)) << (k - k0);
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
  int pair0, w0, w1;  // Wn rows [w0, w1), at most 256 / B
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
    bitplane_tc_kernel(const BitplaneParams *__restrict__ ps, const BitplaneSeg *__restrict__ segs, int nseg, int units,
                       double *__restrict__ Y, int *status) {
  constexpr int CW = kN / B;  // Wn rows per unit
  extern __shared__ __align__(128) uint8_t dsm[];
  __shared__ Smem sm;
  uint8_t *stages = dsm + ((1024 - (tc::smem_u32(dsm) & 1023)) & 1023);

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
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = sm.tmem_base;

  if (tid < kProducers) {
    // ---------------- producers ----------------
    const bool is_a = tid < kM;
    const int rr = is_a ? tid : tid - kM;
    const uint32_t region = tc::smem_u32(stages) + (is_a ? 0 : kStageA);
    const uint32_t my_row = region + (uint32_t)((rr >> 3) * kSBO + (rr & 7) * 128);
    const uint32_t my_sw = (uint32_t)(rr & 7);
    bool ok = true;
    int s = 0, wrap = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
      const Unit un = find_unit<CW>(ps, segs, nseg, u);
      const BitplaneParams &p = *un.p;
      const int G = p.chunks;
      // this thread's row: an a' row, or value plane (mw, k) of the unit
      const uint4 *src = nullptr, *mk = nullptr, *tk = nullptr;
      if (is_a) {
        const int pr = un.pair0 + rr;
        if (pr < p.npairs) src = reinterpret_cast<const uint4 *>(p.At + (long long)p.at_rowb[pr] * p.at_row_bytes);
        mk = reinterpret_cast<const uint4 *>(p.mask);
        tk = reinterpret_cast<const uint4 *>(p.Tt + (long long)p.tt_rowb[un.s->t] * p.tt_row_bytes);
      } else {
        const int mw = un.w0 + rr / B;
        if (mw < un.w1)
          src = reinterpret_cast<const uint4 *>(p.planes + (long long)plane_row(mw, rr % B, p.ncols_per) * p.plane_bytes);
      }
      uint4 rx[kPrefetch], rm[kPrefetch], rt[kPrefetch];
      auto load = [&](int g, uint4 &x, uint4 &m, uint4 &tt) {
        x = m = tt = make_uint4(0, 0, 0, 0);
        if (g < G && src) {
          x = __ldg(src + g);
          if (is_a) {
            m = __ldg(mk + g);
            tt = __ldg(tk + g);
          }
        }
      };
#pragma unroll
      for (int v = 0; v < kPrefetch; ++v) load(v, rx[v], rm[v], rt[v]);
      for (int g0 = 0; g0 < G; g0 += kPrefetch) {
#pragma unroll
        for (int v = 0; v < kPrefetch; ++v) {
          if (g0 + v >= G) break;
          uint4 x = rx[v];
          if (is_a) {  // a' = ~(At ^ Tt) & mask (zero for a missing row: m = 0)
            const uint4 m = rm[v], tt = rt[v];
            x = make_uint4(~(x.x ^ tt.x) & m.x, ~(x.y ^ tt.y) & m.y, ~(x.z ^ tt.z) & m.z, ~(x.w ^ tt.w) & m.w);
          }
          load(g0 + v + kPrefetch, rx[v], rm[v], rt[v]);
          if (wrap > 0 && ok) ok = tc::mbar_wait(&sm.empty[s], (uint32_t)((wrap - 1) & 1), abort, status, 11);
          if (ok) {
            expand_row(my_row + s * kStageBytes, my_sw, x);
            tc::fence_proxy_async();
          }
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&sm.full[s]);
          if (++s == kStages) {
            s = 0;
            ++wrap;
          }
        }
      }
    }
  } else if (warp == kMmaWarp) {
    // ---------------- MMA issue ----------------
    if (lane == 0) {
      constexpr uint32_t idesc = tc::idesc_e4m3_f32(kM, kN);
      const uint32_t st0 = tc::smem_u32(stages);
      bool ok = true;
      int s = 0, wrap = 0, nt = 0;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x, ++nt) {
        const int G = find_unit<CW>(ps, segs, nseg, u).p->chunks;
        const int b = nt & 1;
        if (nt >= 2) ok = tc::mbar_wait(&sm.acc_empty[b], (uint32_t)(((nt >> 1) - 1) & 1), abort, status, 13);
        tc::fence_after_sync();
        for (int g = 0; g < G && ok; ++g) {
          const int cs = s;
          ok = tc::mbar_wait(&sm.full[cs], (uint32_t)(wrap & 1), abort, status, 14);
          if (++s == kStages) {
            s = 0;
            ++wrap;
          }
          if (!ok) break;
          tc::fence_after_sync();
          const uint32_t sa = st0 + cs * kStageBytes, sb = sa + kStageA;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            tc::mma_e4m3(tmem + b * kN, tc::smem_desc_sw128(sa + kk * 32, kSBO), tc::smem_desc_sw128(sb + kk * 32, kSBO),
                         idesc, (g | kk) != 0);
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
    const int q = warp & 3, half = (warp - kMmaWarp - 1) >> 2;
    const int row = 32 * q + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16);
    bool ok = true;
    int nt = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++nt) {
      const Unit un = find_unit<CW>(ps, segs, nseg, u);
      const BitplaneParams &p = *un.p;
      const int t = un.s->t, pr = un.pair0 + row, b = nt & 1;
      const bool live = pr < p.npairs;
      const double mlt = p.mlt_d, inv_mlt = p.inv_mlt;
      double At_base = 0.0;
      double2 zz = make_double2(0.0, 0.0);
      const double *q2 = p.q2;
      const uint8_t *z = p.Zt;
      if (live) {
        At_base = p.At_base[(long long)t * p.npairs + pr];
        zz = p.zz[pr];
        q2 += ((long long)t * p.nblk + p.a_blk[pr]) * p.nW;
        z += (long long)p.zt_rowb[pr] * p.zt_row_bytes;
      }
      const int8_t *vS = p.vS + (long long)t * p.nW;
      double *y = Y + un.s->y0 + pr;
      const bool w = ok && tc::mbar_wait(&sm.acc_full[b], (uint32_t)((nt >> 1) & 1), abort, status, 16);
      ok = __all_sync(0xffffffffu, w);
      tc::fence_after_sync();
#pragma unroll
      for (int i = 0; i < CW / 2; ++i) {
        const int mwl = half * (CW / 2) + i, mw = un.w0 + mwl;
        uint32_t cnt[B];
        if (p.chunks == 0) {  // no patients: no MMA has written the buffer
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
        if (i == CW / 2 - 1) {
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&sm.acc_empty[b]);
        }
        if (!(ok && live && mw < un.w1)) continue;
        const long long v = 2 * weigh_counts<B>(cnt) - __ldg(p.ysum + mw);
        const double X = __dsub_rn(div_mlt(__dadd_rn(At_base, (double)v), mlt, inv_mlt), __ldg(q2 + mw));
        const int mwa = (int)__ldg(p.mw_a + mw);
        const bool zset = (__ldg(z + (mwa >> 3)) >> (7 - (mwa & 7))) & 1;
        // times vS = +1 / -1
        const double Xs = vS[mw] < 0 ? -X : X;
        y[(long long)(mw - un.s->w0) * p.npairs] = __dmul_rn(Xs, zset ? zz.x : zz.y);
      }
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
#pragma unroll
  for (int j = 0; j < kAddAhead; ++j) a[j] = j < nw ? __ldcs(y + j * n) : 0.0;
  for (int w = 0; w < nw; w += kAddAhead) {
#pragma unroll
    for (int j = 0; j < kAddAhead; ++j) {
      if (w + j < nw) acc = __dadd_rn(acc, a[j]);
      if (w + j + kAddAhead < nw) a[j] = __ldcs(y + (long long)(w + j + kAddAhead) * n);
    }
  }
  *out = acc;
}

template <int B>
void launch_b(const BitplaneParams *ps, const BitplaneSeg *segs, const BitplaneBatch &bt, double *Y, cudaStream_t s) {
  static std::once_flag configured;
  std::call_once(configured, [] {
    LAKGB_CUDA(cudaFuncSetAttribute(bitplane_tc_kernel<B>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kSmemBytes));
  });
  bitplane_tc_kernel<B><<<std::min(bt.units, 152), kThreads, kSmemBytes, s>>>(ps, segs + bt.seg0, bt.nseg, bt.units, Y,
                                                                            tc_status_device_ptr());
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
