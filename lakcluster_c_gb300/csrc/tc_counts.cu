// Bit-pair counts of 128 x 64 tiles on the tensor cores, for products whose
// launches are too small for the persistent Gram kernel (gram_tc.cu) or have
// no per-block FP64 fold:
//
//   gram_counts_tc_kernel  the counts of a span of 1920-column blocks per CTA,
//       written as 16-bit integers to scratch.  A Gram weighs its blocks, so its
//       spans are single blocks; gram_fold_kernel then adds each element's
//       weighted counts in block order.  For launches of few tiles: every
//       (tile, block) pair is its own CTA, where one CTA per tile would walk all
//       blocks alone while most SMs idle.
//   attyn_tc_kernel        AtTYn_vv / AtTAn_vv (dir_c/AtTYn_vv.c:5-202,
//       dir_c/AtTAn_vv.c:5-172): the counts of ((At ^ Tt) & mask) xor Yt over
//       all blocks stay in TMEM, and the epilogue forms the outputs.
//
// A bit becomes one e2m1 value (tc_ptx.cuh, kind::mxf4 with unit scale
// factors); the fp32 accumulators hold n = popcount(a & z) exactly (< 2^24),
// and an XOR count is pa + pz - 2 n with the rows' own counts.
//
// CTA of 256 threads, two per SM, so that one expands while the other's MMAs,
// loads or stores run; inside a CTA the phases follow one another: rows of a
// block into shared memory by coalesced cp.async, three groups of five
// 128-column chunks expanded (a thread per row and chunk) and multiplied, the
// row counts taken while the last group's MMAs run.  Every wait is bounded
// (tc_ptx.cuh); a pipeline error is recorded in the tensor-core status word.
#include <algorithm>

#include "fixed_fp64.cuh"
#include "gram.cuh"
#include "lakgb_runtime.cuh"
#include "tc_counts.cuh"
#include "tc_ptx.cuh"
#include "weigh.cuh"

namespace lakgb {

namespace {

constexpr int kM = kCountsM, kN = kCountsN, kRows = kM + kN;
constexpr int kThreads = 256;
constexpr int kRow = kBlockBytes;         // bytes of one row of a block
constexpr int kChunks = 15, kGroup = 5;   // 128-column chunks per block, per stage
constexpr int kTileA = kM * 64, kTileB = kN * 64, kChunkBytes = kTileA + kTileB;
constexpr int kSBO = 8 * 64;
constexpr uint32_t kTmemCols = 128, kSfCol = 64;
constexpr int kStageBytes = kGroup * kChunkBytes;
constexpr int kSpanMax = 65535 / kBlockBits;  // blocks whose counts fit 16 bits
constexpr int kExactBlocks = (1 << 24) / kBlockBits;  // whole blocks whose counts an fp32 sum holds exactly
constexpr size_t kSmemBytes = 1024 + kStageBytes + (size_t)kRows * kRow + 2 * 256 + kRows * (8 + 4);
static_assert(2 * (kSmemBytes + 1024 + 64) <= 228 * 1024, "two CTAs per SM");

// The rows of one tile: A rows are masked, and xored with `xrow` first if it
// is given; Z rows enter as they are (masked for their counts only).
struct TileRows {
  const uint8_t *wA; const uint32_t *a_rowb; int nA; long long a_row_bytes;
  const uint8_t *wZ; const uint32_t *z_rowb; int nZ; long long z_row_bytes;
  const uint8_t *mask, *xrow;
};

struct Smem {
  uint64_t done;
  uint32_t tmem_base;
  int abort;
};

// One CTA's shared memory and the position in its one barrier.
struct Tile {
  Smem *sm;
  uint8_t *stage, *raw, *mask, *xrow;
  long long *off;   // byte offset of each row in its matrix, -1 past the end
  int *cnt;         // row counts
  uint32_t tmem, phase;
  bool ok;

  __device__ __forceinline__ void setup(Smem *s, uint8_t *dsm, const TileRows &t, int m0, int n0) {
    sm = s;
    stage = dsm + ((1024 - (tc::smem_u32(dsm) & 1023)) & 1023);
    raw = stage + kStageBytes;
    mask = raw + kRows * kRow;
    xrow = mask + 256;
    off = reinterpret_cast<long long *>(xrow + 256);
    cnt = reinterpret_cast<int *>(off + kRows);
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
      tc::mbar_init(&sm->done, 1);
      sm->abort = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc::tmem_alloc(&sm->tmem_base, kTmemCols);
    for (int r = tid; r < kRows; r += kThreads) {
      const int i = m0 + r, k = n0 + r - kM;
      off[r] = r < kM ? (i < t.nA ? (long long)t.a_rowb[i] * t.a_row_bytes : -1)
                      : (k < t.nZ ? (long long)t.z_rowb[k] * t.z_row_bytes : -1);
      cnt[r] = 0;
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    tmem = sm->tmem_base;
    phase = 0;
    ok = true;
    if (warp < 4) {  // unit scale factors, one warp per lane quadrant
      uint32_t ones[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) ones[i] = tc::kScaleOnes;
      tc::tmem_st16(tmem + kSfCol + ((uint32_t)(32 * warp) << 16), ones);
      tc::tmem_wait_st();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
  }

  // Every MMA issued so far has completed (all threads call it).
  __device__ __forceinline__ void wait_mma(int *status) {
    const bool w = ok && tc::mbar_wait(&sm->done, (phase - 1) & 1, &sm->abort, status, 21);
    ok = __syncthreads_and(w);
    tc::fence_after_sync();
  }

  // Count block b: the accumulators become (first) or gain its counts, the row
  // counts likewise.  On return the MMAs may still run.
  // ROWS: tile rows in use (kM and some Z rows).
  template <int ROWS>
  __device__ __forceinline__ void block(const TileRows &t, int b, bool first, bool more_before, int *status) {
    const int tid = threadIdx.x;
    const long long boff = (long long)b * kRow;
    for (int i = tid; i < ROWS * kChunks; i += kThreads) {
      const int r = i / kChunks, v = i - r * kChunks;
      const long long o = off[r];
      if (o >= 0) tc::cp_async16(raw + r * kRow + 16 * v, (r < kM ? t.wA : t.wZ) + o + boff + 16 * v);
    }
    if (tid < kChunks) {
      tc::cp_async16(mask + 16 * tid, t.mask + boff + 16 * tid);
      if (t.xrow) tc::cp_async16(xrow + 16 * tid, t.xrow + boff + 16 * tid);
    }
    tc::cp_async_commit();
    tc::cp_async_wait<0>();
    __syncthreads();
    const uint32_t st = tc::smem_u32(stage), rw = tc::smem_u32(raw), mk = tc::smem_u32(mask), xr = tc::smem_u32(xrow);
    for (int g = 0; g < kChunks / kGroup; ++g) {
      if (g > 0 || more_before) wait_mma(status);
      for (int i = tid; i < ROWS * kGroup; i += kThreads) {
        const int u = i / ROWS, r = i - u * ROWS, ch = g * kGroup + u;
        uint4 x = tc::ld_shared_v4(rw + r * kRow + 16 * ch);
        const uint32_t dst = st + u * kChunkBytes;
        if (r < kM) {
          const uint4 m = tc::ld_shared_v4(mk + 16 * ch);
          if (t.xrow) {
            const uint4 q = tc::ld_shared_v4(xr + 16 * ch);
            x = make_uint4(x.x ^ q.x, x.y ^ q.y, x.z ^ q.z, x.w ^ q.w);
          }
          x = make_uint4(x.x & m.x, x.y & m.y, x.z & m.z, x.w & m.w);
          tc::expand_e2m1<0>(dst + r * 64, (r >> 1) & 3, x);
        } else {
          tc::expand_e2m1<1>(dst + kTileA + (r - kM) * 64, (r >> 1) & 3, x);
        }
      }
      tc::fence_proxy_async();
      __syncthreads();
      if (tid == 0) {
        tc::fence_after_sync();
        constexpr uint32_t idesc = tc::idesc_mxf4_f32(kM, kN);
#pragma unroll 1
        for (int u = 0; u < kGroup; ++u)
#pragma unroll
          for (int kk = 0; kk < 2; ++kk)
            tc::mma_mxf4(tmem, tc::smem_desc_sw64(st + u * kChunkBytes + kk * 32, kSBO),
                         tc::smem_desc_sw64(st + u * kChunkBytes + kTileA + kk * 32, kSBO), idesc, tmem + kSfCol,
                         tmem + kSfCol + 4, !(first && g == 0 && u == 0 && kk == 0));
        tc::mma_commit(&sm->done);
      }
      ++phase;
    }
    // the row counts, while the last group's MMAs run
    if (tid < ROWS) {
      int c = 0;
#pragma unroll 5
      for (int ch = 0; ch < kChunks; ++ch) {
        uint4 x = tc::ld_shared_v4(rw + tid * kRow + 16 * ch);
        const uint4 m = tc::ld_shared_v4(mk + 16 * ch);
        if (t.xrow && tid < kM) {
          const uint4 q = tc::ld_shared_v4(xr + 16 * ch);
          x = make_uint4(x.x ^ q.x, x.y ^ q.y, x.z ^ q.z, x.w ^ q.w);
        }
        c += __popc(x.x & m.x) + __popc(x.y & m.y) + __popc(x.z & m.z) + __popc(x.w & m.w);
      }
      cnt[tid] += c;
    }
    __syncthreads();  // the raw rows have been read
  }

  // This warp's NC columns of the accumulators (the lane's row).
  template <int NC>
  __device__ __forceinline__ void read(uint32_t (&v)[NC]) {
    const int warp = threadIdx.x >> 5;
    const uint32_t at = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + NC * (warp >> 2);
    if constexpr (NC == 32) tc::tmem_ld32(at, v);
    else tc::tmem_ld8(at, v);
    tc::tmem_wait_ld();
    tc::reg_fence(v);
  }

  __device__ __forceinline__ void finish() {
    // after a wait that ran out: every MMA issued has completed before the
    // tensor and shared memory go (within the same time limit)
    if (!ok && phase) tc::mbar_wait_landed(&sm->done, (phase - 1) & 1);
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) {
      tc::fence_after_sync();
      tc::tmem_dealloc(tmem, kTmemCols);
    }
  }
};

__device__ __forceinline__ int decode_count(uint32_t bits) {
  return (int)__float2int_rn(__uint_as_float(bits));
}

// Span blockIdx.z: blocks [span * z, span * z + span) of p.P, span <= kSpanMax.
template <int TYPE>
__global__ void __launch_bounds__(kThreads, 2)
    gram_counts_tc_kernel(GramParams p, int span, uint16_t *__restrict__ out, uint16_t *__restrict__ zcnt, int *status) {
  extern __shared__ __align__(128) uint8_t dsm[];
  __shared__ Smem sm;
  const int m0 = blockIdx.y * kM, n0 = blockIdx.x * kN, b = blockIdx.z;
  release_next();
  if (p.symmetric && m0 > n0 + kN - 1) return;  // no pair i <= k
  const TileRows t{p.wA, p.a_rowb, p.nA, p.a_row_bytes, p.wZ, p.z_rowb, p.nZ, p.z_row_bytes, p.mask, nullptr};
  Tile tile;
  tile.setup(&sm, dsm, t, m0, n0);
  const int b0 = span * b;
  for (int k = b0; k < min(p.P, b0 + span); ++k) tile.block<kRows>(t, k, k == b0, k > b0, status);
  tile.wait_mma(status);
  if (zcnt && m0 == 0 && threadIdx.x < kN && n0 + (int)threadIdx.x < p.nZ)
    zcnt[(size_t)b * p.nZ + n0 + threadIdx.x] = (uint16_t)tile.cnt[kM + threadIdx.x];
  if (tile.ok) {
    uint32_t v[32];
    tile.read(v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = 32 * (warp & 3) + lane, c0 = 32 * (warp >> 2), i = m0 + row;
    if (i < p.nA) {
      const int pa = tile.cnt[row];
      uint16_t *o = out + ((size_t)b * p.nZ + n0 + c0) * p.nA + i;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int n = decode_count(v[j]);
        const int c = TYPE == 1 ? pa + tile.cnt[kM + c0 + j] - 2 * n : n;
        if (n0 + c0 + j < p.nZ) o[(size_t)j * p.nA] = (uint16_t)c;
      }
    }
  }
  tile.finish();
}

// The weighted counts of every element added over the blocks in order, then
// the score combine, in the reference's operation order.  A block costs a thread
// an add and what it waits for its count and weight: with few elements that wait
// is the kernel (128 x 112 elements, 5000 blocks: a call of 2984 us with loads
// that follow one another, 1596 with four blocks' ahead), with many the integer
// operations (500 x 500 x 69 blocks: 151 us, 127 with the FP64 multiply of odd
// weights out of line; 129 with eight blocks ahead).
constexpr int kFoldAhead = 4;
template <int TYPE>
__global__ void __launch_bounds__(256) gram_fold_kernel(GramParams p, const uint16_t *__restrict__ cnt) {
  const size_t n = (size_t)p.nA * p.nZ;
  const int ga = blockIdx.x * blockDim.x + threadIdx.x;
  await_previous();
  if (ga >= p.nA) return;
  for (int gz = blockIdx.y * blockDim.y + threadIdx.y; gz < p.nZ; gz += gridDim.y * blockDim.y) {
    if (p.symmetric && ga > gz) continue;
    const uint16_t *ce = cnt + (size_t)gz * p.nA + ga;
    double acc = 0.0;
    if (!p.D) {  // unit weights: integers below 2^53
      long long s = 0;
      for (int b = 0; b < p.P; ++b) s += ce[(size_t)b * n];
      acc = (double)s;
    } else {
      // the multiplies in integers, beside the adds that have to be FP64; the
      // counts and weights of the next kFoldAhead blocks are on their way while
      // these are added
      int b = 0;
      if (p.P >= 2 * kFoldAhead) {
        uint32_t c[kFoldAhead];
        double d[kFoldAhead], x[kFoldAhead];
        auto load = [&](int from) {
#pragma unroll
          for (int u = 0; u < kFoldAhead; ++u) {
            c[u] = ce[(size_t)(from + u) * n];
            d[u] = __ldg(p.D + from + u);
          }
        };
        auto weigh_all = [&]() {
#pragma unroll
          for (int u = 0; u < kFoldAhead; ++u) x[u] = times_count(d[u], c[u]);
        };
        auto add_all = [&]() {
#pragma unroll
          for (int u = 0; u < kFoldAhead; ++u) acc = __dadd_rn(acc, x[u]);
        };
        load(0);
        for (; b + 2 * kFoldAhead <= p.P; b += kFoldAhead) {
          weigh_all();
          load(b + kFoldAhead);
          add_all();
        }
        weigh_all();
        add_all();
        b += kFoldAhead;
      }
#pragma unroll 4
      for (; b < p.P; ++b) acc = __dadd_rn(acc, times_count(__ldg(p.D + b), ce[(size_t)b * n]));
    }
    double o = acc;
    if (TYPE == 1)
      o = __dsub_rn(p.a0d1, __longlong_as_double((long long)fixed::twice_bits((unsigned long long)__double_as_longlong(acc))));
    if (p.lfA && p.lfZ) o = __dsub_rn(o, __dsub_rn(__dadd_rn(p.lfA[ga], p.lfZ[gz]), p.a2d1));
    p.out[(long long)p.out_r[ga] + (long long)p.out_c[gz] * p.out_stride] = o;
    if (p.symmetric) p.out[(long long)p.out_r2[gz] + (long long)p.out_c2[ga] * p.out_stride] = o;
  }
}

// v as a double (the conversion is an instruction of the FP64 pipe).
__device__ __forceinline__ double int_to_double(int v) {
  const uint32_t n = v < 0 ? 0u - (uint32_t)v : (uint32_t)v;
  const int z = __clz((int)n);
  const uint32_t m = n << (z & 31);
  const uint32_t hi = ((uint32_t)v & 0x80000000u) | (((uint32_t)(1053 - z) << 20) + (m >> 11));
  return n ? __hiloint2double((int)hi, (int)(m << 21)) : 0.0;
}

// out = ((hhAY - hhAy aY) - aA hhaY) + (aA hhay) aY.  A thread holds one At row
// and NC Yt rows: where a warp's rows share aA and its columns share aY (both
// change once per 1920 SNPs) the products with aY are formed once and aA hhaY
// of the NC Yt rows one per lane, so an element costs three FP64 operations
// instead of seven.  Those bound a CTA's time (80 cycles a warp each), so a
// product of few tiles takes NC = 8: four times as many CTAs with a quarter of
// the elements each.
template <int NC>
__global__ void __launch_bounds__(kThreads, 2) attyn_tc_kernel(AtTYnParams p, int *status) {
  extern __shared__ __align__(128) uint8_t dsm[];
  __shared__ Smem sm;
  const int m0 = blockIdx.y * kM, n0 = blockIdx.x * 2 * NC, t = blockIdx.z;
  if (p.symmetric && m0 > n0 + 2 * NC - 1) return;
  const TileRows rows{p.At, p.a_rowb, p.nA, p.a_row_bytes, p.Yt, p.y_rowb, min(p.nY, n0 + 2 * NC), p.y_row_bytes, p.mask,
                      p.Tt + (long long)p.t_rowb[t] * p.t_row_bytes};
  Tile tile;
  tile.setup(&sm, dsm, rows, m0, n0);
  int n[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) n[j] = 0;
  // kExactBlocks blocks at a time: their counts stay below 2^24
  for (int b0 = 0; b0 < p.P; b0 += kExactBlocks) {
    for (int b = b0; b < min(p.P, b0 + kExactBlocks); ++b) tile.block<kM + 2 * NC>(rows, b, b == b0, b > b0, status);
    tile.wait_mma(status);
    if (tile.ok) {
      uint32_t v[NC];
      tile.read(v);
#pragma unroll
      for (int j = 0; j < NC; ++j) n[j] += decode_count(v[j]);
    }
    tc::fence_before_sync();
    __syncthreads();  // read before the next blocks' MMAs overwrite them
  }
  if (tile.ok) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = 32 * (warp & 3) + lane, c0 = NC * (warp >> 2), na = m0 + row;
    const bool live = na < p.nA;
    const int nac = live ? na : p.nA - 1;  // every lane takes part in the votes
    const double aA = p.aA[nac], hhAy = p.hhAy[(long long)t * p.nA + nac];
    const double aAh = __dmul_rn(aA, p.hhay[t]);
    const unsigned long long oa = p.out_a[nac] + p.out_t[t];
    const long long base = 2ll * tile.cnt[row] - p.cpop;
    // this warp's Yt rows, one per lane, in the operand tiles' shared memory
    // (the MMAs have read them): hhaY, aY and aA hhaY
    double *y = reinterpret_cast<double *>(tile.stage) + 96 * warp;
    const int nyl = min(n0 + c0 + min(lane, NC - 1), p.nY - 1);
    const double aYl = p.aY[nyl], hhaYl = p.hhaY[(long long)t * p.nY + nyl];
    y[lane] = hhaYl;
    y[32 + lane] = aYl;
    y[64 + lane] = __dmul_rn(aA, hhaYl);
    __syncwarp();
    const long long aA0 = __shfl_sync(0xffffffffu, __double_as_longlong(aA), 0);
    const long long aY0 = __shfl_sync(0xffffffffu, __double_as_longlong(aYl), 0);
    // (counts below 2^30 for the conversion)
    const bool shared = __all_sync(0xffffffffu, __double_as_longlong(aA) == aA0 && __double_as_longlong(aYl) == aY0) &&
                        p.P < (1 << 30) / (2 * kBlockBits);
    auto store = [&](int j, double o) {
      const int ny = n0 + c0 + j;
      if (live && ny < p.nY && !(p.symmetric && na > ny)) {
        p.out[oa + p.out_y[ny]] = o;
        if (p.symmetric) p.out[p.out_a2[ny] + p.out_y2[na] + p.out_t[t]] = o;
      }
    };
    // hhAY = 2 (pa + py - 2 n) - cpop
    if (shared) {
      const double q1 = __dmul_rn(hhAy, aYl), q3 = __dmul_rn(aAh, aYl);
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const double hhAY = int_to_double((int)base + 2 * tile.cnt[kM + c0 + j] - 4 * n[j]);
        store(j, __dadd_rn(__dsub_rn(__dsub_rn(hhAY, q1), y[64 + j]), q3));
      }
    } else {
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const volatile double *yj = y + j;  // read here: no FP64 operation above the branch
        const double aY = yj[32], hhAY = (double)(base + 2ll * tile.cnt[kM + c0 + j] - 4ll * n[j]);
        store(j, __dadd_rn(__dsub_rn(__dsub_rn(hhAY, __dmul_rn(hhAy, aY)), __dmul_rn(aA, yj[0])), __dmul_rn(aAh, aY)));
      }
    }
  }
  tile.finish();
}

template <class K>
void allow_smem(K kernel) {
  LAKGB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
}

template <int TYPE>
void launch_counts(const GramParams &p, int span, uint16_t *cnt, uint16_t *zcnt, cudaStream_t s) {
  static const bool configured = [] {
    allow_smem(gram_counts_tc_kernel<TYPE>);
    return true;
  }();
  (void)configured;
  const dim3 grid((p.nZ + kN - 1) / kN, (p.nA + kM - 1) / kM, (p.P + span - 1) / span);
  gram_counts_tc_kernel<TYPE><<<grid, kThreads, kSmemBytes, s>>>(p, span, cnt, zcnt, tc_status_device_ptr());
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
}

template <int TYPE>
void launch_split_type(const GramParams &p, uint16_t *cnt, cudaStream_t s) {
  launch_counts<TYPE>(p, 1, cnt, nullptr, s);
  const int bx = std::min(256, (p.nA + 31) / 32 * 32), by = 256 / bx;
  const dim3 fold((p.nA + bx - 1) / bx, std::min((p.nZ + by - 1) / by, 65535));
  launch_after(gram_fold_kernel<TYPE>, fold, dim3(bx, by), 0, s, p, cnt);
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
}

}  // namespace

void launch_gram_tc_split(const GramParams &p, uint16_t *cnt, cudaStream_t s) {
  if (p.type == 1)
    launch_split_type<1>(p, cnt, s);
  else
    launch_split_type<2>(p, cnt, s);
}

// As many blocks as leave two rounds of the 304 CTAs that run at once (one or
// four rounds: within 10 % either way).  A CTA per block writes, and the sum
// reads, the counts of every block: for 16384 rows x 99 planes x 69 blocks, 224
// MB of them, 503 us and 200 us, a call of 780 us where one CTA per tile walking
// all blocks had taken 667; with spans it takes 440.
int and_counts_span(long long nA, long long nZ, int P) {
  const long long tiles = ((nA + kM - 1) / kM) * ((nZ + kN - 1) / kN);
  return (int)std::max(1ll, std::min<long long>(kSpanMax, tiles * P / 608));
}

void launch_and_counts_tc(const GramParams &p, int span, uint16_t *cnt, uint16_t *zcnt, cudaStream_t s) {
  launch_counts<2>(p, span, cnt, zcnt, s);
}

namespace {
template <int NC>
void launch_attyn(const AtTYnParams &p, int nT, cudaStream_t s) {
  static const bool configured = [] {
    allow_smem(attyn_tc_kernel<NC>);
    return true;
  }();
  (void)configured;
  const dim3 grid((p.nY + 2 * NC - 1) / (2 * NC), (p.nA + kM - 1) / kM, nT);
  attyn_tc_kernel<NC><<<grid, kThreads, kSmemBytes, s>>>(p, tc_status_device_ptr());
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
}
}  // namespace

void launch_attyn_tc(const AtTYnParams &p, int nT, cudaStream_t s) {
  // Narrow tiles while all of them still fit the 304 places at once; above,
  // expanding the A rows four times would cost more than it gains.
  const long long tiles = (long long)((p.nY + kN - 1) / kN) * ((p.nA + kM - 1) / kM) * nT;
  if (4 * tiles <= 304)
    launch_attyn<8>(p, nT, s);
  else
    launch_attyn<32>(p, nT, s);
}

}  // namespace lakgb
