// +/-1 Gram of packed bit rows on the tensor cores (tcgen05, e2m1 operands).
//
// Computes exactly what the popcount kernel (gram.cu) computes, bit for bit:
//   out[i,k] = a0d1 - 2*S_ik - ((lfA_i + lfZ_k) - a2d1),  S_ik = sum_b D_b * c_ikb
// with c_ikb = popcount((A_i xor Z_k) & mask) over 1920-bit block b (TYPE_pm),
// or out = S_ik with c_ikb = popcount(A_i & Z_k & mask) (TYPE_00) -- the
// arithmetic of get_AnZt_vv__run (dir_c/AnZt_vv.c:62-95) with the block-
// weighted popcounts of popcount_xor_lf / popcount_and_lf
// (dir_c/popcount.c:310-423).
//
// Integer part on the tensor cores.  Every packed bit becomes one e2m1 value
// (4 bits, kind::mxf4 with unit scale factors), the mask applied to the A
// side, so that a product of two set bits is 1 and the fp32 accumulator of a
// block holds n_ikb = popcount(A_i & mask & Z_k) <= 1920 exactly.  The XOR
// count is c = pa_ib + pz_kb - 2 n_ikb with the row counts
// pa = popcount(A_i & mask), pz = popcount(Z_k & mask) that the producer
// threads take while they expand the bits.  Which bit goes to which K position
// does not matter (a dot product is order-free) as long as A and Z use the
// same map (tc::expand_e2m1).  Against one e4m3 byte per bit this halves the
// shared-memory bytes written by the producers and read by the MMAs, which
// together were over half of the kernel's shared-memory traffic, and takes a
// third of the expansion's integer operations.
//
// FP64 part on the CUDA cores, in the reference's order: acc = RN(acc + x),
// x = RN(D_b * c), blocks ascending.  An FP64 instruction of a warp holds its
// sub-partition's FP64 pipe for 80 cycles, so one FP64 add per element and
// block bounds the kernel (8960 cycles per tile and block; whole kernel 75.9 ms
// on 16384 x 16384 rows x 131072 columns of three bins, 60.3 ms with half of
// the adds left out), and integer adds alone are more instructions than the SM
// issues in that time (88 ms).  So rounds of four columns add with FP64 and with
// integers in turn: 62.7 ms (two or four of seven in integers: 63.8 and 64.7;
// two columns of every round: 64.8, a warp that waits for one pipe can not
// issue to the other).  Neither pipe is full then: of the issue slots 58 % (9
// blocks) to 70 % (69 blocks) are used, and the warps wait for TMEM, table and add latencies with no registers
// left for more of them.
// FP64: x comes from a table of the block's products.
// Integers: while acc lies in one binade its bit pattern counts units in the
// last place, and adding x is adding the integer RN(x / ulp), ties to even.
// For two exponents the table holds, for every count c and parity of acc,
//   RN(x / ulp) - c * floor(D / ulp)   (at most c + 1: 12 bits)
// and on which side of x / ulp that lies, so that an add is a 32 x 64-bit
// multiply-add and one more add.  A sum that leaves its binade is rounded once
// more, one bit up.  A round of which an element has another exponent or no
// entry (zero sums; negative, tiny or non-finite weights) is done again with
// FP64.
// The two exponents lie around the block's expected sums, estimated from a few
// row pairs when the table is made; the estimate decides only how often that
// happens.
//
// Persistent CTAs, one per SM, each looping over 128 (A rows) x 112 (Z rows)
// output tiles; the pipeline runs on across tile boundaries.  25 warps:
//   warps 0-7   producers, one tile row each (A rows 0-127, then Z rows
//               0-111): per step of 384 columns, read the row's 48 bytes from
//               the raw buffer, mask, expand to three 64-byte rows of e2m1 in
//               shared memory (K-major, 64-byte swizzle), count pa / pz.  A
//               producer warp works alone on its rows, so its time per step is
//               instruction latency: three chunks of 128 columns at once give
//               it independent instructions, and one wait, proxy fence and
//               arrival serve all three.  Each warp brings its 32 rows' next
//               steps into its own raw slots by cp.async, one block ahead, a
//               fixed (row, 16 bytes) per lane and copy: 16 bytes of its own
//               row per thread took 32 wavefronts per warp load, and one bulk
//               copy per row 68 cycles of the copy engine each (241 a block,
//               16400 cycles: slower than everything else).
//   warp 8      owns TMEM; lane 0 issues the MMAs (M=128, N=112, K=64; 6 per
//               step, 5 steps per block) into one of two count buffers.
//   warps 9-24  fold, four warps per lane quadrant (warp w reads TMEM lanes
//               32*(w%4)..+31), each for 28 of the 112 columns: per block,
//               read the counts from TMEM, look up the table, add into the
//               FP64 sums, which live in TMEM as well (columns 256..479,
//               two 32-bit halves per value).
// Shared memory: 6 raw slots (11 KB each) + 2 stages x 3 x (8 KB A + 7 KB B) +
// 2 block tables (30 KB) + counts.
// The table buffers are filled by bulk copies on mbarriers, issued by whichever
// fold warp finishes a block last, so fold warps drift apart by up to a block
// instead of meeting at every block boundary.
// TMEM: 2 x 112 count columns (0.., 128..), the scale factors (112..127) and
// 224 accumulator columns; N = 112 leaves room for the scale factors.
#include <algorithm>

#include "fixed_fp64.cuh"
#include "gram.cuh"
#include "lakgb_runtime.cuh"
#include "tc_ptx.cuh"

namespace lakgb {

// Test hook: when set, producer warp 0 of CTA 0 withholds its arrival for
// the first operand stage, so the MMA warp's wait for that stage runs out
// (lakgb_debug_tc_withhold).
static __device__ int g_withhold;

namespace {

constexpr int kBM = kGramTileM, kBN = kGramTileN;
constexpr int kStages = 2;
constexpr int kChunk = 3;                 // 128-column chunks per step
constexpr int kSteps = 5;                 // steps per 1920-column block
constexpr int kBlockRow = 240;            // bytes of one row of a block
constexpr int kRawRow = 16 * kChunk;      // bytes of one row of a step
constexpr int kRawSlots = kSteps + 1;
constexpr int kRawBytes = (kBM + kBN) * kRawRow;
constexpr int kTileA = kBM * 64;          // bytes: 128 rows x 128 e2m1
constexpr int kTileB = kBN * 64;
constexpr int kChunkBytes = kTileA + kTileB;
constexpr int kStageBytes = kChunk * kChunkBytes;
constexpr int kTabStride = 1922;          // doubles per block table (1921 used, 16-byte multiple)
constexpr int kTabExps = 2;               // exponents of the integer entries
constexpr int kTabInt = kTabStride * 8;   // their place in a block's table
constexpr int kTabExpBytes = kTabStride * 4;
constexpr int kTabHdr = kTabInt + kTabExps * kTabExpBytes;
struct TabHdr {
  unsigned long long unit[kTabExps];      // floor(D / ulp) of exponent etop, etop - 1
  uint32_t etop, pad[3];                  // biased exponent
};
constexpr int kTabBytes = kTabHdr + (int)sizeof(TabHdr);
constexpr uint32_t kTabInvalid = 0xFFFFu, kTabValue = 0xFFFu;
constexpr int kTabRestShift = 12;         // x / ulp - RN(x / ulp): 0 zero, 1 above, 2 below
static_assert(kTabInt % 16 == 0 && kTabHdr % 16 == 0 && kTabBytes % 16 == 0, "bulk copies");
constexpr int kSBO = 8 * 64;              // bytes between 8-row swizzle atoms (8 rows of 64 B)
constexpr int kProducers = 256;           // warps 0-7
constexpr int kMmaWarp = 8;
constexpr int kFold = 512;                // warps 9-24
constexpr int kFoldWarps = kFold / 32;
constexpr int kRound = 4;                 // columns per TMEM round of a fold warp
constexpr int kFoldCols = kBN / (kFold / 128);  // tile columns per fold warp
constexpr int kRounds = kFoldCols / kRound;
constexpr int kThreads = kProducers + 32 + kFold;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kCntCols = 128;        // columns from one count buffer to the next
constexpr uint32_t kSfCol = 112;          // scale factors: 16 columns of ones
constexpr uint32_t kAccCol = 256;
static_assert(kFoldCols % kRound == 0 && kBN <= (int)kSfCol && kAccCol + 2 * kBN <= kTmemCols, "TMEM layout");
static_assert(kChunkBytes % 512 == 0 && kSteps * kRawRow == kBlockRow, "swizzle atoms, whole blocks");
constexpr size_t kSmemBytes =
    (size_t)kStages * kStageBytes + kRawSlots * kRawBytes + 2 * kTabBytes + 2 * 256 * 4 + 1024;
static_assert(kSmemBytes + 512 <= 227 * 1024, "one CTA per SM");

struct Smem {
  uint64_t full[kStages], empty[kStages];
  uint64_t acc_full[2], acc_empty[2], aux_full[2], aux_empty[2], done;
  uint64_t tab_full[2];            // T_b buffer t loaded (bulk copy)
  unsigned tab_read[2];            // fold warps done with buffer t (monotonic)
  unsigned tab_issued[2];          // bulk copies issued into buffer t
  uint32_t tmem_base;
  int abort;
};

template <int R>
__device__ __forceinline__ void tmem_ld_n(uint32_t taddr, uint32_t (&v)[R]) {
  if constexpr (R == 4) tc::tmem_ld4(taddr, v);
  else if constexpr (R == 8) tc::tmem_ld8(taddr, v);
  else if constexpr (R == 16) tc::tmem_ld16(taddr, v);
  else tc::tmem_ld32(taddr, v);
}
template <int R>
__device__ __forceinline__ void tmem_st_n(uint32_t taddr, const uint32_t (&v)[R]) {
  if constexpr (R == 8) tc::tmem_st8(taddr, v);
  else if constexpr (R == 16) tc::tmem_st16(taddr, v);
  else tc::tmem_st32(taddr, v);
}

__device__ __forceinline__ int popc4(uint4 x) { return __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w); }
__device__ __forceinline__ uint4 and4(uint4 a, uint4 b) {
  return make_uint4(a.x & b.x, a.y & b.y, a.z & b.z, a.w & b.w);
}

// Counts decoded from the accumulator (exact for n < 2^22).
__device__ __forceinline__ int decode_count(uint32_t bits) {
  return __float_as_int(__fadd_rn(__uint_as_float(bits), 12582912.0f)) - 0x4B400000;
}

// (tile_m, tile_n) of tile r of one Gram's list.  A full grid is walked in
// bands of kBand tile rows, each band column by column: the CTAs of a wave
// (consecutive r) then share a few A row panels and a few Z row panels, a
// working set that stays in L2 even when a whole side of the product does
// not (32768-row bins: 2 MB per 128-row panel).  A symmetric Gram lists only
// the tiles that hold a pair i <= k, row by row: those of tile row i from
// tile column i * 128 / 112 on.
constexpr int kBand = 8;
__device__ __forceinline__ void tile_coords(int ntm, int ntn, bool sym, int r, int &tile_m, int &tile_n) {
  if (!sym) {
    const int band = r / (kBand * ntn), in = r - band * (kBand * ntn);
    const int rows = min(kBand, ntm - band * kBand);
    tile_m = (band * kBand + in % rows) * kBM;
    tile_n = (in / rows) * kBN;
    return;
  }
  int i = 0, first = 0;
  while (r >= ntn - first) {
    r -= ntn - first;
    ++i;
    first = i * kBM / kBN;
  }
  tile_m = i * kBM;
  tile_n = (first + r) * kBN;
}

// The instance of a grouped launch that holds global tile (or table row) k:
// the last i with start[i] <= k.
template <typename I>
__device__ __forceinline__ int find_instance(const I *start, int n, long long k) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((long long)start[mid] <= k) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Tile order shared by every role: tile k of the launch's list goes to CTA
// k % gridDim.x, so the active tiles, not all tiles, are spread evenly over
// the CTAs.  A single Gram lists its own tiles (tile_coords); a grouped launch
// lists the tiles of its instances one instance after another.
template <bool GRP>
struct TileWalk {
  int ntiles, k;
  __device__ TileWalk(int tiles, const GramGroupDev &g)
      : ntiles(GRP ? g.tile0[g.n] : tiles), k((int)blockIdx.x - (int)gridDim.x) {}
  __device__ bool next(const GramParams &p, const GramGroupDev &g, int &inst, int &tile_m, int &tile_n) {
    k += gridDim.x;
    if (k >= ntiles) return false;
    inst = GRP ? find_instance(g.tile0, g.n, k) : 0;
    const GramParams &q = GRP ? g.ps[inst] : p;
    tile_coords((q.nA + kBM - 1) / kBM, (q.nZ + kBN - 1) / kBN, q.symmetric, GRP ? k - g.tile0[inst] : k, tile_m, tile_n);
    return true;
  }
};

// The parameters of instance `inst` (a grouped launch) or the launch's own.
template <bool GRP>
__device__ __forceinline__ const GramParams &params_of(const GramParams &p, const GramGroupDev &g, int inst) {
  if constexpr (GRP) return g.ps[inst];
  else return p;
}

// Rounds of kRound columns of a fold warp that hold results: not those past
// the last Z row or, in a symmetric Gram, left of the warp's first row.  A warp
// past the last A row has none.  [first, end)
__device__ __forceinline__ void live_rounds(const GramParams &pp, int row0, int colbase, int &first, int &end) {
  first = 0;
  end = row0 < pp.nA ? min(kRounds, (max(pp.nZ - colbase, 0) + kRound - 1) / kRound) : 0;
  if (pp.symmetric && row0 > colbase) first = min((row0 - colbase) / kRound, end);
}

// The results of a fold warp's 32 rows x kFoldCols columns from its sums S in
// TMEM (acc): a0d1 - 2 S - ((lfA + lfZ) - a2d1).  As four FP64 operations and a
// predicated multiply for 2 S that took 52000 cycles a tile (a block's fold:
// 10400), now about 25000 (2018 x 2025 rows x 820 columns: 65.3 -> 49 us).  So S doubles in its bits; where all of the warp's terms have a
// fixed-point form (fixed_fp64.cuh), every other round is computed in integers,
// the even ones by half of a sub-partition's warps and the odd ones by the other.
template <int TYPE>
__device__ __forceinline__ void write_results(const GramParams &pp, int tile_m, int tile_n, int col0, int row, int lane,
                                              int first, int end, int phase, uint32_t acc) {
  const int ga = tile_m + row, gl = tile_n + col0 + lane;
  const bool row_in = ga < pp.nA, lf = pp.lfA && pp.lfZ;
  const double lfa = (lf && row_in) ? pp.lfA[ga] : 0.0, a0 = TYPE == 1 ? pp.a0d1 : 0.0, a2 = pp.a2d1;
  // Everything else that a result needs is read here, before the first store
  // (which may change any of it, for all the compiler knows); lane l holds what
  // belongs to the warp's column l.
  const bool sym = pp.symmetric, col_in = lane < kFoldCols && gl < pp.nZ;
  const long long stride = pp.out_stride;
  const int nZ = pp.nZ;
  const double *plfz = pp.lfZ;
  const double lfz = (lf && col_in) ? plfz[gl] : 0.0;
  const uint32_t oc = col_in ? pp.out_c[gl] : 0u, or2 = (sym && col_in) ? pp.out_r2[gl] : 0u;
  double *out = pp.out + (row_in ? (long long)pp.out_r[ga] : 0);
  double *out2 = pp.out + ((sym && row_in) ? (long long)pp.out_c2[ga] * stride : 0);
  long long fa = 0, fz = 0, f0 = 0, f2 = 0;
  int emax = 0;
  bool fixed = false;
  if (lf) {
    const uint32_t e = max(max((uint32_t)__double2hiint(lfa) << 1, (uint32_t)__double2hiint(lfz) << 1),
                           max((uint32_t)__double2hiint(a0) << 1, (uint32_t)__double2hiint(a2) << 1));
    emax = (int)(__reduce_max_sync(0xffffffffu, e) >> 21);
    const bool good = fixed::from_bits((unsigned long long)__double_as_longlong(lfa), emax, &fa) &
                      fixed::from_bits((unsigned long long)__double_as_longlong(lfz), emax, &fz) &
                      fixed::from_bits((unsigned long long)__double_as_longlong(a0), emax, &f0) &
                      fixed::from_bits((unsigned long long)__double_as_longlong(a2), emax, &f2);
    fixed = __all_sync(0xffffffffu, good && fixed::in_range(emax));
  }
#pragma unroll 1
  for (int r = first; r < end; ++r) {
    uint32_t a[2 * kRound];
    __syncwarp();
    tmem_ld_n<2 * kRound>(acc + 2 * r * kRound, a);
    double o[kRound];
    tc::tmem_wait_ld();
    tc::reg_fence(a);
    // in integers where every S has a fixed-point form too (not a zero, a
    // smaller or larger S)
    bool good = fixed && ((r ^ phase) & 1);
#pragma unroll
    for (int j = 0; j < kRound; ++j)
      good = good && (a[2 * j + 1] >> 20) - (uint32_t)(emax - fixed::kBelow) <= (uint32_t)fixed::kBelow;
    if (__all_sync(0xffffffffu, good || (!row_in && fixed && ((r ^ phase) & 1)))) {
#pragma unroll
      for (int j = 0; j < kRound; ++j) {
        const uint32_t sh = ((a[2 * j + 1] >> 20) - (uint32_t)(emax - fixed::kBelow)) & 15u;
        const long long v = (long long)(((unsigned long long)((a[2 * j + 1] & 0xFFFFFu) | 0x100000u) << 32 | a[2 * j]) << sh);
        const long long t = fixed::round53(fixed::round53(fa + __shfl_sync(0xffffffffu, fz, r * kRound + j)) - f2);
        const long long u = TYPE == 1 ? fixed::round53(f0 - 2 * v) : v;
        o[j] = __longlong_as_double((long long)fixed::to_bits(u - t, emax));
      }
    } else {
#pragma unroll
      for (int j = 0; j < kRound; ++j) {
        const unsigned long long s = (unsigned long long)a[2 * j + 1] << 32 | a[2 * j];
        o[j] = TYPE == 1 ? __dsub_rn(a0, __longlong_as_double((long long)fixed::twice_bits(s))) : __longlong_as_double((long long)s);
        // read here, so that the compiler can not hoist the FP64 operations
        // above the branch
        if (lf)
          o[j] = __dsub_rn(o[j], __dsub_rn(__dadd_rn(lfa, __ldcv(plfz + min(tile_n + col0 + r * kRound + j, nZ - 1))), a2));
      }
    }
#pragma unroll
    for (int j = 0; j < kRound; ++j) {
      const int gz = tile_n + col0 + r * kRound + j;
      const uint32_t c = __shfl_sync(0xffffffffu, oc, r * kRound + j), r2 = __shfl_sync(0xffffffffu, or2, r * kRound + j);
      if (!row_in || gz >= nZ || (sym && ga > gz)) continue;
      out[(long long)c * stride] = o[j];
      if (sym) out2[r2] = o[j];
    }
  }
}

// acc = RN(acc + RN(D c)) for the warp's 32 x kRound sums (a: low and high
// words; old: the same in TMEM), in integers as described at the top.
// Lanes without a row hold no sums.
__device__ __forceinline__ void add_round(const uint8_t *tab, uint32_t etop, const int (&c)[kRound],
                                          uint32_t (&a)[2 * kRound], uint32_t old, bool row_in) {
  uint32_t far = 0u, left = 0u, last = 0u, below = 0u, ent[kRound];
#pragma unroll
  for (int j = 0; j < kRound; ++j) {
    const uint32_t lo = a[2 * j], hi = a[2 * j + 1], x = etop - (hi >> 20), xi = x & 1u;
    ent[j] = *reinterpret_cast<const uint16_t *>(tab + kTabInt + xi * kTabExpBytes + 4 * c[j] + 2 * (lo & 1u));
    const unsigned long long unit = reinterpret_cast<const TabHdr *>(tab + kTabHdr)->unit[xi];
    const unsigned long long v =
        (((unsigned long long)hi << 32) | lo) + (unsigned)c[j] * unit + (ent[j] & kTabValue);
    a[2 * j] = (uint32_t)v;
    a[2 * j + 1] = (uint32_t)(v >> 32);
    far |= x;
    below |= xi << j;
    left |= a[2 * j + 1] ^ hi;
    last = max(last, ent[j]);
  }
  const bool bad = row_in && (far > 1u || last == kTabInvalid);
  if (__any_sync(0xffffffffu, bad || (row_in && (left >> 20)))) {
    if (__any_sync(0xffffffffu, bad)) {
      tmem_ld_n<2 * kRound>(old, a);
      tc::tmem_wait_ld();
      tc::reg_fence(a);
#pragma unroll
      for (int j = 0; j < kRound; ++j) {
        const double v = __dadd_rn(__hiloint2double((int)a[2 * j + 1], (int)a[2 * j]),
                                   reinterpret_cast<const double *>(tab)[c[j]]);
        a[2 * j] = (uint32_t)__double2loint(v);
        a[2 * j + 1] = (uint32_t)__double2hiint(v);
      }
    } else {
      // Sums that left their binade e: v counts (e << 52) + m - 2^52 with m in
      // [2^53, 2^54) and becomes (e << 52) + RN(m / 2), m odd rounded by what
      // the first rounding left.
#pragma unroll
      for (int j = 0; j < kRound; ++j) {
        const uint32_t e = etop - ((below >> j) & 1u);
        if ((a[2 * j + 1] >> 20) == e) continue;
        const uint32_t lo = a[2 * j], hi = a[2 * j + 1] - (e << 20) + 0x00100000u;
        const uint32_t rest = ent[j] >> kTabRestShift, half = __funnelshift_r(lo, hi, 1);
        const uint32_t up = lo & 1u & (rest == 0u ? half : rest);
        const unsigned long long h = (((unsigned long long)((hi >> 1) + (e << 20))) << 32 | half) + up;
        a[2 * j] = (uint32_t)h;
        a[2 * j + 1] = (uint32_t)(h >> 32);
      }
    }
  }
}

template <int TYPE, bool GRP>
__global__ void __launch_bounds__(kThreads, 1)
    gram_tc_kernel(GramParams p, GramGroupDev grp, int tiles, const uint8_t *__restrict__ T, int *status) {
  extern __shared__ __align__(128) uint8_t dsm[];
  __shared__ Smem sm;
  // stages first, on a 1024-byte boundary (swizzle atoms)
  uint8_t *stages = dsm + ((1024 - (tc::smem_u32(dsm) & 1023)) & 1023);
  uint8_t *raw = stages + (size_t)kStages * kStageBytes;                       // [kRawSlots][kRawBytes]
  uint8_t *sT = raw + kRawSlots * (size_t)kRawBytes;                           // [2][kTabBytes]
  int *s_cnt = reinterpret_cast<int *>(sT + 2 * kTabBytes);                    // [2][256]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int *abort = &sm.abort;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(&sm.full[s], kProducers / 32);  // one arrival per warp
      tc::mbar_init(&sm.empty[s], 1);
    }
    for (int t = 0; t < 2; ++t) {
      tc::mbar_init(&sm.acc_full[t], 1);
      tc::mbar_init(&sm.acc_empty[t], kFoldWarps);
      tc::mbar_init(&sm.aux_full[t], kProducers / 32);
      tc::mbar_init(&sm.aux_empty[t], kFoldWarps);
      tc::mbar_init(&sm.tab_full[t], 1);
      sm.tab_read[t] = sm.tab_issued[t] = 0;
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
  // unit scale factors in every lane: one warp per lane quadrant
  if (warp > kMmaWarp && warp <= kMmaWarp + 4) {
    uint32_t ones[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) ones[i] = tc::kScaleOnes;
    tc::tmem_st16(tmem + kSfCol + ((uint32_t)(32 * (warp & 3)) << 16), ones);
    tc::tmem_wait_st();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  TileWalk<GRP> walk(tiles, grp);
  int inst, tile_m, tile_n;

  if (tid < kProducers) {
    // ---------------- producers ----------------
    const int side = tid >> 7, rr = tid & 127;  // side 0: A row rr, side 1: Z row rr
    const bool has_row = side == 0 || rr < kBN;
    const uint32_t my_row = tc::smem_u32(stages) + side * kTileA + (uint32_t)(rr * 64);
    const uint32_t my_sw = (uint32_t)((rr >> 1) & 3);
    const int row0 = side * kBM + (rr & ~31);  // this warp's first tile row
    const uint32_t my_raw = tc::smem_u32(raw) + (uint32_t)((row0 + (has_row ? lane : 0)) * kRawRow);
    // the test hook, read once: this thread withholds its first arrival
    bool withhold = g_withhold && blockIdx.x == 0 && tid == 0;
    bool ok = true;
    // A tile's mask, blocks and the global addresses of this lane's kChunk
    // copies of a step (copy j of a lane: piece i % 3 of the warp's row i / 3,
    // i = lane + 32 j; null: a row past the matrix).
    struct Src {
      const uint8_t *mask, *piece[kChunk];
      int P;
    };
    auto next_tile = [&](Src &v) {
      if (!walk.next(p, grp, inst, tile_m, tile_n)) return false;
      const GramParams &q = params_of<GRP>(p, grp, inst);
      v.mask = q.mask;
      v.P = q.P;
      const int first = (side ? tile_n : tile_m) + (rr & ~31);
      const int last = side ? min(q.nZ, tile_n + kBN) : q.nA;
#pragma unroll
      for (int j = 0; j < kChunk; ++j) {
        const int i = lane + 32 * j, r = first + i / kChunk;
        v.piece[j] = nullptr;
        if (r < last)
          v.piece[j] = (side ? q.wZ : q.wA) + (long long)(side ? q.z_rowb : q.a_rowb)[r] * (side ? q.z_row_bytes : q.a_row_bytes) +
                       16 * (i % kChunk);
      }
      return true;
    };
    uint8_t *my_dst = raw + row0 * kRawRow + 16 * lane;  // copy j: + 512 j
    auto fetch = [&](const Src &v, int step, int slot) {  // step: from the tile's first column
#pragma unroll
      for (int j = 0; j < kChunk; ++j)
        if (v.piece[j])
          tc::cp_async16(my_dst + (size_t)slot * kRawBytes + 512 * j, v.piece[j] + (long long)step * kRawRow);
      tc::cp_async_commit();
    };
    Src cur{}, nxt{};
    bool have = next_tile(cur);
    for (int j = 0; j < kSteps; ++j) {
      if (have) fetch(cur, j, j);
      else tc::cp_async_commit();
    }
    int s = 0, wrap = 0;   // ring position of the next step: stage s, in pass `wrap` over the ring
    int slot = 0;          // raw slot of the next step
    int gbb = 0, b = 0;    // blocks this CTA has produced; block of the tile
    while (have) {
      const int t = gbb & 1;
      bool more = true;
      int nb = b + 1;
      nxt = cur;
      if (nb == cur.P) {
        nb = 0;
        more = next_tile(nxt);
      }
      const uint4 *mk = reinterpret_cast<const uint4 *>(cur.mask) + (long long)b * (kSteps * kChunk);
      int cnt = 0;
#pragma unroll 1
      for (int j = 0; j < kSteps; ++j) {
        // the step kSteps ahead, into the slot read before this one
        if (more) fetch(nxt, nb * kSteps + j, slot ? slot - 1 : kRawSlots - 1);
        else tc::cp_async_commit();
        uint4 x[kChunk], m[kChunk];
#pragma unroll
        for (int u = 0; u < kChunk; ++u) m[u] = __ldg(mk + j * kChunk + u);
        tc::cp_async_wait<kSteps>();
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kChunk; ++u) x[u] = tc::ld_shared_v4(my_raw + slot * kRawBytes + 16 * u);
        if (wrap > 0 && ok) ok = tc::mbar_wait(&sm.empty[s], (uint32_t)((wrap - 1) & 1), abort, status, 1);
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
          // A rows enter masked; Z rows unmasked (the mask on A already
          // restricts every product), their count masked
          const uint4 xm = and4(x[u], m[u]);
          if (TYPE == 1) cnt += popc4(xm);
          if (!side) x[u] = xm;
        }
        if (ok && has_row) {
          const uint32_t dst = my_row + s * kStageBytes;
          if (side) {
#pragma unroll
            for (int u = 0; u < kChunk; ++u) tc::expand_e2m1<1>(dst + u * kChunkBytes, my_sw, x[u]);
          } else {
#pragma unroll
            for (int u = 0; u < kChunk; ++u) tc::expand_e2m1<0>(dst + u * kChunkBytes, my_sw, x[u]);
          }
          tc::fence_proxy_async();
        }
        __syncwarp();
        if (lane == 0 && !withhold) tc::mbar_arrive(&sm.full[s]);
        withhold = false;
        if (++s == kStages) {
          s = 0;
          ++wrap;
        }
        if (++slot == kRawSlots) slot = 0;
      }
      // publish the row counts
      if (gbb >= 2 && ok)
        ok = tc::mbar_wait(&sm.aux_empty[t], (uint32_t)(((gbb >> 1) - 1) & 1), abort, status, 2);
      s_cnt[t * 256 + tid] = cnt;
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&sm.aux_full[t]);
      ++gbb;
      b = nb;
      cur = nxt;
      have = more;
    }
    tc::cp_async_wait<0>();
  } else if (warp == kMmaWarp) {
    // ---------------- MMA issue ----------------
    if (lane == 0) {
      constexpr uint32_t idesc = tc::idesc_mxf4_f32(kBM, kBN);
      const uint32_t st0 = tc::smem_u32(stages);
      bool ok = true;
      int s = 0, wrap = 0, gbb = 0;
      while (ok && walk.next(p, grp, inst, tile_m, tile_n)) {
        const int P = params_of<GRP>(p, grp, inst).P;
        for (int b = 0; b < P && ok; ++b, ++gbb) {
          const int t = gbb & 1;
          if (gbb >= 2)
            ok = tc::mbar_wait(&sm.acc_empty[t], (uint32_t)(((gbb >> 1) - 1) & 1), abort, status, 3);
          tc::fence_after_sync();
          for (int st = 0; st < kSteps && ok; ++st) {
            const int cs = s;
            ok = tc::mbar_wait(&sm.full[cs], (uint32_t)(wrap & 1), abort, status, 4);
            if (++s == kStages) {
              s = 0;
              ++wrap;
            }
            if (!ok) break;
            tc::fence_after_sync();
#pragma unroll
            for (int u = 0; u < kChunk; ++u) {
              const uint32_t sa = st0 + cs * kStageBytes + u * kChunkBytes, sb = sa + kTileA;
#pragma unroll
              for (int kk = 0; kk < 2; ++kk)
                tc::mma_mxf4(tmem + t * kCntCols, tc::smem_desc_sw64(sa + kk * 32, kSBO),
                             tc::smem_desc_sw64(sb + kk * 32, kSBO), idesc, tmem + kSfCol, tmem + kSfCol + 4,
                             (st | u | kk) != 0);
            }
            tc::mma_commit(&sm.empty[cs]);
          }
          if (ok) tc::mma_commit(&sm.acc_full[t]);
        }
      }
      // every issued MMA has completed before TMEM is released (waited for
      // even after an abort, within the same time limit)
      tc::mma_commit(&sm.done);
      const unsigned long long t0 = tc::globaltimer();
      while (!tc::mbar_try(&sm.done, 0)) {
        if (tc::globaltimer() - t0 > tc::g_wait_ns) {
          atomicCAS(status, 0, 5);
          break;
        }
      }
    }
  } else {
    // ---------------- FP64 fold ----------------
    const int et = tid - (kProducers + 32);  // 0..kFold-1
    const int q = warp & 3;
    const int col0 = (et >> 7) * kFoldCols;   // this warp's columns of the tile
    const int phase = et >> 7;
    const int row = 32 * q + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16);
    // The table T_b of the CTA's g-th block goes into buffer g & 1 by one
    // bulk copy.  Copies g = 0, 1 start here; the last fold warp to finish
    // block g issues g + 2 into the buffer g read, so the fold warps are never
    // held together at block boundaries.  issue_table(t, jt, boff) loads the
    // block `boff` blocks after the start of this CTA's tile jt: block
    // boff % P of a single Gram (every tile has P blocks); in a grouped launch
    // it is found by walking on through this CTA's tiles, and nothing is
    // loaded past its last block.  (Copies issued past the CTA's last block
    // of a single Gram are waited for at the end.)
    const int ntiles_grp = GRP ? grp.tile0[grp.n] : 0;
    auto issue_table = [&](int t, int jt, int boff) {
      int in = 0, blk = 0;
      if constexpr (GRP) {
        for (;;) {
          const int k = (int)blockIdx.x + jt * (int)gridDim.x;
          if (k >= ntiles_grp) return;
          in = find_instance(grp.tile0, grp.n, k);
          const int pj = grp.ps[in].P;
          if (boff < pj) break;
          boff -= pj;
          ++jt;
        }
        blk = boff;
      } else {
        blk = boff % p.P;
      }
      const uint8_t *src = T + ((GRP ? grp.blk0[in] : 0ll) + blk) * (long long)kTabBytes;
      tc::fence_proxy_async();
      tc::mbar_arrive_expect_tx(&sm.tab_full[t], kTabBytes);
      tc::bulk_g2s(sT + t * kTabBytes, src, kTabBytes, &sm.tab_full[t]);
      atomicAdd(&sm.tab_issued[t], 1u);
    };
    await_previous();  // the tables; nothing before the first block's fold needs them
    if (et == 0) {
      issue_table(0, 0, 0);
      issue_table(1, 0, 1);
    }
    bool ok = true;
    long long gb0 = 0;
    int jt = 0;  // this CTA's tiles so far
    while (walk.next(p, grp, inst, tile_m, tile_n)) {
      const GramParams &pp = params_of<GRP>(p, grp, inst);
      const int P = pp.P;
      int first, end;
      live_rounds(pp, tile_m + 32 * q, tile_n + col0, first, end);
      const bool row_in = tile_m + row < pp.nA;
      for (int b = 0; b < P; ++b) {
        const long long gbb = gb0 + b;
        const int t = (int)(gbb & 1);
        bool w = ok && tc::mbar_wait(&sm.tab_full[t], (uint32_t)((gbb >> 1) & 1), abort, status, 8);
        w = w && tc::mbar_wait(&sm.aux_full[t], (uint32_t)((gbb >> 1) & 1), abort, status, 6);
        w = w && tc::mbar_wait(&sm.acc_full[t], (uint32_t)((gbb >> 1) & 1), abort, status, 7);
        ok = __all_sync(0xffffffffu, w);
        tc::fence_after_sync();
        const uint8_t *tab = sT + t * kTabBytes;
        const double *Tb = reinterpret_cast<const double *>(tab);
        const uint32_t etop = reinterpret_cast<const TabHdr *>(tab + kTabHdr)->etop;
        const int pa = s_cnt[t * 256 + row];
        const int *pzb = s_cnt + t * 256 + 128;
        // Rounds of kRound columns, software-pipelined: the TMEM loads of
        // round r + 1 (counts, and accumulators after block 0) are in flight
        // while round r is added, so their latency hides behind the adds.
        uint32_t cn[2][kRound], a[2][2 * kRound];
        auto load_round = [&](int r, int buf) {
          const int c0 = col0 + r * kRound;
          tmem_ld_n<kRound>(lane_base + t * kCntCols + c0, cn[buf]);
          if (b > 0) tmem_ld_n<2 * kRound>(lane_base + kAccCol + 2 * c0, a[buf]);
        };
        if (first == end) {  // no results: no sums
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&sm.acc_empty[t]);
        } else {
          if (ok) {
            load_round(0, 0);
            tc::tmem_wait_ld();
            tc::reg_fence(cn[0]);
            tc::reg_fence(a[0]);
          }
#pragma unroll
          for (int r = 0; r < kRounds; ++r) {
            const int cur = r & 1, nxt = cur ^ 1;
            const int c0 = col0 + r * kRound;
            if (!ok) {
#pragma unroll
              for (int j = 0; j < kRound; ++j) cn[cur][j] = 0;
            }
            if (ok && r + 1 < kRounds) load_round(r + 1, nxt);
            if (r == kRounds - 1) {
              // all this warp's count columns of buffer t have been read
              tc::fence_before_sync();
              __syncwarp();
              if (lane == 0) tc::mbar_arrive(&sm.acc_empty[t]);
            }
            // the four columns' Z row counts in one 16-byte load (c0 is a
            // multiple of kRound = 4)
            static_assert(kRound == 4, "one int4 of Z row counts per round");
            const int4 pz4 = *reinterpret_cast<const int4 *>(pzb + c0);
            const int pzr[4] = {pz4.x, pz4.y, pz4.z, pz4.w};
            int c[kRound];
#pragma unroll
            for (int j = 0; j < kRound; ++j) {
              const int n = decode_count(cn[cur][j]);
              // 0 <= c <= 1920 for counts of a completed block; anything else
              // (counts of an aborted pipeline) reads the NaN entry 1921
              c[j] = (int)min((unsigned)((TYPE == 1) ? pa + pzr[j] - 2 * n : n), (unsigned)(kTabStride - 1));
            }
            // (not staggered between warps: both forms of every round in the
            // code take 75 ms)
            if (b > 0 && (r & 1)) {
              if (ok) add_round(tab, etop, c, a[cur], lane_base + kAccCol + 2 * c0, row_in);
            } else {
#pragma unroll
              for (int j = 0; j < kRound; ++j) {
                const double x = Tb[c[j]];
                const double v =
                    (b > 0) ? __dadd_rn(__hiloint2double((int)a[cur][2 * j + 1], (int)a[cur][2 * j]), x) : x;
                a[cur][2 * j] = (uint32_t)__double2loint(v);
                a[cur][2 * j + 1] = (uint32_t)__double2hiint(v);
              }
            }
            // accumulators of columns c0 + j: TMEM columns kAccCol + 2 (c0 + j)
            // (low word) and + 1 (high word)
            if (ok) tmem_st_n<2 * kRound>(lane_base + kAccCol + 2 * c0, a[cur]);
            if (ok && r + 1 < kRounds) {
              tc::tmem_wait_ld();
              tc::reg_fence(cn[nxt]);
              tc::reg_fence(a[nxt]);
            }
          }
        }
        // this warp no longer reads T buffer t; the last of the fold warps
        // to get here loads block gbb + 2 into it (after the copy it read
        // has landed; no new copies once the CTA has aborted)
        __syncwarp();
        if (lane == 0) {
          __threadfence_block();
          const unsigned prev = atomicAdd(&sm.tab_read[t], 1u);
          if ((prev + 1) % kFoldWarps == 0) {
            __threadfence_block();
            if (!*abort) {
              if (tc::mbar_wait_landed(&sm.tab_full[t], (uint32_t)((gbb >> 1) & 1)))
                issue_table(t, jt, b + 2);
              else
                atomicCAS(status, 0, 9);
            }
          }
        }
        __syncwarp();
        if (ok) tc::tmem_wait_st();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&sm.aux_empty[t]);
      }
      if (ok) write_results<TYPE>(pp, tile_m, tile_n, col0, row, lane, first, end, phase, lane_base + kAccCol + 2 * col0);
      gb0 += P;
      ++jt;
    }
    // every bulk copy into the tables has landed before the CTA exits (each
    // copy was issued after the previous one into its buffer landed)
    tc::named_bar_sync(1, kFold);
    if (et == 0) {
      for (int t = 0; t < 2; ++t) {
        const unsigned n = *(volatile unsigned *)&sm.tab_issued[t];
        if (n && !tc::mbar_wait_landed(&sm.tab_full[t], (n - 1) & 1)) atomicCAS(status, 0, 10);
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

// The table of block b of Gram p, shared out over kTableParts CTAs of 256
// threads (each makes the same estimate).
constexpr int kTableParts = 4;
__device__ void write_block_table(const GramParams &p, int b, uint8_t *__restrict__ tab) {
  __shared__ double s_sum[8];
  __shared__ int s_diff[8], s_all[8];
  release_next();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const double D = p.D ? p.D[b] : 1.0;
  double *prod = reinterpret_cast<double *>(tab);
  if (b == 0) {  // the first block's products are the sums: no integer entries
    for (int c = tid + blockDim.x * blockIdx.y; c < kTabStride; c += blockDim.x * kTableParts)
      prod[c] = c < kTabStride - 1 ? __dmul_rn(D, (double)c) : __longlong_as_double(0x7ff8dead00000000ll);
    return;
  }
  // Expected sums before this block: the earlier blocks' weighted mask counts (of
  // one block in `step` where there are more than threads: all of them, in every
  // block's table, took 1.3 ms of 24 at 5000 blocks), times the share of differing
  // (TYPE_pm) or common (TYPE_00) bits of four row pairs in this block (first A
  // rows against last Z rows).
  double sum = 0.0;
  const int step = (b + (int)blockDim.x - 1) / (int)blockDim.x, i = tid * step;
  if (i < b) {
    const uint4 *m = reinterpret_cast<const uint4 *>(p.mask + (long long)i * kBlockRow);
    int n = 0;
    for (int v = 0; v < kBlockRow / 16; ++v) n += popc4(__ldg(m + v));
    sum = __dmul_rn(p.D ? p.D[i] : 1.0, (double)(n * min(step, b - i)));
  }
  int diff = 0, all = 0;
  if (tid < 4 * (kBlockRow / 4)) {
    const int pair = tid / (kBlockRow / 4), w = tid % (kBlockRow / 4);
    const long long off = (long long)b * kBlockRow + 4 * w;
    const uint32_t m = __ldg(reinterpret_cast<const uint32_t *>(p.mask + off));
    const uint32_t ai = p.a_rowb[min(pair, p.nA - 1)], zi = p.z_rowb[max(p.nZ - 1 - pair, 0)];
    const uint32_t x = __ldg(reinterpret_cast<const uint32_t *>(p.wA + (long long)ai * p.a_row_bytes + off));
    const uint32_t z = __ldg(reinterpret_cast<const uint32_t *>(p.wZ + (long long)zi * p.z_row_bytes + off));
    diff = __popc((p.type == 1 ? x ^ z : x & z) & m);
    all = __popc(m);
  }
  diff = __reduce_add_sync(0xffffffffu, diff);
  all = __reduce_add_sync(0xffffffffu, all);
  if (32 * warp < b)
    for (int o = 16; o > 0; o >>= 1) sum = __dadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
  if (lane == 0) {
    s_sum[warp] = sum;
    s_diff[warp] = diff;
    s_all[warp] = all;
  }
  __syncthreads();
  sum = s_sum[0];
  diff = all = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    if (w && 32 * w < b) sum = __dadd_rn(sum, s_sum[w]);
    diff += s_diff[w];
    all += s_all[w];
  }
  const double share = (diff > 0 && all > 0) ? (double)diff / (double)all : 0.25;
  // two exponents: the expected sum's, and the one above where its mantissa
  // is above about sqrt(2), else the one below
  const uint32_t est = (uint32_t)__double2hiint(__dmul_rn(sum, share));
  const int etop = (int)((est >> 20) & 0x7ff) + ((est & 0xFFFFF) > 0x6A000 ? 1 : 0);

  const unsigned long long db = (unsigned long long)__double_as_longlong(D);
  const int ed = (int)((db >> 52) & 0x7ff);
  const unsigned long long dm = (db & 0x000fffffffffffffull) | 0x0010000000000000ull;
  const bool ok_d = !(db >> 63) && ed >= 64 && ed <= 1900;
  for (int c = tid + blockDim.x * blockIdx.y; c < kTabStride; c += blockDim.x * kTableParts) {
    const double x = c < kTabStride - 1 ? __dmul_rn(D, (double)c) : __longlong_as_double(0x7ff8dead00000000ll);
    prod[c] = x;
    const unsigned long long xb = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)((xb >> 52) & 0x7ff);
    const unsigned long long xm = (xb & 0x000fffffffffffffull) | 0x0010000000000000ull;
    for (int j = 0; j < kTabExps; ++j) {
      const int e = etop - j, k = e - ed, sh = e - ex;
      uint32_t entry = kTabInvalid | kTabInvalid << 16;
      if (ok_d && k >= 0 && k <= 52 && e >= 64 && e <= 2000 && c < kTabStride - 1) {
        if (c == 0) {
          entry = 0u;
        } else if (sh >= 0) {
          // floor(x / ulp) and its fraction: 0, below, at, above one half
          unsigned long long f = 0ull;
          uint32_t code = 1u;
          if (sh <= 60) {
            f = xm >> sh;
            const unsigned long long rem = xm & ((1ull << sh) - 1ull), half = (1ull << sh) >> 1;
            code = rem == 0ull ? 0u : rem < half ? 1u : rem == half ? 2u : 3u;
          }
          const uint32_t d = (uint32_t)(f - (unsigned long long)c * (dm >> k));  // at most c
          entry = 0u;
          for (uint32_t odd = 0; odd < 2; ++odd) {
            const uint32_t up = (code + (((uint32_t)f ^ odd) & 1u) + 1u) >> 2;
            entry |= (d + up | (code == 0u ? 0u : up ? 2u : 1u) << kTabRestShift) << (16 * odd);
          }
        }
      }
      reinterpret_cast<uint32_t *>(tab + kTabInt + j * kTabExpBytes)[c] = entry;
    }
  }
  if (tid == 0 && blockIdx.y == 0) {
    TabHdr *h = reinterpret_cast<TabHdr *>(tab + kTabHdr);
    for (int j = 0; j < kTabExps; ++j) {
      const int k = etop - j - ed;
      h->unit[j] = k >= 0 && k <= 52 ? dm >> k : 0ull;
    }
    h->etop = (uint32_t)etop;
  }
}

__global__ void __launch_bounds__(256) gram_table_kernel(GramParams p, uint8_t *__restrict__ T) {
  write_block_table(p, blockIdx.x, T + (size_t)blockIdx.x * kTabBytes);
}

// Table rows of a grouped launch: row r is block r - blk0[i] of instance i.
__global__ void __launch_bounds__(256) gram_table_group_kernel(GramGroupDev g, uint8_t *__restrict__ T) {
  const long long r = blockIdx.x;
  const int in = find_instance(g.blk0, g.n, r);
  write_block_table(g.ps[in], (int)(r - g.blk0[in]), T + (size_t)r * kTabBytes);
}

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    LAKGB_CUDA(cudaGetDevice(&dev));
    LAKGB_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
  }
  return n;
}

// Tiles a launch computes (symmetric Grams: those that hold a pair i <= k).
int active_tiles(const GramParams &p) {
  const int ntm = (p.nA + kBM - 1) / kBM, ntn = (p.nZ + kBN - 1) / kBN;
  if (!p.symmetric) return ntm * ntn;
  int n = 0;
  for (int i = 0; i < ntm; ++i) n += std::max(0, ntn - i * kBM / kBN);
  return n;
}

template <int TYPE, bool GRP>
void configure_tc() {
  static bool configured = false;
  if (!configured) {
    LAKGB_CUDA(cudaFuncSetAttribute(gram_tc_kernel<TYPE, GRP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kSmemBytes));
    configured = true;
  }
}

template <int TYPE>
void launch_tc_type(const GramParams &p, const uint8_t *T, cudaStream_t s) {
  configure_tc<TYPE, false>();
  const int tiles = active_tiles(p), grid = std::max(1, std::min(tiles, sm_count()));
  launch_after(gram_tc_kernel<TYPE, false>, grid, kThreads, kSmemBytes, s, p, GramGroupDev{}, tiles, T, tc_status_device_ptr());
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
}

template <int TYPE>
void launch_tc_group_type(const GramGroupDev &g, int total_tiles, const uint8_t *T, cudaStream_t s) {
  configure_tc<TYPE, true>();
  const int grid = std::max(1, std::min(total_tiles, sm_count()));
  launch_after(gram_tc_kernel<TYPE, true>, grid, kThreads, kSmemBytes, s, GramParams{}, g, total_tiles, T,
               tc_status_device_ptr());
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
}

}  // namespace

void launch_gram_tc(const GramParams &p, cudaStream_t s) {
  uint8_t *T = static_cast<uint8_t *>(scratch_alloc((size_t)p.P * kTabBytes, s));
  gram_table_kernel<<<dim3(p.P, kTableParts), 256, 0, s>>>(p, T);
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
  if (p.type == 1)
    launch_tc_type<1>(p, T, s);
  else
    launch_tc_type<2>(p, T, s);
  LAKGB_CUDA(cudaFreeAsync(T, s));
}

int gram_tc_tiles(const GramParams &p) { return active_tiles(p); }

size_t gram_tc_table_row_bytes() { return (size_t)kTabBytes; }

void launch_gram_tc_group(const GramGroupDev &g, int type, int total_tiles, long long total_blocks, void *T,
                          cudaStream_t s) {
  uint8_t *tab = static_cast<uint8_t *>(T);
  if (total_tiles <= 0 || total_blocks <= 0) return;
  gram_table_group_kernel<<<dim3((unsigned)total_blocks, kTableParts), 256, 0, s>>>(g, tab);
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
  if (type == 1)
    launch_tc_group_type<1>(g, total_tiles, tab, s);
  else
    launch_tc_group_type<2>(g, total_tiles, tab, s);
}

// The status word of the calling host thread's launches: every thread (a
// solve, a server worker) has its own, so a pipeline timeout in one solve is
// reported to that solve alone.
int *tc_status_device_ptr() { return thread_word(kTcStatus); }

// Read and clear the calling thread's status word (after every launch made
// so far has finished: the launches may be on a caller's stream).
int tc_status_take() {
  int *status = thread_word(kTcStatus, false);
  if (!status) return 0;
  int v = 0;
  LAKGB_CUDA(cudaDeviceSynchronize());
  LAKGB_CUDA(cudaMemcpy(&v, status, sizeof v, cudaMemcpyDeviceToHost));
  if (v) {
    LAKGB_CUDA(cudaMemsetAsync(status, 0, sizeof(int), stream()));
    LAKGB_CUDA(cudaStreamSynchronize(stream()));
  }
  return v;
}

// As tc_status_take, for launches on the calling thread's own stream only
// (a whole solve): waits for that stream, not for the device.
int tc_status_take_stream() {
  int *status = thread_word(kTcStatus, false);
  if (!status) return 0;
  int v = 0;
  LAKGB_CUDA(cudaMemcpyAsync(&v, status, sizeof v, cudaMemcpyDeviceToHost, stream()));
  LAKGB_CUDA(cudaStreamSynchronize(stream()));
  if (v) {
    LAKGB_CUDA(cudaMemsetAsync(status, 0, sizeof(int), stream()));
    LAKGB_CUDA(cudaStreamSynchronize(stream()));
  }
  return v;
}

void tc_debug_set(unsigned long long wait_ns, int withhold) {
  LAKGB_CUDA(cudaDeviceSynchronize());
  LAKGB_CUDA(cudaMemcpyToSymbol(tc::g_wait_ns, &wait_ns, sizeof wait_ns));
  LAKGB_CUDA(cudaMemcpyToSymbol(g_withhold, &withhold, sizeof withhold));
  LAKGB_CUDA(cudaDeviceSynchronize());
}

}  // namespace lakgb

// ---------------------------------------------------------------------------
// Throughput of the FP64 add on this device: the pipe that bounds the fold of
// the tensor-core Gram (one add per element per block).  Independent add
// chains on every SM, timed with CUDA events.

namespace lakgb {
namespace {

__global__ void fp64_add_rate_kernel(double *out, double y, int iters) {
  double a[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = threadIdx.x * 1e-3 + j;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = __dadd_rn(a[j], y);
  }
  double s = 0.0;
#pragma unroll
  for (int j = 0; j < 8; ++j) s = __dadd_rn(s, a[j]);
  out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

}  // namespace
}  // namespace lakgb

extern "C" double lakgb_measure_fp64_add_rate(void) {
  using namespace lakgb;
  const int blocks = sm_count() * 4, threads = 256, iters = 4096;
  double *d = nullptr;
  cudaEvent_t e0, e1;
  LAKGB_CUDA(cudaMalloc(&d, sizeof(double) * blocks * threads));
  LAKGB_CUDA(cudaEventCreate(&e0));
  LAKGB_CUDA(cudaEventCreate(&e1));
  float best = 0.f;
  for (int rep = 0; rep < 4; ++rep) {
    LAKGB_CUDA(cudaEventRecord(e0, stream()));
    fp64_add_rate_kernel<<<blocks, threads, 0, stream()>>>(d, 1.5e-9, iters);
    LAKGB_CUDA(cudaGetLastError());
    count_launch();
    LAKGB_CUDA(cudaEventRecord(e1, stream()));
    LAKGB_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    LAKGB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (rep > 0 && (best == 0.f || ms < best)) best = ms;
  }
  LAKGB_CUDA(cudaEventDestroy(e0));
  LAKGB_CUDA(cudaEventDestroy(e1));
  LAKGB_CUDA(cudaFree(d));
  return (double)blocks * threads * iters * 8 / (best * 1e-3);
}
