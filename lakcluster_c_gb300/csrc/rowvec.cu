// Row-vector products over packed bit rows (HBM-bound scans).
//
//  An_v    (dir_c/An_v.c:5-57):       out_r = -cpop_j + 2*popcount(row & mc_j)   (TYPE_pm)
//                                      out_r =          popcount(row & mc_j)    (TYPE_00)
//  An_ajdk (dir_c/An_ajdk_v.c:272-363): for each of the 15 weight vectors w_k,
//          out_rk = -sum_b w_kb*popcount(mc_j block b) + 2*sum_b w_kb*c_rb  (TYPE_pm)
//          with the block sums accumulated in ascending block order, one multiply
//          and one add per block and no FMA, as popcount_lf (popcount.c:252-308).
//
// An_v: one warp per row; lanes 0..29 read the 240-byte block as 8-byte
// words and the warp reduces the block count with shuffles.  An_ajdk: two rows
// per warp, one 16-byte piece of a row per lane.
#include "lakgb_runtime.cuh"
#include "rowvec.cuh"
#include "weigh.cuh"

namespace lakgb {

namespace {

__device__ __forceinline__ int block_count(const uint8_t *row, const uint8_t *mask, int lane) {
  int c = 0;
  if (lane < 30) {
    const uint2 x = __ldg(reinterpret_cast<const uint2 *>(row) + lane);
    const uint2 m = __ldg(reinterpret_cast<const uint2 *>(mask) + lane);
    c = __popc(x.x & m.x) + __popc(x.y & m.y);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  return c;
}

__global__ void an_v_kernel(RowvecParams p) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= p.n) return;
  const uint8_t *row = p.w + (long long)p.rowb[warp] * p.row_bytes;
  long long tot = 0;
  for (int b = 0; b < p.P; ++b)
    tot += block_count(row + (long long)b * kBlockBytes, p.mask + (long long)b * kBlockBytes, lane);
  if (lane == 0) {
    double o = (p.type == 1) ? __dadd_rn(-(double)p.cpop_j, __dmul_rn(2.0, (double)tot)) : (double)tot;
    p.out[p.out_r[warp]] = o;
  }
}

// Two rows per warp: lanes 0..14 read the pieces of row 2w's block, lanes
// 15..29 those of row 2w + 1, kAhead blocks ahead; one warp reduction gives both
// counts (16 bits each), and lanes 0..14 and 16..30 carry the two rows' 15 FP64
// sums.  The products with the counts are formed in integers, so a block costs
// one FP64 instruction (80 cycles of its sub-partition's FP64 pipe) per two
// rows: the floor beside the memory's.  8192 rows x 65536 columns: 64 us with
// two FP64 instructions per row and no loads ahead.
constexpr int kAhead = 4;
__global__ void __launch_bounds__(256) an_ajdk_kernel(RowvecParams p) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int r0 = 2 * warp;
  if (r0 >= p.n) return;
  const bool two = r0 + 1 < p.n;
  const int piece = lane < 15 ? lane : lane - 15;
  const bool reads = lane < 30;
  const uint4 *row = reinterpret_cast<const uint4 *>(p.w + (long long)p.rowb[lane >= 15 && two ? r0 + 1 : r0] * p.row_bytes) + piece;
  const uint4 *mask = reinterpret_cast<const uint4 *>(p.mask) + piece;
  const int k = lane & 15;
  const bool mine = k < 15 && (lane < 16 || two);
  const double *w = p.ajdk + (long long)(k < 15 ? k : 0) * p.P;
  uint4 x[kAhead], m[kAhead];
  double d[kAhead];
  auto load = [&](int b, int u) {
    x[u] = m[u] = make_uint4(0u, 0u, 0u, 0u);
    d[u] = 0.0;
    if (b < p.P) {
      if (reads) {
        x[u] = __ldg(row + 15 * b);
        m[u] = __ldg(mask + 15 * b);
      }
      d[u] = __ldg(w + b);
    }
  };
#pragma unroll
  for (int u = 0; u < kAhead; ++u) load(u, u);
  double s = 0.0;
  for (int b0 = 0; b0 < p.P; b0 += kAhead) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int b = b0 + u;
      if (b >= p.P) break;
      const uint32_t c = (uint32_t)(__popc(x[u].x & m[u].x) + __popc(x[u].y & m[u].y) + __popc(x[u].z & m[u].z) +
                                    __popc(x[u].w & m[u].w));
      const uint32_t both = __reduce_add_sync(0xffffffffu, lane < 15 ? c : c << 16);
      const double v = times_count(d[u], lane < 16 ? both & 0xffffu : both >> 16);
      load(b + kAhead, u);
      s = __dadd_rn(s, v);
    }
  }
  if (mine) {
    double o = (p.type == 1) ? __dadd_rn(-p.base[k], __dmul_rn(2.0, s)) : s;
    p.out[(long long)p.out_r[r0 + (lane >> 4)] + (long long)k * p.out_stride] = o;
  }
}

}  // namespace

void launch_an_v(const RowvecParams &p) {
  if (p.n <= 0) return;
  const int threads = 256;
  const int blocks = (int)(((long long)p.n * 32 + threads - 1) / threads);
  an_v_kernel<<<blocks, threads, 0, stream()>>>(p);
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
}

void launch_an_ajdk(const RowvecParams &p) {
  if (p.n <= 0) return;
  const int threads = 256;
  const long long warps = ((long long)p.n + 1) / 2;
  an_ajdk_kernel<<<(int)((warps * 32 + threads - 1) / threads), threads, 0, stream()>>>(p);
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
}

}  // namespace lakgb
