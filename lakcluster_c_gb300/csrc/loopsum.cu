// Loop-sum products over FP64 score matrices, and the SNP x SNP product AtTYn.
//
// AnZt_S_WnYt_vv (dir_c/AnZt_S_WnYt_vv.c:5-101, wrapper :103-145):
//   out[ma, s] = sum over Zn rows mz, in order, of (AnZt[ma,mz] * vS(s,mz)) * YnWt[ma,mz]
// AtTYn____WtSZn_vv (dir_c/AtTYn____WtSZn_vv.c:5-115, wrapper :117-159): over
// paired rows (na with nz) and paired inner rows (ny with nw), in order,
//   out[na, s] = sum (AtTYn[na,ny,s] * D_Yn[ny]) * ZtSWn[nz,nw,s]
// Both are sequential FP64 sums, added left to right by one lane per output.
//
// AtTYn_vv (dir_c/AtTYn_vv.c:5-202, wrapper :204-235):
//   out[na, ny, t] = ((hhAY - hhAy*aY) - aA*hhaY) + (aA*hhay)*aY
//   hhAY = cpop_j(At) - 2*popcount(~(At_na ^ Tt_t ^ Yt_ny) & mc_j(At))
//        = 2*popcount((At_na ^ Tt_t ^ Yt_ny) & mc_j) - cpop_j
//   hhAy = AtTn[na,t], hhaY = YtTn[ny,t] (integers read from FP64),
//   hhay = -cpop_j(Tt) + 2*popcount(Tt_t & mc_j(Tt)), aA / aY the column
//   means of the At / Yt rows' 1920-bit blocks.
// The counts run on the tensor cores (tc_counts.cu).
#include <optional>

#include "abi_common.cuh"
#include "lmirror.cuh"
#include "bcc_model.h"
#include "tc_counts.cuh"

namespace lakgb {

namespace {

inline unsigned long long pick_u(int s, unsigned long long j, unsigned long long b, unsigned long long a) {
  return s == LAKGB_SPACING_j ? j : (s == LAKGB_SPACING_b ? b : a);
}

// Number of values in the populated part of an L_handle (2-D or 3-D).
unsigned long long populated(const L_handle *L, bool three_d) {
  unsigned long long n = L->row_stride * L->col_stride * (three_d ? L->lyr_stride : 1);
  return n > L->length ? L->length : n;
}

unsigned long long max_index(const std::vector<unsigned long long> &v) {
  unsigned long long m = 0;
  for (unsigned long long x : v) m = x > m ? x : m;
  return m;
}

// Upload the populated part of an L_handle's values.
DBuf upload_L(const L_handle *L, bool three_d) {
  const unsigned long long n = populated(L, three_d);
  DBuf d((size_t)(n ? n : 1) * sizeof(double));
  if (n) d.upload(L->lf, (size_t)n * sizeof(double));
  return d;
}

// Both sums: one CTA per 32 rows (or pairs) and covariate.  Nine warps form the
// terms of kTerms columns into one half of a shared buffer -- the lane's row,
// so that reads of one column are contiguous in the column-major matrix --
// while one warp adds the other half's in order, a lane per row.  The chain of
// one FP64 add (80 cycles) per term bounds a row; a sum and its products in one
// thread took three operations per term, and 16 rows per CTA with the two
// phases one after the other twice the adding warps.  Two warps do nothing:
// they share the adding warp's FP64 pipe, which their products held for a fifth (two of
// eight forming warps there, one product a term) to a third of the time.  Which
// quarter of the warps that is goes round with the CTA, so that several CTAs on
// an SM add on different pipes.
constexpr int kSumRows = 32, kFormWarps = 9, kTermsPerWarp = 4, kTerms = kFormWarps * kTermsPerWarp, kSumT = 32 * 12;
struct SwnytCall {
  const double *A; const unsigned long long *a_r, *a_c;
  const double *Y; const unsigned long long *y_r, *y_c;
  const int8_t *vS; int nA, nZ, nS;
  const unsigned long long *out_r, *s_off;
  double *out;
  int tile0;  // grouped launch: first CTA of this call
};

struct WtszCall {
  const double *AY; const unsigned long long *ay_a, *ay_y, *ay_s;
  const double *ZW; const unsigned long long *zw_z, *zw_w, *zw_s;
  const double *Dy; int npairs, ninner, nS;
  const unsigned long long *out_r, *s_off;
  double *out;
  int tile0;  // grouped launch: first CTA of this call
};

// The terms of row i and covariate s: where term k's operands are, the operands
// and the product, in the reference's order of operations; the product with
// vS = +1 / -1 is exact.
struct SwnytTerm {
  const double *A, *Y;
  const unsigned long long *a_c, *y_c;
  const int8_t *vs;
  __device__ SwnytTerm(const SwnytCall &c, int i, int s)
      : A(c.A + c.a_r[i]), Y(c.Y + c.y_r[i]), a_c(c.a_c), y_c(c.y_c), vs(c.vS + (long long)s * c.nZ) {}
  // few rows and long chains: operands ahead pay (a call 203 -> 139 us)
  static constexpr bool kAhead = true;
  static constexpr int kCtas = 2;
  struct At { unsigned long long a, y; int8_t v; };
  struct Of { double a, y; };
  __device__ __forceinline__ At at(int z) const { return {a_c[z], y_c[z], vs[z]}; }
  __device__ __forceinline__ Of of(const At &p) const {
    const double a = A[p.a];
    return {p.v < 0 ? -a : a, Y[p.y]};
  }
  __device__ __forceinline__ double operator()(const Of &o) const { return __dmul_rn(o.a, o.y); }
};
struct WtszTerm {
  const double *AY, *ZW, *Dy;
  const unsigned long long *ay_y, *zw_w;
  __device__ WtszTerm(const WtszCall &c, int i, int s)
      : AY(c.AY + c.ay_a[i] + c.ay_s[s]), ZW(c.ZW + c.zw_z[i] + c.zw_s[s]), Dy(c.Dy), ay_y(c.ay_y), zw_w(c.zw_w) {}
  // many rows: more CTAs per SM hide the loads, the registers go to them
  static constexpr bool kAhead = false;
  static constexpr int kCtas = 3;
  struct At { unsigned long long a, z; double d; };
  struct Of { double a, d, z; };
  __device__ __forceinline__ At at(int k) const { return {ay_y[k], zw_w[k], Dy[k]}; }
  __device__ __forceinline__ Of of(const At &p) const { return {AY[p.a], p.d, ZW[p.z]}; }
  __device__ __forceinline__ double operator()(const Of &o) const { return __dmul_rn(__dmul_rn(o.a, o.d), o.z); }
};
__host__ __device__ inline int sum_rows(const SwnytCall &c) { return c.nA; }
__host__ __device__ inline int sum_rows(const WtszCall &c) { return c.npairs; }
__device__ inline int sum_terms(const SwnytCall &c) { return c.nZ; }
__device__ inline int sum_terms(const WtszCall &c) { return c.ninner; }

// CTA (row tile rt, covariate s) of one call.
template <class Term, class Call>
__device__ __forceinline__ void ordered_sum_tile(const Call &c, int rt, int s) {
  __shared__ double term[2][kTerms][kSumRows];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = sum_rows(c), n = sum_terms(c), i = rt * kSumRows + lane;
  const Term t(c, min(i, rows - 1), s);
  const int tiles = (n + kTerms - 1) / kTerms;
  double acc = 0.0;
  // kAhead: the operands of the next tile and the places of the one after are on
  // their way while a tile's terms are formed.  (Past the last term: the last
  // one's.)
  const int quarter = (int)(blockIdx.x + blockIdx.x / 152) & 3, own = warp & 3;
  const int w = 3 * (warp >> 2) + own - (own > quarter);
  const bool adds = warp == quarter, forms = own != quarter && n > 0;
  typename Term::At at[kTermsPerWarp];
  typename Term::Of of[kTermsPerWarp];
  auto places = [&](int j) {
#pragma unroll
    for (int u = 0; u < kTermsPerWarp; ++u) at[u] = t.at(min(j * kTerms + w + kFormWarps * u, n - 1));
  };
  auto operands = [&]() {
#pragma unroll
    for (int u = 0; u < kTermsPerWarp; ++u) of[u] = t.of(at[u]);
  };
  if (forms && Term::kAhead) {
    places(0);
    operands();
    places(1);
  }
  for (int j = 0; j <= tiles; ++j) {
    if (forms) {
      if (j < tiles) {
        double v[kTermsPerWarp];
#pragma unroll
        for (int u = 0; u < kTermsPerWarp; ++u) {
          if (!Term::kAhead) of[u] = t.of(t.at(min(j * kTerms + w + kFormWarps * u, n - 1)));
          v[u] = t(of[u]);
        }
        if (Term::kAhead) {
          operands();
          places(j + 2);
        }
#pragma unroll
        for (int u = 0; u < kTermsPerWarp; ++u) term[j & 1][w + kFormWarps * u][lane] = v[u];
      }
    } else if (adds && j > 0) {
      const int m = min(kTerms, n - (j - 1) * kTerms);
      const double(*q)[kSumRows] = term[(j - 1) & 1];
#pragma unroll 8
      for (int k = 0; k < m; ++k) acc = __dadd_rn(acc, q[k][lane]);
    }
    __syncthreads();
  }
  if (adds && i < rows) c.out[c.out_r[i] + c.s_off[s]] = acc;
}

__global__ void __launch_bounds__(kSumT, SwnytTerm::kCtas) anzt_s_wnyt_kernel(SwnytCall c) {
  ordered_sum_tile<SwnytTerm>(c, blockIdx.x, blockIdx.y);
}
__global__ void __launch_bounds__(kSumT, WtszTerm::kCtas) attyn_wtszn_kernel(WtszCall c) {
  ordered_sum_tile<WtszTerm>(c, blockIdx.x, blockIdx.y);
}

// Several calls in one launch (a deferred group, lakgb_defer_end): CTA k
// belongs to the last call whose tile0 <= k; within it, row tile (k - tile0)
// % row tiles, covariate (k - tile0) / row tiles.
template <class Term, class Call>
__device__ __forceinline__ void ordered_sum_group(const Call *calls, int n) {
  const int k = blockIdx.x;
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (calls[mid].tile0 <= k) lo = mid; else hi = mid - 1;
  }
  const Call c = calls[lo];
  const int rtiles = (sum_rows(c) + kSumRows - 1) / kSumRows;
  const int j = k - c.tile0;
  ordered_sum_tile<Term>(c, j % rtiles, j / rtiles);
}
__global__ void __launch_bounds__(kSumT, SwnytTerm::kCtas) anzt_s_wnyt_group_kernel(const SwnytCall *calls, int n) {
  ordered_sum_group<SwnytTerm>(calls, n);
}
__global__ void __launch_bounds__(kSumT, WtszTerm::kCtas) attyn_wtszn_group_kernel(const WtszCall *calls, int n) {
  ordered_sum_group<WtszTerm>(calls, n);
}

// The calls a deferral scope holds back (this host thread): their device
// inputs and outputs, and where each output goes on the host.
struct SwnytDeferred {
  SwnytCall c{};
  std::vector<DBuf> keep;   // uploads and the device output
  double *host_out = nullptr;
  unsigned long long length = 0;
};

struct WtszDeferred {
  WtszCall c{};
  std::vector<DBuf> keep;
  double *host_out = nullptr;
  unsigned long long length = 0;
};
thread_local int t_defer_depth = 0;
thread_local std::vector<SwnytDeferred> t_swnyt;
thread_local std::vector<WtszDeferred> t_wtsz;
struct DeferKind { void (*enqueue)(); void (*clear)(); };
thread_local std::vector<DeferKind> t_kinds;  // groups of other translation units
struct DeferCopy { double *host; DBuf dev; unsigned long long length; };
thread_local std::vector<DeferCopy> t_copies;  // other calls' outputs

// Page-locked host chunks and their device twins for held-back calls'
// inputs: bump-allocated, 16-byte aligned; `sent` is how much has been
// copied.  Arrays larger than a chunk get a chunk of their own.  Reset (not
// freed) when the outermost scope ends; kept in the thread's ThreadBuffers.

// Page-locked buffer for a scope's small outputs: a copy into pageable memory
// holds the host for about 8 us (and until the kernels before it are done), one
// into page-locked memory under 1 us, so outputs of up to kDownEach bytes come
// back there, as far as they fit, and are copied on after the scope's one wait.
constexpr size_t kDownEach = 64u << 10;
struct DownCopy { double *host; size_t off, bytes; };

// Wait for the copies into the page-locked buffer and pass them on.
void finish_down(std::vector<DownCopy> &later) {
  LAKGB_CUDA(cudaStreamSynchronize(stream()));
  for (const DownCopy &c : later) memcpy(c.host, thread_buffers().down + c.off, c.bytes);
  later.clear();
}

// Enqueue the copy of `length` doubles of `dev` to `host`.  Where two calls of a
// scope write the same host memory the later copy's values stay: a direct copy
// comes after the held-back ones that it overlaps.
void copy_down(double *host, const double *dev, unsigned long long length, size_t &used, std::vector<DownCopy> &later) {
  const size_t bytes = length * sizeof(double);
  if (!bytes) return;
  if (bytes > kDownEach || used + bytes > kDownBytes) {
    const auto at = [](const double *p) { return reinterpret_cast<uintptr_t>(p); };
    for (const DownCopy &c : later)
      if (at(c.host) < at(host) + bytes && at(host) < at(c.host) + c.bytes) {
        finish_down(later);
        break;
      }
    LAKGB_CUDA(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, stream()));
    return;
  }
  uint8_t *&down = thread_buffers().down;
  if (!down) LAKGB_CUDA(cudaHostAlloc((void **)&down, kDownBytes, cudaHostAllocDefault));
  LAKGB_CUDA(cudaMemcpyAsync(down + used, dev, bytes, cudaMemcpyDeviceToHost, stream()));
  later.push_back(DownCopy{host, used, bytes});
  used += (bytes + 15) & ~(size_t)15;
}
}  // namespace

bool defer_active() { return t_defer_depth > 0; }

const void *defer_put(const void *h, size_t n) {
  ThreadBuffers &b = thread_buffers();
  const size_t need = (n + 15) & ~(size_t)15;
  while (b.up_cur < b.up.size() && b.up[b.up_cur].used + need > b.up[b.up_cur].cap) ++b.up_cur;
  if (b.up_cur == b.up.size()) {
    if (!b.up.empty()) defer_flush();  // the earlier chunks' pending bytes go first
    UpChunk c;
    c.cap = std::max(kUpChunk, need);
    LAKGB_CUDA(cudaHostAlloc((void **)&c.h, c.cap, cudaHostAllocDefault));
    LAKGB_CUDA(cudaMalloc((void **)&c.d, c.cap));
    b.up.push_back(c);
  }
  UpChunk &c = b.up[b.up_cur];
  if (n) memcpy(c.h + c.used, h, n);
  const void *d = c.d + c.used;
  c.used += need;
  return d;
}

void defer_flush() {
  for (UpChunk &c : thread_buffers().up) {
    if (c.used > c.sent)
      LAKGB_CUDA(cudaMemcpyAsync(c.d + c.sent, c.h + c.sent, c.used - c.sent, cudaMemcpyHostToDevice, stream()));
    c.sent = c.used;
  }
}

void defer_copy(double *host, DBuf &&dev, unsigned long long length) {
  t_copies.push_back(DeferCopy{host, std::move(dev), length});
}

void defer_register(void (*enqueue)(), void (*clear)()) {
  for (const DeferKind &k : t_kinds)
    if (k.enqueue == enqueue) return;
  t_kinds.push_back({enqueue, clear});
}

}  // namespace lakgb

using namespace lakgb;

extern "C" int wrap_AnZt_S_WnYt_vv__run(int *tidx, void **vpra, pthread_t *thread_in, int output_spacing_a,
                                        int output_spacing_s, M_handle *M_An, M_handle *M_St, M_handle *M_Zn,
                                        L_handle *lf_AnZt, L_handle *lf_YnWt, L_handle **output_p) {
  LAKGB_PROFILE_CALL("wrap_AnZt_S_WnYt_vv__run");
  (void)tidx; (void)vpra; (void)thread_in;
  const unsigned long long length_a = spacing_length(output_spacing_a, M_An);
  const unsigned long long length_s = spacing_length(output_spacing_s, M_St);
  const unsigned long long length = length_a * length_s;
  L_handle *out = ensure_output(output_p, length, "wrap_AnZt_S_WnYt_vv__run", false);
  HostOutputFill fill{out, length};
  if (!out) return (int)length;
  out->spacing_row = output_spacing_a; out->row_stride = length_a;
  out->spacing_col = output_spacing_s; out->col_stride = length_s;
  const int nA = (int)M_An->rpop_j, nZ = (int)M_Zn->rpop_j, nS = (int)M_St->rpop_j;
  if (!lf_AnZt || !lf_YnWt || nA == 0 || nS == 0) return (int)length;
  using Idx = unsigned long long;
  const auto a_r = spacing_index_of<Idx>(lf_AnZt->spacing_row, M_An, nA);
  const auto y_r = spacing_index_of<Idx>(lf_YnWt->spacing_row, M_An, nA);
  const auto out_r = spacing_index_of<Idx>(output_spacing_a, M_An, nA);
  const auto a_c = spacing_index_of<Idx>(lf_AnZt->spacing_col, M_Zn, nZ, lf_AnZt->row_stride);
  const auto y_c = spacing_index_of<Idx>(lf_YnWt->spacing_col, M_Zn, nZ, lf_YnWt->row_stride);
  std::vector<Idx> s_off(nS);
  std::vector<int8_t> vS((size_t)nS * (nZ > 0 ? nZ : 1));
  for (int s = 0; s < nS; ++s) {
    s_off[s] = pick_u(output_spacing_s, s, M_St->m_b_[s], M_St->m_a_[s]) * length_a;
    const unsigned char *st = M_St->wX + (size_t)M_St->m_b_[s] * M_St->mc_length;
    for (int k = 0; k < nZ; ++k) {
      vS[(size_t)s * nZ + k] = (int8_t)lakbcc::bget_pm(st, M_Zn->m_a_[k]);
      if (!lakbcc::bget_on(M_St->mc_j, M_Zn->m_a_[k]))
        printf(" %% Warning! bit %d,%d,%d off in M_St->mc_j\n", k, (int)M_Zn->m_b_[k], (int)M_Zn->m_a_[k]);
    }
  }
  if (max_index(a_r) + max_index(a_c) >= populated(lf_AnZt, false) ||
      max_index(y_r) + max_index(y_c) >= populated(lf_YnWt, false)) {
    set_error(4, "wrap_AnZt_S_WnYt_vv__run: L_handle smaller than the rows and columns it is indexed by");
    return (int)length;
  }
  // Mirrored matrices (lmirror.cu) are read in place.
  Mirror *mA = find_mirror(lf_AnZt), *mY = find_mirror(lf_YnWt);
  // Inside a deferral scope the uploads are owned buffers (they must outlive
  // the call), and the kernel runs at the end of the scope.
  const bool defer = t_defer_depth > 0;
  std::optional<Stager> st;
  if (!defer) st.emplace();
  DBuf dA = mA ? DBuf() : upload_L(lf_AnZt, false);
  DBuf dY = (mY || lf_YnWt == lf_AnZt) ? DBuf() : upload_L(lf_YnWt, false);
  const double *pA = mA ? mA->d : dA.as<double>();
  const double *pY = mY ? mY->d : ((lf_YnWt == lf_AnZt) ? pA : dY.as<double>());
  auto up = [&](const auto &v) { return defer ? defer_upload(v) : upload_vec(v); };
  DBuf d_ar = up(a_r), d_yr = up(y_r), d_ac = up(a_c), d_yc = up(y_c);
  DBuf d_vS = up(vS), d_or = up(out_r), d_so = up(s_off);
  if (defer) defer_flush();
  DBuf d_out(length * sizeof(double));
  if ((unsigned long long)nA * nS != length) d_out.zero();
  SwnytCall c{};
  c.A = pA; c.a_r = d_ar.as<unsigned long long>(); c.a_c = d_ac.as<unsigned long long>();
  c.Y = pY; c.y_r = d_yr.as<unsigned long long>(); c.y_c = d_yc.as<unsigned long long>();
  c.vS = d_vS.as<int8_t>(); c.nA = nA; c.nZ = nZ; c.nS = nS;
  c.out_r = d_or.as<unsigned long long>(); c.s_off = d_so.as<unsigned long long>(); c.out = d_out.as<double>();
  if (defer) {
    SwnytDeferred d;
    d.c = c;
    d.host_out = out->lf;
    d.length = length;
    fill.copied = true;
    for (DBuf *b : {&dA, &dY, &d_ar, &d_yr, &d_ac, &d_yc, &d_vS, &d_or, &d_so, &d_out}) d.keep.push_back(std::move(*b));
    t_swnyt.push_back(std::move(d));
    return (int)length;
  }
  st->flush();
  anzt_s_wnyt_kernel<<<dim3((nA + kSumRows - 1) / kSumRows, nS), kSumT, 0, stream()>>>(c);
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
  copy_back(out->lf, d_out, length, &fill);
  return (int)length;
}

// Deferral scope: AnZt_S_WnYt and AtTYn____WtSZn calls made inside it (the
// reference runs them on thread slots and joins them afterwards,
// GLOBAL_pthread_tuc) are held back and run together when the outermost scope
// ends -- one grouped launch per kind, then every output copied into its host
// L_handle.  Outputs are not to be read before the scope ends.
extern "C" void lakgb_defer_begin(void) { ++t_defer_depth; }

extern "C" void lakgb_defer_end(void) {
  if (t_defer_depth <= 0 || --t_defer_depth > 0) return;
  if (t_swnyt.empty() && t_wtsz.empty() && t_kinds.empty() && t_copies.empty()) return;
  LAKGB_PROFILE_CALL("lakgb_defer_end");
  std::vector<SwnytCall> c1;
  std::vector<WtszCall> c2;
  int tiles1 = 0, tiles2 = 0;
  for (auto &d : t_swnyt) {
    d.c.tile0 = tiles1;
    tiles1 += ((d.c.nA + kSumRows - 1) / kSumRows) * d.c.nS;
    c1.push_back(d.c);
  }
  for (auto &d : t_wtsz) {
    d.c.tile0 = tiles2;
    tiles2 += ((d.c.npairs + kSumRows - 1) / kSumRows) * d.c.nS;
    c2.push_back(d.c);
  }
  {
    DBuf d_c1, d_c2;
    if (!c1.empty()) {
      d_c1 = defer_upload(c1);
      defer_flush();
      anzt_s_wnyt_group_kernel<<<tiles1, kSumT, 0, stream()>>>(d_c1.as<SwnytCall>(), (int)c1.size());
      LAKGB_CUDA(cudaGetLastError());
      count_launch();
    }
    if (!c2.empty()) {
      d_c2 = defer_upload(c2);
      defer_flush();
      attyn_wtszn_group_kernel<<<tiles2, kSumT, 0, stream()>>>(d_c2.as<WtszCall>(), (int)c2.size());
      LAKGB_CUDA(cudaGetLastError());
      count_launch();
    }
    for (const DeferKind &k : t_kinds) k.enqueue();
    if (profile_calls_on()) {
      LAKGB_PROFILE_CALL("(kernel wait)");
      LAKGB_CUDA(cudaStreamSynchronize(stream()));
    }
    LAKGB_PROFILE_CALL("(copy back + sync)");
    std::vector<DownCopy> later;
    size_t used = 0;
    for (auto &d : t_swnyt) copy_down(d.host_out, d.c.out, d.length, used, later);
    for (auto &d : t_wtsz) copy_down(d.host_out, d.c.out, d.length, used, later);
    for (auto &c : t_copies) copy_down(c.host, c.dev.as<double>(), c.length, used, later);
    finish_down(later);
  }
  t_copies.clear();
  for (UpChunk &c : thread_buffers().up) c.used = c.sent = 0;  // the stream has drained: reuse the chunks
  thread_buffers().up_cur = 0;
  t_swnyt.clear();
  t_wtsz.clear();
  for (const DeferKind &k : t_kinds) k.clear();
  t_kinds.clear();
}

extern "C" int wrap_AtTYn____WtSZn_vv__run(int *tidx, void **vpra, pthread_t *thread_in, int output_spacing_a,
                                           int output_spacing_s, M_handle *M_At, M_handle *M_Tt, M_handle *M_Yt,
                                           M_handle *M_Wt, M_handle *M_St, M_handle *M_Zt, double *Y_ajdk,
                                           L_handle *lf_AtTYn, L_handle *lf_ZtSWn, L_handle **output_p) {
  LAKGB_PROFILE_CALL("wrap_AtTYn____WtSZn_vv__run");
  (void)tidx; (void)vpra; (void)thread_in; (void)M_Tt;
  const unsigned long long length_a = spacing_length(output_spacing_a, M_At);
  const unsigned long long length_s = spacing_length(output_spacing_s, M_St);
  const unsigned long long length = length_a * length_s;
  L_handle *out = ensure_output(output_p, length, "wrap_AtTYn____WtSZn_vv__run", false);
  HostOutputFill fill{out, length};
  if (!out) return (int)length;
  out->spacing_row = output_spacing_a; out->row_stride = length_a;
  out->spacing_col = output_spacing_s; out->col_stride = length_s;
  const int npairs = (int)std::min(M_At->rpop_j, M_Zt->rpop_j);
  const int ninner = (int)std::min(M_Yt->rpop_j, M_Wt->rpop_j);
  const int nS = (int)M_St->rpop_j;
  // no pairs, covariates or inner rows: every sum is empty (the zeros written above)
  if (npairs == 0 || nS == 0 || ninner == 0) return (int)length;
  const int Y_pcols = (int)lakbcc::psize(M_Yt->nrows);
  const double *D_Yn = Y_ajdk + (size_t)lakbcc::AJDK_0_1 * Y_pcols;
  const L_handle *LA = lf_AtTYn, *LZ = lf_ZtSWn;
  using Idx = unsigned long long;
  const auto ay_a = spacing_index_of<Idx>(LA->spacing_row, M_At, npairs);
  const auto zw_z = spacing_index_of<Idx>(LZ->spacing_row, M_Zt, npairs);
  const auto out_r = spacing_index_of<Idx>(output_spacing_a, M_At, npairs);
  const auto ay_y = spacing_index_of<Idx>(LA->spacing_col, M_Yt, ninner, LA->row_stride);
  const auto zw_w = spacing_index_of<Idx>(LZ->spacing_col, M_Wt, ninner, LZ->row_stride);
  std::vector<Idx> ay_s(nS), zw_s(nS), s_off(nS);
  std::vector<double> Dy(ninner);
  for (int k = 0; k < ninner; ++k) Dy[k] = D_Yn[M_Yt->m_a_[k] / lakbcc::POPLENGTH];
  for (int s = 0; s < nS; ++s) {
    ay_s[s] = pick_u(LA->spacing_lyr, s, M_St->m_b_[s], M_St->m_a_[s]) * LA->row_stride * LA->col_stride;
    zw_s[s] = pick_u(LZ->spacing_lyr, s, M_St->m_b_[s], M_St->m_a_[s]) * LZ->row_stride * LZ->col_stride;
    s_off[s] = pick_u(output_spacing_s, s, M_St->m_b_[s], M_St->m_a_[s]) * length_a;
  }
  if (max_index(ay_a) + max_index(ay_y) + max_index(ay_s) >= populated(LA, true) ||
      max_index(zw_z) + max_index(zw_w) + max_index(zw_s) >= populated(LZ, true)) {
    set_error(4, "wrap_AtTYn____WtSZn_vv__run: L_handle smaller than the rows and columns it is indexed by");
    return (int)length;
  }
  // Mirrored inputs (lmirror.cu) are read in place; inside a deferral scope
  // the uploads are owned buffers and the kernel runs when the scope ends.
  Mirror *mLA = find_mirror(LA), *mLZ = find_mirror(LZ);
  const bool defer = t_defer_depth > 0;
  std::optional<Stager> st;
  if (!defer) st.emplace();
  DBuf dA = mLA ? DBuf() : upload_L(LA, true);
  DBuf dZ = (mLZ || LZ == LA) ? DBuf() : upload_L(LZ, true);
  const double *pA = mLA ? mLA->d : dA.as<double>();
  const double *pZ = mLZ ? mLZ->d : ((LZ == LA) ? pA : dZ.as<double>());
  auto up = [&](const auto &v) { return defer ? defer_upload(v) : upload_vec(v); };
  DBuf d_aa = up(ay_a), d_ay = up(ay_y), d_as = up(ay_s);
  DBuf d_zz = up(zw_z), d_zw = up(zw_w), d_zs = up(zw_s);
  DBuf d_D = up(Dy), d_or = up(out_r), d_so = up(s_off);
  if (defer) defer_flush();
  DBuf d_out(length * sizeof(double));
  if ((unsigned long long)npairs * nS != length) d_out.zero();
  WtszCall c{};
  c.AY = pA; c.ay_a = d_aa.as<unsigned long long>(); c.ay_y = d_ay.as<unsigned long long>();
  c.ay_s = d_as.as<unsigned long long>();
  c.ZW = pZ; c.zw_z = d_zz.as<unsigned long long>(); c.zw_w = d_zw.as<unsigned long long>();
  c.zw_s = d_zs.as<unsigned long long>();
  c.Dy = d_D.as<double>(); c.npairs = npairs; c.ninner = ninner; c.nS = nS;
  c.out_r = d_or.as<unsigned long long>(); c.s_off = d_so.as<unsigned long long>(); c.out = d_out.as<double>();
  if (defer) {
    WtszDeferred d;
    d.c = c;
    d.host_out = out->lf;
    d.length = length;
    fill.copied = true;
    for (DBuf *b : {&dA, &dZ, &d_aa, &d_ay, &d_as, &d_zz, &d_zw, &d_zs, &d_D, &d_or, &d_so, &d_out})
      d.keep.push_back(std::move(*b));
    t_wtsz.push_back(std::move(d));
    return (int)length;
  }
  st->flush();
  attyn_wtszn_kernel<<<dim3((npairs + kSumRows - 1) / kSumRows, nS), kSumT, 0, stream()>>>(c);
  LAKGB_CUDA(cudaGetLastError());
  count_launch();
  copy_back(out->lf, d_out, length, &fill);
  return (int)length;
}

namespace {

int attyn_entry(bool symmetric, const char *who, int output_spacing_a, int output_spacing_y, int output_spacing_t,
                M_handle *M_At, M_handle *M_Tt, M_handle *M_Yt, double *A_ajdk, double *Y_ajdk,
                L_handle *lf_AtTn, L_handle *lf_YtTn, L_handle **output_p) {
  const unsigned long long la = spacing_length(output_spacing_a, M_At);
  const unsigned long long ly = spacing_length(output_spacing_y, M_Yt);
  const unsigned long long lt = spacing_length(output_spacing_t, M_Tt);
  const unsigned long long length = la * ly * lt;
  // every element is written where all rows are retained; otherwise the rest is zero
  const bool all = (unsigned long long)M_At->rpop_j * (unsigned long long)M_Yt->rpop_j * (unsigned long long)M_Tt->rpop_j == length &&
                   M_Yt->mc_length == M_At->mc_length && M_Tt->mc_length == M_At->mc_length && (!symmetric || M_At == M_Yt);
  // A mirrored output (lmirror.cu) is produced on the device only.
  Mirror *mo = *output_p ? find_mirror(*output_p) : nullptr;
  L_handle *out = nullptr;
  HostOutputFill fill;
  if (mo) {
    out = *output_p;
    if (out->length < length || mo->n < length) {
      set_error(2, "output length %llu < %llu in %s", out->length, length, who);
      return (int)length;
    }
    if (length && !all) LAKGB_CUDA(cudaMemsetAsync(mo->d, 0, length * sizeof(double), stream()));
    mo->host_stale = true;
  } else {
    out = ensure_output(output_p, length, who, false);
    fill.L = out;
    fill.n = length;
  }
  if (!out) return (int)length;
  out->spacing_row = output_spacing_a; out->row_stride = la;
  out->spacing_col = output_spacing_y; out->col_stride = ly;
  out->spacing_lyr = output_spacing_t; out->lyr_stride = lt;
  const int nA = (int)M_At->rpop_j, nY = (int)M_Yt->rpop_j, nT = (int)M_Tt->rpop_j;
  if (nA == 0 || nY == 0 || nT == 0) return (int)length;
  if (M_Yt->mc_length != M_At->mc_length || M_Tt->mc_length != M_At->mc_length) {
    set_error(4, "%s: rows of unequal length", who);
    return (int)length;
  }
  const int A_pcols = (int)lakbcc::psize(M_At->nrows), Y_pcols = (int)lakbcc::psize(M_Yt->nrows);
  const double *a_An = A_ajdk + (size_t)lakbcc::AJDK_1_0 * A_pcols;
  const double *a_Yn = Y_ajdk + (size_t)lakbcc::AJDK_1_0 * Y_pcols;
  const std::vector<uint32_t> a_rowb(M_At->m_b_, M_At->m_b_ + nA), y_rowb(M_Yt->m_b_, M_Yt->m_b_ + nY);
  std::vector<uint32_t> t_rowb(nT);
  std::vector<double> hhAy((size_t)nT * nA), hhaY((size_t)nT * nY), hhay(nT), aA(nA), aY(nY);
  using Idx = unsigned long long;
  const auto out_a = spacing_index_of<Idx>(output_spacing_a, M_At, nA);
  const auto out_y = spacing_index_of<Idx>(output_spacing_y, M_Yt, nY, la);
  std::vector<Idx> out_t(nT);
  for (int i = 0; i < nA; ++i) aA[i] = a_An[M_At->m_a_[i] / lakbcc::POPLENGTH];
  for (int k = 0; k < nY; ++k) aY[k] = a_Yn[M_Yt->m_a_[k] / lakbcc::POPLENGTH];
  // row indices of the integer sums, read at their covariate's column
  const auto ia = spacing_index_of<Idx>(lf_AtTn->spacing_row, M_At, nA);
  const auto iy = spacing_index_of<Idx>(lf_YtTn->spacing_row, M_Yt, nY);
  for (int t = 0; t < nT; ++t) {
    const unsigned tb = M_Tt->m_b_[t], ta = M_Tt->m_a_[t];
    t_rowb[t] = tb;
    out_t[t] = pick_u(output_spacing_t, t, tb, ta) * la * ly;
    hhay[t] = (double)(-M_Tt->cpop_j + 2ll * popcount_bytes_masked(M_Tt->wX + (size_t)tb * M_Tt->mc_length, M_Tt->mc_j, (long)M_Tt->mc_length));
    const double *ca = lf_AtTn->lf + lakbcc::pick(lf_AtTn->spacing_col, t, tb, ta) * lf_AtTn->row_stride;
    const double *cy = lf_YtTn->lf + lakbcc::pick(lf_YtTn->spacing_col, t, tb, ta) * lf_YtTn->row_stride;
    for (int i = 0; i < nA; ++i) hhAy[(size_t)t * nA + i] = (double)(long long)ca[ia[i]];
    for (int k = 0; k < nY; ++k) hhaY[(size_t)t * nY + k] = (double)(long long)cy[iy[k]];
  }
  AtTYnParams p{};
  Stager st;
  p.At = (const uint8_t *)resident(M_At->wX, (size_t)M_At->rpop_b * M_At->mc_length);
  p.Yt = (const uint8_t *)resident(M_Yt->wX, (size_t)M_Yt->rpop_b * M_Yt->mc_length);
  p.Tt = (const uint8_t *)resident(M_Tt->wX, (size_t)M_Tt->rpop_b * M_Tt->mc_length);
  p.a_row_bytes = p.y_row_bytes = p.t_row_bytes = (long long)M_At->mc_length;
  DBuf d_ar = upload_vec(a_rowb), d_yr = upload_vec(y_rowb), d_tr = upload_vec(t_rowb);
  p.a_rowb = d_ar.as<uint32_t>(); p.y_rowb = d_yr.as<uint32_t>(); p.t_rowb = d_tr.as<uint32_t>();
  p.nA = nA; p.nY = nY;
  DBuf mask = upload_bytes(M_At->mc_j, M_At->mc_length);
  p.mask = mask.as<uint8_t>(); p.P = (int)(M_At->mc_length / kBlockBytes); p.cpop = M_At->cpop_j;
  DBuf d_hAy = upload_vec(hhAy), d_haY = upload_vec(hhaY), d_hay = upload_vec(hhay), d_aA = upload_vec(aA), d_aY = upload_vec(aY);
  DBuf d_oa = upload_vec(out_a), d_oy = upload_vec(out_y), d_ot = upload_vec(out_t);
  p.hhAy = d_hAy.as<double>(); p.hhaY = d_haY.as<double>(); p.hhay = d_hay.as<double>();
  p.aA = d_aA.as<double>(); p.aY = d_aY.as<double>();
  p.out_a = d_oa.as<unsigned long long>(); p.out_y = d_oy.as<unsigned long long>(); p.out_t = d_ot.as<unsigned long long>();
  DBuf d_oa2, d_oy2;
  if (symmetric) {
    // transposed positions: Yt row k as an output row, At row i as a column
    d_oa2 = upload_vec(spacing_index_of<Idx>(output_spacing_a, M_Yt, nY));
    d_oy2 = upload_vec(spacing_index_of<Idx>(output_spacing_y, M_At, nA, la));
    p.symmetric = 1;
    p.out_a2 = d_oa2.as<unsigned long long>();
    p.out_y2 = d_oy2.as<unsigned long long>();
  }
  DBuf d_out;
  if (mo) {
    p.out = mo->d;
  } else {
    d_out = DBuf(length * sizeof(double));
    if (!all) d_out.zero();
    p.out = d_out.as<double>();
  }
  st.flush();
  launch_attyn_tc(p, nT, stream());
  if (mo) return (int)length;
  copy_back(out->lf, d_out, length, &fill);
  return (int)length;
}

}  // namespace

extern "C" int wrap_AtTYn_vv__run(int *tidx, void **vpra, pthread_t *thread_in, int output_spacing_a,
                                  int output_spacing_y, int output_spacing_t, M_handle *M_At, M_handle *M_Tt,
                                  M_handle *M_Yt, double *A_ajdk, double *Y_ajdk, L_handle *lf_AtTn,
                                  L_handle *lf_YtTn, L_handle **output_p) {
  LAKGB_PROFILE_CALL("wrap_AtTYn_vv__run");
  (void)tidx; (void)vpra; (void)thread_in;
  return attyn_entry(false, "wrap_AtTYn_vv__run", output_spacing_a, output_spacing_y, output_spacing_t, M_At, M_Tt,
                     M_Yt, A_ajdk, Y_ajdk, lf_AtTn, lf_YtTn, output_p);
}

extern "C" int wrap_AtTAn_vv__run(int *tidx, void **vpra, pthread_t *thread_in, int output_spacing_a,
                                  int output_spacing_y, int output_spacing_t, M_handle *M_At, M_handle *M_Tt,
                                  M_handle *M_Yt, double *A_ajdk, double *Y_ajdk, L_handle *lf_AtTn,
                                  L_handle *lf_YtTn, L_handle **output_AtTAn_p) {
  LAKGB_PROFILE_CALL("wrap_AtTAn_vv__run");
  (void)tidx; (void)vpra; (void)thread_in;
  return attyn_entry(true, "wrap_AtTAn_vv__run", output_spacing_a, output_spacing_y, output_spacing_t, M_At, M_Tt,
                     M_Yt, A_ajdk, Y_ajdk, lf_AtTn, lf_YtTn, output_AtTAn_p);
}
