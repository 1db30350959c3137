// HBM-bound block kernels: element-wise ops, permute (tensor_block_copy_),
// permuted add/subtract, slice/insert, deterministic dot/norm reductions,
// orbital-energy denominators and the scalar cases of tensor_block_contract_.
//
// Arithmetic follows the reference's operation order with explicit
// round-to-nearest intrinsics (__dmul_rn/__dadd_rn/__dsub_rn), so no multiply
// and add are fused and element-wise results match the reference bit for bit.
#include <algorithm>
#include <cstring>

#include "a4g_internal.h"
#include "exact_fp.h"

namespace a4g {

namespace {

constexpr int kThreads = 256;

int grid_for(int64_t n, int per_thread = 4) {
  const int sms = ctx()->num_sms > 0 ? ctx()->num_sms : 152;
  int64_t want = (n + int64_t(kThreads) * per_thread - 1) / (int64_t(kThreads) * per_thread);
  want = std::max<int64_t>(1, std::min<int64_t>(want, int64_t(sms) * 8));
  return int(want);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// ---------------------------------------------------------------- element-wise
enum class EwOp { kFill, kScale, kScaleCopy, kIncrement, kAddScaled, kAdd, kAxpy };

template <EwOp OP>
__device__ __forceinline__ double ew(double d, double s, double a) {
  if constexpr (OP == EwOp::kFill) return a;
  else if constexpr (OP == EwOp::kScale) return __dmul_rn(d, a);
  else if constexpr (OP == EwOp::kScaleCopy) return __dmul_rn(s, a);
  else if constexpr (OP == EwOp::kIncrement) return __dadd_rn(d, a);
  else if constexpr (OP == EwOp::kAddScaled) return __dadd_rn(d, __dmul_rn(s, a));
  else if constexpr (OP == EwOp::kAdd) return __dadd_rn(d, s);
  else return fma(a, s, d);  // _gpu_axpy: cuBLAS daxpy semantics
}

// Bound by HBM, or by the FP64 pipes where an element takes two operations
// (add_scaled: 340 us for 96^4 elements, of 336 measured).  A CTA per share of
// 256 threads x 4 pairs (a fill: 8), all loaded before the first is stored, and
// no loop.  96^4 elements, grid held to 8 CTAs per SM and one pair at a time ->
// now: scale_copy 234 -> 201 us (24^6: 527 -> 440), add 364 -> 285, fill 108 ->
// 93; two pairs: scale_copy 252; eight: 198, but a 20^4 block 8.9 us, not 7.4.
template <EwOp OP>
struct EwReads {
  static constexpr bool d = !(OP == EwOp::kFill || OP == EwOp::kScaleCopy);
  static constexpr bool s = OP == EwOp::kScaleCopy || OP == EwOp::kAddScaled || OP == EwOp::kAdd || OP == EwOp::kAxpy;
  static constexpr int pairs = d || s ? 4 : 8;
};
template <EwOp OP, bool VEC>
__global__ void __launch_bounds__(kThreads) ew_kernel(double* __restrict__ d,
                                                      const double* __restrict__ s, int64_t n,
                                                      double a) {
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  constexpr bool kReadD = EwReads<OP>::d, kReadS = EwReads<OP>::s;
  constexpr int kEwPairs = EwReads<OP>::pairs;
  if constexpr (VEC) {
    const int64_t n2 = n / 2;
    double2* d2 = reinterpret_cast<double2*>(d);
    const double2* s2 = reinterpret_cast<const double2*>(s);
    for (int64_t b = int64_t(blockIdx.x) * blockDim.x * kEwPairs + threadIdx.x; b < n2; b += kEwPairs * stride) {
      double2 dv[kEwPairs], sv[kEwPairs];
#pragma unroll
      for (int u = 0; u < kEwPairs; ++u) {
        const int64_t k = b + u * int64_t(blockDim.x);
        dv[u] = kReadD && k < n2 ? d2[k] : make_double2(0.0, 0.0);
        sv[u] = kReadS && k < n2 ? __ldg(&s2[k]) : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < kEwPairs; ++u) {
        const int64_t k = b + u * int64_t(blockDim.x);
        if (k < n2) d2[k] = make_double2(ew<OP>(dv[u].x, sv[u].x, a), ew<OP>(dv[u].y, sv[u].y, a));
      }
    }
    if (i == 0 && (n & 1)) {
      const int64_t k = n - 1;
      d[k] = ew<OP>(kReadD ? d[k] : 0.0, kReadS ? s[k] : 0.0, a);
    }
  } else {
    for (int64_t k = i; k < n; k += stride) d[k] = ew<OP>(kReadD ? d[k] : 0.0, kReadS ? s[k] : 0.0, a);
  }
}

template <EwOp OP>
int launch_ew(double* d, const double* s, int64_t n, double a, cudaStream_t st) {
  if (n < 0) return fail(A4G_ERR_ARG, "negative element count");
  if (n == 0) return A4G_OK;
  if (!d) return fail(A4G_ERR_ARG, "null block pointer");
  const bool vec = aligned16(d) && (s == nullptr || aligned16(s));
  constexpr int kShare = EwReads<OP>::pairs * kThreads;
  const int64_t g = std::max<int64_t>(1, std::min<int64_t>((n / 2 + kShare - 1) / kShare, 0x7fffffff));
  if (vec) ew_kernel<OP, true><<<unsigned(g), kThreads, 0, st>>>(d, s, n, a);
  else ew_kernel<OP, false><<<grid_for(n), kThreads, 0, st>>>(d, s, n, a);
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

// ---------------------------------------------------------------- permute
constexpr int kPermMax = kMaxRank;

struct PermParams {
  int rank;           // after merging
  int a_dim, b_dim;   // input dim 0 (read-contiguous), input dim that is output dim 0
  int ext[kPermMax];  // input-order extents
  int64_t sin[kPermMax], sout[kPermMax];  // strides of each input dim in input / output
  int rest_dims[kPermMax];                // input dims other than a_dim, b_dim
  int n_rest;
  int64_t n_rest_total;
};

// Describes a permute after dropping unit extents and merging runs of input
// dims that stay adjacent and in order in the output (input dim i and i+1 merge
// when their output positions are consecutive).  o2n is 0-based.
void make_perm(int rank, const int* ext, const int* o2n, PermParams* p) {
  int e[kPermMax], o[kPermMax], r = 0;
  for (int i = 0; i < rank; ++i)
    if (ext[i] != 1) {
      e[r] = ext[i];
      o[r] = o2n[i];
      ++r;
    }
  int dense[kPermMax];
  for (int i = 0; i < r; ++i) {
    int c = 0;
    for (int j = 0; j < r; ++j) c += o[j] < o[i];
    dense[i] = c;
  }
  int ge[kPermMax], gpos[kPermMax], m = 0;
  for (int i = 0; i < r; ++i) {
    if (i > 0 && dense[i] == dense[i - 1] + 1) {
      ge[m - 1] *= e[i];
      continue;
    }
    ge[m] = e[i];
    gpos[m] = dense[i];
    ++m;
  }
  int ord[kPermMax];
  for (int i = 0; i < m; ++i) ord[i] = i;
  std::sort(ord, ord + m, [&](int x, int y) { return gpos[x] < gpos[y]; });
  int64_t so = 1;
  for (int q = 0; q < m; ++q) {
    p->sout[ord[q]] = so;
    so *= ge[ord[q]];
  }
  int64_t si = 1;
  for (int i = 0; i < m; ++i) {
    p->ext[i] = ge[i];
    p->sin[i] = si;
    si *= ge[i];
  }
  p->rank = m;
  p->a_dim = 0;
  p->b_dim = m > 0 ? ord[0] : 0;
  p->n_rest = 0;
  p->n_rest_total = 1;
  for (int i = 0; i < m; ++i)
    if (i != p->a_dim && i != p->b_dim) {
      p->rest_dims[p->n_rest++] = i;
      p->n_rest_total *= ge[i];
    }
}

// Element op of the permute family: OP 0 out = r (permute), 1 out = l + r,
// 2 out = l - r (block add/subtract with a permuted right operand).
template <int OP>
__device__ __forceinline__ double perm_op(const double* l, int64_t o, double rv) {
  if constexpr (OP == 0) return rv;
  else if constexpr (OP == 1) return __dadd_rn(l[o], rv);
  else return __dsub_rn(l[o], rv);
}

// Division of an unsigned below 2^31 by d: x * mul >> 31 + shift, exact.
struct FastDiv {
  unsigned mul;
  int shift;
};
FastDiv fast_div(unsigned d) {
  FastDiv f{0, 0};
  while ((uint64_t(1) << f.shift) < d) ++f.shift;
  f.mul = unsigned(((uint64_t(1) << (31 + f.shift)) + d - 1) / d);
  return f;
}
__device__ __forceinline__ unsigned fast_quot(unsigned x, FastDiv f) {
  return unsigned((uint64_t(x) * f.mul) >> (31 + f.shift));
}

// Input dim 0 is also output dim 0: runs of dim 0 are contiguous on both
// sides.  As T (pairs where every run starts on 16 bytes and has an even length,
// else single elements), kPermLoads a thread in input order, all loaded before
// the first is stored; fewer than 2^31 elements.  (A CTA per 96-element run:
// 432 us on 96^4 elements, 199 now; with an addition 464 and 290.)
constexpr int kPermLoads = 4;
struct PermRuns {
  int rank;
  unsigned ext[kPermMax];
  FastDiv div[kPermMax];
  int64_t sout[kPermMax];
};
template <int OP, class T>
__global__ void __launch_bounds__(kThreads) perm_runs_kernel(PermRuns p, const T* __restrict__ in, T* out, const T* l,
                                                             unsigned n) {
  const unsigned first = blockIdx.x * (kThreads * kPermLoads) + threadIdx.x;
  int64_t at[kPermLoads];
  T v[kPermLoads], lv[kPermLoads];
#pragma unroll
  for (int u = 0; u < kPermLoads; ++u) {
    const unsigned i = first + u * kThreads;
    unsigned rem = i;
    int64_t o = 0;
    for (int q = 0; q < p.rank - 1; ++q) {
      const unsigned d = fast_quot(rem, p.div[q]);
      o += int64_t(rem - d * p.ext[q]) * p.sout[q];
      rem = d;
    }
    at[u] = o + int64_t(rem) * p.sout[p.rank - 1];
    if (i < n) {
      v[u] = in[i];
      if constexpr (OP != 0) lv[u] = l[at[u]];
    }
  }
#pragma unroll
  for (int u = 0; u < kPermLoads; ++u) {
    if (first + u * kThreads >= n) continue;
    if constexpr (OP == 0) {
      out[at[u]] = v[u];
    } else if constexpr (sizeof(T) == sizeof(double2)) {
      T x;
      x.x = OP == 1 ? __dadd_rn(lv[u].x, v[u].x) : __dsub_rn(lv[u].x, v[u].x);
      x.y = OP == 1 ? __dadd_rn(lv[u].y, v[u].y) : __dsub_rn(lv[u].y, v[u].y);
      out[at[u]] = x;
    } else {
      out[at[u]] = OP == 1 ? __dadd_rn(lv[u], v[u]) : __dsub_rn(lv[u], v[u]);
    }
  }
}

// The same beyond 2^31 elements: a block takes several runs and decodes each
// run's output offset once.
template <int OP>
__global__ void __launch_bounds__(kThreads) perm_direct_kernel(PermParams p, const double* __restrict__ in,
                                                               double* out, const double* l, int64_t nruns,
                                                               int runs_per_block) {
  const int E0 = p.ext[0];
  const int64_t r0 = int64_t(blockIdx.x) * runs_per_block;
  const int64_t r1 = r0 + runs_per_block < nruns ? r0 + runs_per_block : nruns;
  for (int64_t run = r0; run < r1; ++run) {
    int64_t rem = run, base_out = 0;
    for (int q = 1; q < p.rank; ++q) {
      const int64_t x = rem % p.ext[q];
      rem /= p.ext[q];
      base_out += x * p.sout[q];
    }
    const int64_t base_in = run * E0;
    for (int e = threadIdx.x; e < E0; e += blockDim.x)
      out[base_out + e] = perm_op<OP>(l, base_out + e, __ldg(&in[base_in + e]));
  }
}

// Shared-memory tiled transpose between input dim a (contiguous reads) and
// input dim b (contiguous writes); the remaining dims index the grid, several
// of them per block (a block moves 16 KB per slice, so one slice per block
// would be bound by block scheduling, not by HBM).
constexpr int kTile = 32;
template <int OP>
__global__ void __launch_bounds__(kTile * 8) perm_tiled_kernel(PermParams p, const double* __restrict__ in,
                                                               double* out, const double* l,
                                                               int rest_per_block) {
  __shared__ double tile[2][kTile][kTile + 1];
  const int Ea = p.ext[p.a_dim], Eb = p.ext[p.b_dim];
  const int ta = (Ea + kTile - 1) / kTile, tb = (Eb + kTile - 1) / kTile;
  const int64_t tiles = int64_t(ta) * tb;
  const int64_t t = blockIdx.x % tiles;
  const int ia = int(t % ta), ib = int(t / ta);
  const int64_t rest0 = (blockIdx.x / tiles) * rest_per_block;
  const int64_t rest1 = rest0 + rest_per_block < p.n_rest_total ? rest0 + rest_per_block : p.n_rest_total;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int a0 = ia * kTile, b0 = ib * kTile;
  const int64_t sb_in = p.sin[p.b_dim], sa_out = p.sout[p.a_dim];
  // two slices per iteration: eight loads in flight per thread before the
  // first shared-memory write
  for (int64_t rest = rest0; rest < rest1; rest += 2) {
    int64_t bin[2], bout[2];
    bool have[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      have[u] = rest + u < rest1;
      int64_t rem = rest + u, bi = 0, bo = 0;
      for (int q = 0; q < p.n_rest; ++q) {
        const int d = p.rest_dims[q];
        const int64_t x = rem % p.ext[d];
        rem /= p.ext[d];
        bi += x * p.sin[d];
        bo += x * p.sout[d];
      }
      bin[u] = bi;
      bout[u] = bo;
    }
    double v[2][kTile / 8];
    double lv[2][kTile / 8];  // add/subtract: the left operand at this thread's store positions
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int k = 0; k < kTile / 8; ++k) {
        const int a = a0 + tx, b = b0 + ty + 8 * k;
        v[u][k] = (have[u] && a < Ea && b < Eb) ? __ldg(&in[bin[u] + a + int64_t(b) * sb_in]) : 0.0;
        if constexpr (OP != 0) {
          const int bs = b0 + tx, as = a0 + ty + 8 * k;
          lv[u][k] = (have[u] && as < Ea && bs < Eb) ? l[bout[u] + bs + int64_t(as) * sa_out] : 0.0;
        }
      }
    __syncthreads();  // the previous iteration's stores have read the tiles
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int k = 0; k < kTile / 8; ++k) tile[u][ty + 8 * k][tx] = v[u][k];
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (!have[u]) continue;
#pragma unroll
      for (int k = 0; k < kTile / 8; ++k) {
        const int b = b0 + tx, a = a0 + ty + 8 * k;
        if (a < Ea && b < Eb) {
          const int64_t o = bout[u] + b + int64_t(a) * sa_out;
          const double rv = tile[u][tx][ty + 8 * k];
          if constexpr (OP == 0) out[o] = rv;
          else out[o] = OP == 1 ? __dadd_rn(lv[u][k], rv) : __dsub_rn(lv[u][k], rv);
        }
      }
    }
  }
}

// Launches the permute family for a described permute (make_perm) of
// `total` elements: OP 0 permute in -> out; 1 / 2: out = l +/- permute(in).
template <int OP>
int launch_perm_op(const PermParams& p, const double* in, double* out, const double* l, int64_t total,
                   cudaStream_t s) {
  const int sms = ctx()->num_sms > 0 ? ctx()->num_sms : 152;
  if (p.rank <= 1 || p.b_dim == p.a_dim) {
    if (total <= 0) return A4G_OK;
    if (total <= 0x7fffffff - kThreads * kPermLoads) {
      PermRuns r{};
      r.rank = std::max(1, p.rank);
      bool pairs = aligned16(in) && aligned16(out) && (OP == 0 || aligned16(l)) && (p.ext[0] & 1) == 0;
      for (int q = 1; q < p.rank; ++q) pairs = pairs && (p.sout[q] & 1) == 0;
      for (int q = 0; q < r.rank; ++q) {
        r.ext[q] = unsigned(q == 0 && pairs ? p.ext[0] / 2 : p.ext[q]);
        r.sout[q] = q > 0 && pairs ? p.sout[q] / 2 : p.sout[q];
        r.div[q] = fast_div(r.ext[q]);
      }
      const unsigned n = unsigned(pairs ? total / 2 : total), grid = (n + kThreads * kPermLoads - 1) / (kThreads * kPermLoads);
      if (pairs)
        perm_runs_kernel<OP><<<grid, kThreads, 0, s>>>(r, reinterpret_cast<const double2*>(in), reinterpret_cast<double2*>(out),
                                                       reinterpret_cast<const double2*>(l), n);
      else perm_runs_kernel<OP><<<grid, kThreads, 0, s>>>(r, in, out, l, n);
      A4G_CUDA(cudaGetLastError());
      return A4G_OK;
    }
    const int E0 = p.rank >= 1 ? p.ext[0] : 1;
    const int64_t nruns = total / E0;
    const int threads = E0 >= kThreads ? kThreads : (E0 + 31) / 32 * 32;
    const int rpb = int(std::max<int64_t>(1, std::min<int64_t>(64, nruns / (int64_t(sms) * 16))));
    const int64_t blocks = (nruns + rpb - 1) / rpb;
    if (blocks > 0x7fffffffLL) return fail(A4G_ERR_RANGE, "permute grid too large");
    if (blocks > 0) perm_direct_kernel<OP><<<unsigned(blocks), threads, 0, s>>>(p, in, out, l, nruns, rpb);
  } else {
    const int Ea = p.ext[p.a_dim], Eb = p.ext[p.b_dim];
    const int64_t tiles = int64_t((Ea + kTile - 1) / kTile) * ((Eb + kTile - 1) / kTile);
    // 2 to 16 slices a block, the most that leave 16 blocks an SM: with fewer
    // blocks the last wave costs more than the blocks' starts (33 x 20 x 29 x 20:
    // 6.2 us by 2, 12.4 by 16), with many the starts do (24^6: 1050 us by 2, 962 by
    // 4, 922 by 16; 96^4 260, 250 and 248; 30 x 100 x 30 x 100 39, 37 and 46)
    int rpb = 2;
    while (rpb < 16 && p.n_rest_total * tiles / (int64_t(sms) * 16) >= 2 * rpb) rpb *= 2;
    const int64_t blocks = tiles * ((p.n_rest_total + rpb - 1) / rpb);
    if (blocks > 0x7fffffffLL) return fail(A4G_ERR_RANGE, "permute grid too large");
    perm_tiled_kernel<OP><<<unsigned(blocks), dim3(kTile, 8), 0, s>>>(p, in, out, l, rpb);
  }
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

// ---------------------------------------------------------------- reductions
constexpr int kDotBlocks = Context::kReducePartials;  // partials of a reduction: at most so many CTAs

// Deterministic sum of acc over the grid, in the launch that forms it: every
// CTA writes its sum, and the last one to arrive adds them in a fixed order.
// True, with the total, in one thread of the grid; the counter is back at zero
// afterwards.  (A second kernel for the partials cost 4 us a call.)
__device__ __forceinline__ bool grid_sum(double acc, double* partial, unsigned* counter, double* total) {
  __shared__ double red[32];
  __shared__ unsigned last;
  const int nw = int(blockDim.x + 31) / 32, lane = int(threadIdx.x) & 31;
  const unsigned blocks = gridDim.x * gridDim.y, self = blockIdx.y * gridDim.x + blockIdx.x;
  auto block_sum = [&]() {  // in thread 0
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
      for (int w = 0; w < nw; ++w) s += red[w];
    return s;
  };
  const double s = block_sum();
  if (threadIdx.x == 0) {
    __stcg(partial + self, s);
    unsigned arrived;  // releases the partial, and acquires the others' for the last one
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(arrived) : "l"(counter) : "memory");
    last = arrived == blocks - 1 ? 1u : 0u;
  }
  __syncthreads();
  if (!last) return false;
  acc = 0.0;
  for (unsigned q = threadIdx.x; q < blocks; q += 8 * blockDim.x) {  // eight loads in flight
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = q + k * blockDim.x < blocks ? __ldcg(partial + q + k * blockDim.x) : 0.0;
#pragma unroll
    for (int k = 0; k < 8; k += 2) acc += v[k] + v[k + 1];
  }
  const double sum = block_sum();
  if (threadIdx.x != 0) return false;
  *counter = 0u;
  *total = sum;
  return true;
}

// ---------------------------------------------------------------- dot / norm
// *out (=|+=) sum_i a[offA[i]] b[offB[i]] (full contraction).
__global__ void __launch_bounds__(kThreads) dot_kernel(const double* __restrict__ a, const double* __restrict__ b,
                                                       const int64_t* __restrict__ offA,
                                                       const int64_t* __restrict__ offB, int64_t n, double* out,
                                                       int beta, double* partial, unsigned* counter) {
  double acc = 0.0;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
    acc = fma(a[offA[i]], b[offB[i]], acc);
  double total;
  if (grid_sum(acc, partial, counter, &total)) *out = beta ? *out + total : total;
}

// *out = sum_i a[i]^2: eight 16-byte loads in flight per thread (one 8-byte
// load at a time ran at 61 % of the copy bandwidth), four running sums.
__global__ void __launch_bounds__(kThreads) norm2_kernel(const double* __restrict__ a, int64_t n, int vec, double* out,
                                                         double* partial, unsigned* counter) {
  constexpr int kLoads = 8;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  const int64_t stride = int64_t(gridDim.x) * blockDim.x, first = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  int64_t done = 0;  // elements taken as pairs
  if (vec) {
    const double2* a2 = reinterpret_cast<const double2*>(a);
    const int64_t n2 = n / 2;
    done = 2 * n2;
    int64_t i = first;
    for (; i + (kLoads - 1) * stride < n2; i += kLoads * stride) {
      double2 v[kLoads];
#pragma unroll
      for (int k = 0; k < kLoads; ++k) v[k] = __ldg(a2 + i + k * stride);
#pragma unroll
      for (int k = 0; k < kLoads; ++k) {
        acc[2 * (k & 1)] = fma(v[k].x, v[k].x, acc[2 * (k & 1)]);
        acc[2 * (k & 1) + 1] = fma(v[k].y, v[k].y, acc[2 * (k & 1) + 1]);
      }
    }
    for (; i < n2; i += stride) {
      const double2 v = __ldg(a2 + i);
      acc[0] = fma(v.x, v.x, acc[0]);
      acc[1] = fma(v.y, v.y, acc[1]);
    }
  }
  for (int64_t i = done + first; i < n; i += stride) acc[0] = fma(a[i], a[i], acc[0]);
  double total;
  if (grid_sum((acc[0] + acc[1]) + (acc[2] + acc[3]), partial, counter, &total)) *out = total;
}

// ---------------------------------------------------------------- slice/insert
struct SliceParams {
  int rank;
  int sext[kPermMax];
  int64_t tstride[kPermMax];
  int64_t tbase;
  FastDiv div[kPermMax];  // slice_runs_kernel: division by sext
};

// Beyond 2^31 slice elements: an element at a time, 64-bit divisions.
__global__ void __launch_bounds__(kThreads) slice_insert_kernel(SliceParams p, int insert,
                                                                double* tens, double* slice,
                                                                int64_t n) {
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    int64_t rem = i, o = p.tbase;
    for (int q = 0; q < p.rank; ++q) {
      const int64_t x = rem % p.sext[q];
      rem /= p.sext[q];
      o += x * p.tstride[q];
    }
    if (insert) tens[o] = slice[i];
    else slice[i] = tens[o];
  }
}

// Fewer than 2^31 slice elements, as T (pairs where every run starts on 16
// bytes and has an even length, else single elements): kSliceLoads a thread, all
// loaded before the first is stored, offsets by multiplications
// (FastDiv).  HBM bounds it; an element's 64-bit
// divisions did: a 72^4 slice of a 96^4
// block 190 -> 66 us, its insertion 190 -> 60.
constexpr int kSliceLoads = 4;
template <int INSERT, class T>
__global__ void __launch_bounds__(kThreads) slice_runs_kernel(SliceParams p, T* __restrict__ tens,
                                                              T* __restrict__ slice, unsigned n) {
  const unsigned first = blockIdx.x * (kThreads * kSliceLoads) + threadIdx.x;
  int64_t at[kSliceLoads];
  T v[kSliceLoads];
#pragma unroll
  for (int u = 0; u < kSliceLoads; ++u) {
    const unsigned i = first + u * kThreads;
    unsigned rem = i;
    int64_t o = p.tbase;
    for (int q = 0; q < p.rank - 1; ++q) {
      const unsigned d = fast_quot(rem, p.div[q]);
      o += int64_t(rem - d * unsigned(p.sext[q])) * p.tstride[q];
      rem = d;
    }
    at[u] = o + int64_t(rem) * p.tstride[p.rank - 1];
    if (i < n) v[u] = INSERT ? slice[i] : tens[at[u]];
  }
#pragma unroll
  for (int u = 0; u < kSliceLoads; ++u) {
    const unsigned i = first + u * kThreads;
    if (i < n) (INSERT ? tens[at[u]] : slice[i]) = v[u];
  }
}

// ---------------------------------------------------------------- denominator
struct DenParams {
  int rank0, rank1, ld1;
  int ext[6];  // extents in storage order
  int off[6];  // first orbital of each storage dimension's segment
  int pos[6];  // storage dimension holding denominator position q
  int poff[6];  // off[pos[q]]: first orbital of the segment at position q
};

// x[k] for a run-time k without indexing a register array (which would put
// it in local memory)
__device__ __forceinline__ int pick6(const int (&x)[6], int k) {
  return k == 0 ? x[0] : k == 1 ? x[1] : k == 2 ? x[2] : k == 3 ? x[3] : k == 4 ? x[4] : x[5];
}

__device__ __forceinline__ double eps_at(const DenParams& p, const double* e, int orb) {
  return p.rank1 == 2 ? e[int64_t(orb) + int64_t(orb) * p.ld1] : e[orb];
}

// Denominator of the element with storage coordinates x, in the reference's
// order of additions (energy_denominator_rhf.F do_rhf_den2/4/6): positions
// 0, 2, 4 are virtual (subtracted), 1, 3, 5 occupied (added).
// div_rn (a / b rounded to the nearest double: integer arithmetic for normal
// operands and results, the FP64 divide otherwise) and nonzero come from
// exact_fp.h.

__device__ __forceinline__ double den_eps(const DenParams& p, const double* e, const int (&x)[6]) {
  const double ea = eps_at(p, e, pick6(x, p.pos[0]) + p.poff[0]);
  const double eb = eps_at(p, e, pick6(x, p.pos[1]) + p.poff[1]);
  if (p.rank0 == 2) return __dsub_rn(eb, ea);  // epsb - epsa
  const double ec = eps_at(p, e, pick6(x, p.pos[2]) + p.poff[2]);
  const double ed = eps_at(p, e, pick6(x, p.pos[3]) + p.poff[3]);
  if (p.rank0 == 4) return __dsub_rn(__dsub_rn(__dadd_rn(eb, ed), ea), ec);  // epsb + epsd - epsa - epsc
  const double e5 = eps_at(p, e, pick6(x, p.pos[4]) + p.poff[4]);
  const double e6 = eps_at(p, e, pick6(x, p.pos[5]) + p.poff[5]);
  return __dsub_rn(__dsub_rn(__dsub_rn(__dadd_rn(__dadd_rn(eb, ed), e6), ea), ec), e5);
}

__device__ __forceinline__ void den_coords(const DenParams& p, int64_t i, int (&x)[6]) {
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    if (q < p.rank0) {
      x[q] = int(i % p.ext[q]);
      i /= p.ext[q];
    } else {
      x[q] = 0;
    }
  }
}

// Four consecutive elements per thread: the coordinates are decoded once
// (64-bit divisions are dear) and stepped along dimension 0 with carries.
constexpr int kDenRun = 4;

// The denominators of the run of elements from x on, the first `live` of them
// (1 for the rest); x moves to the element behind the last live one.
__device__ __forceinline__ void den_run(const DenParams& p, const double* e, int (&x)[6], int live,
                                        double (&d)[kDenRun]) {
#pragma unroll
  for (int u = 0; u < kDenRun; ++u) {
    d[u] = 1.0;
    if (u >= live) continue;
    d[u] = den_eps(p, e, x);
#pragma unroll
    for (int q = 0; q < 6; ++q) {  // next element: x[0] + 1 with carries
      if (q >= p.rank0) break;
      if (++x[q] < p.ext[q]) break;
      x[q] = 0;
    }
  }
}

__global__ void __launch_bounds__(kThreads) denominator_kernel(DenParams p, double* data,
                                                               const double* __restrict__ e,
                                                               int64_t n) {
  const int64_t stride = int64_t(gridDim.x) * blockDim.x * kDenRun;
  for (int64_t i0 = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) * kDenRun; i0 < n; i0 += stride) {
    int x[6];
    den_coords(p, i0, x);
    double v[kDenRun];
#pragma unroll
    for (int u = 0; u < kDenRun; ++u) v[u] = i0 + u < n ? data[i0 + u] : 0.0;
    double d[kDenRun], quot[kDenRun];
    den_run(p, e, x, int(min(int64_t(kDenRun), n - i0)), d);
    div_rn_n<kDenRun>(v, d, quot);
#pragma unroll
    for (int u = 0; u < kDenRun; ++u)
      if (i0 + u < n) data[i0 + u] = quot[u];
  }
}

// ---------------------------------------------------------------- (T) energy
// The (T)-energy pattern of rccsdpt_aaa.sialx:2163-2172 on one block of W:
// divide by the orbital-energy denominators (energy_denominator_rhf), then
// contract the divided block with the undivided one to a scalar:
//     partial += w(x) * fl(w(x) / eps(x))
// in FP64 throughout: eps summed in the reference's order (do_rhf_den2/4/6:
// the occupied positions 1, 3, 5 added left to right, then the virtual
// positions 0, 2, 4 subtracted), the quotient rounded to nearest exactly as
// the FP64 divide rounds it (div_rn), and the products accumulated in FP64
// (one fused multiply-add per element).  Each CTA writes one partial sum; the
// partials are added in a fixed order, so a GPU gives the same bits every run.

// Storage in the denominator's order (position q = storage dimension q), rank
// 4 or 6: eps = ((((e1 + e3) + e5) - e0) - e2) - e4, or ((e1 + e3) - e0) - e2.
// The chain's prefix is formed where its terms are fixed: a thread owns one
// (x0, x1) position of the block and a work unit fixes the occupied
// coordinates x3 (and x5), so (e1 + e3) (+ e5) - e0 is formed once per unit,
// - e2 once per x2, and (rank 6) - e4 per element: one FP64 subtraction per
// element instead of five, the same roundings in the same order.  The
// division runs in integer arithmetic (div_rn, the same bits as the FP64
// divide).  (An integer form of the subtraction, exact as well, ran slower
// than the FP64 one.)  Units (x3 [x5], a range of x2) are spread over
// gridDim.y CTAs in a fixed order.
constexpr int kEnLoads = 4;  // loads in flight per thread, and divisions interleaved
constexpr int kEnThreads = 384;  // two CTAs per SM at 80 registers: four divisions in flight per thread
// DIVIDE: the denominator drop-in on the same walk, in place: each element
// becomes fl(w / eps) (zeros included: 0 / eps keeps the IEEE sign), nothing
// is summed.
template <bool DIVIDE>
__global__ void __launch_bounds__(kEnThreads, 2) energy_chain_kernel(DenParams p, double* w,
                                                            const double* __restrict__ e, int x2_per_unit,
                                                            int64_t nunits, double efact, double* esum,
                                                            double* partial, unsigned* counter) {
  extern __shared__ double en[];  // e2 energies [ext2], then e4 energies [ext4]
  const int n0 = p.ext[0], n1 = p.ext[1], n2 = p.ext[2], n3 = p.ext[3];
  const bool r6 = p.rank0 == 6;
  const int n4 = r6 ? p.ext[4] : 1;
  for (int t = threadIdx.x; t < n2; t += blockDim.x) en[t] = eps_at(p, e, t + p.off[2]);
  if (r6)
    for (int t = threadIdx.x; t < n4; t += blockDim.x) en[n2 + t] = eps_at(p, e, t + p.off[4]);
  __syncthreads();
  const int64_t n01 = int64_t(n0) * n1;
  const int64_t pp = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int x2_chunks = (n2 + x2_per_unit - 1) / x2_per_unit;
  // the energy form only reads w (read-only cache); the divide form writes it
  auto load = [](const double* q) -> double {
    if constexpr (DIVIDE) return *q;
    else return __ldg(q);
  };
  double acc = 0.0;
  if (pp < n01) {
    const int x0 = int(pp % n0), x1 = int(pp / n0);
    const double e1v = eps_at(p, e, x1 + p.off[1]), e0v = eps_at(p, e, x0 + p.off[0]);
    for (int64_t u = blockIdx.y; u < nunits; u += gridDim.y) {
      const int chunk = int(u % x2_chunks);
      const int64_t occ = u / x2_chunks;  // x3 + n3 * x5
      const int x3 = int(occ % n3), x5 = int(occ / n3);
      double t = __dadd_rn(e1v, eps_at(p, e, x3 + p.off[3]));
      if (r6) t = __dadd_rn(t, eps_at(p, e, x5 + p.off[5]));
      t = __dsub_rn(t, e0v);
      const int x2b = chunk * x2_per_unit, x2e = min(n2, x2b + x2_per_unit);
      // one run of elements at stride st whose denominators are tt - es[k]
      auto run = [&](double* base, int64_t st, double tt, const double* es, int n) {
        int k0 = 0;
        for (; k0 + kEnLoads <= n; k0 += kEnLoads) {
          double v[kEnLoads], d[kEnLoads], q[kEnLoads];
#pragma unroll
          for (int k = 0; k < kEnLoads; ++k) v[k] = load(base + st * (k0 + k));
#pragma unroll
          for (int k = 0; k < kEnLoads; ++k) d[k] = __dsub_rn(tt, es[k0 + k]);
          if constexpr (DIVIDE) {
            div_rn_n<kEnLoads>(v, d, q);
#pragma unroll
            for (int k = 0; k < kEnLoads; ++k) base[st * (k0 + k)] = q[k];
          } else {
            bool ok[kEnLoads];
#pragma unroll
            for (int k = 0; k < kEnLoads; ++k) ok[k] = div_rn_int(v[k], d[k], &q[k]);
#pragma unroll
            for (int k = 0; k < kEnLoads; ++k)
              if (ok[k]) acc = fma(v[k], q[k], acc);
              else if (nonzero(v[k])) acc = fma(v[k], div_rn_slow(v[k], d[k]), acc);
          }
        }
        for (; k0 < n; ++k0) {
          const double v = load(base + st * k0);
          if constexpr (DIVIDE) base[st * k0] = div_rn(v, __dsub_rn(tt, es[k0]));
          else if (nonzero(v)) acc = fma(v, div_rn(v, __dsub_rn(tt, es[k0])), acc);
        }
      };
      if (!r6) {
        run(w + pp + n01 * (x2b + int64_t(n2) * x3), n01, t, en + x2b, x2e - x2b);
      } else {
        const int64_t s4 = n01 * int64_t(n2) * n3;  // stride of x4
        for (int x2 = x2b; x2 < x2e; ++x2)
          run(w + pp + n01 * (x2 + int64_t(n2) * x3) + s4 * int64_t(n4) * x5, s4, __dsub_rn(t, en[x2]), en + n2, n4);
      }
    }
  }
  if constexpr (!DIVIDE) {
    double total;
    if (grid_sum(acc, partial, counter, &total)) *esum = __dadd_rn(*esum, __dmul_rn(total, efact));
  }
}

// Any other storage order or rank: the whole chain per element (den_eps, the
// same additions as energy_denominator_rhf), coordinates stepped as in the
// denominator kernel; a fixed grid, one partial per CTA.
__global__ void __launch_bounds__(kThreads) energy_generic_kernel(DenParams p, const double* __restrict__ w,
                                                                  const double* __restrict__ e, int64_t n,
                                                                  double efact, double* esum, double* partial,
                                                                  unsigned* counter) {
  const int64_t stride = int64_t(gridDim.x) * blockDim.x * kDenRun;
  double acc = 0.0;
  for (int64_t i0 = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) * kDenRun; i0 < n; i0 += stride) {
    int x[6];
    den_coords(p, i0, x);
    double v[kDenRun];
#pragma unroll
    for (int u = 0; u < kDenRun; ++u) v[u] = i0 + u < n ? __ldg(w + i0 + u) : 0.0;
    double d[kDenRun], quot[kDenRun];
    bool ok[kDenRun];
    den_run(p, e, x, int(min(int64_t(kDenRun), n - i0)), d);
#pragma unroll
    for (int u = 0; u < kDenRun; ++u) ok[u] = div_rn_int(v[u], d[u], &quot[u]);
#pragma unroll
    for (int u = 0; u < kDenRun; ++u)
      if (ok[u]) acc = fma(v[u], quot[u], acc);
      else if (nonzero(v[u])) acc = fma(v[u], div_rn_slow(v[u], d[u]), acc);
  }
  double total;
  if (grid_sum(acc, partial, counter, &total)) *esum = __dadd_rn(*esum, __dmul_rn(total, efact));
}

// ---------------------------------------------------------------- amplitude update
// updatet2 of rlccd_rhf.sialx:557-600 for one block (a,i,b,j), both pardo
// passes fused into one read of the four input blocks:
//   t  = T2new[b,j,a,i] + T2new[a,i,b,j]        (the partner block in its own storage)
//   t1 = T2old[b,j,a,i] + T2old[a,i,b,j]
//   E(a,i,b,j)      = -0.5 * (t1 - t / eps)      (DIIS error vector)
//   T2old'(a,i,b,j) = (0.5 * t) / eps            (next amplitudes, a separate buffer:
//                                                 the partner block still reads T2old)
//   partial[block] = sum of E^2                  (its residual norm, deterministic)
// eps = ((e_i + e_j) - e_a) - e_b, energy_denominator_rhf's rank-4 order.
// (0.5 t)/eps is formed as 0.5 (t/eps): both are t/(2 eps) correctly rounded
// while the quotient and 0.5 t are normal numbers; below and beyond that (t/eps
// may overflow where its half does not) the division is redone.
//
// A work unit is one (a,b) tile at fixed (i,j).  The plane is cut evenly into
// tiles of at most 48 x 24 (a 33 x 37 plane is two of 33 x 19, 96 x 96 eight of
// 48 x 24): threads walk the tile's own elements, so the lanes are as full as
// the plane allows (32 x 32 tiles left 73 % of the lanes of a 33 x 33 plane
// idle).  The partner tiles are read along b and transposed through shared
// memory so that all loads coalesce.  Four elements per thread at a time, their
// loads (the first own ones before the partner's) and divisions in flight
// together.  One resident wave of CTAs, each over several units;
// the last one to finish adds the partial norms in a fixed order.
// o=40/v=300 (400 blocks of about 33 x 20 x 33 x 20, 48 B an element):
// 20 us a block before.
constexpr int kUpdA = 48, kUpdB = 24, kUpdGroup = 4, kUpdThreads = 128;
constexpr uint32_t kHalvable = 2u << 21;  // the high word, less its sign, of 2^-1021: the least number with a normal half
struct UpdParams {
  int ea, ei, eb, ej;   // extents
  int oa, oi, ob, oj;   // first orbitals
  int rank1, ld1;
  int ta, tb;           // tile extents
  int tiles_a, tiles_b;
  int64_t units;
  uint32_t mul_a, mul_b;  // ceil(2^20 / ta), ceil(2^20 / tb): e / t = (e mul) >> 20 for e < 48 * 24 + 512
};

__device__ __forceinline__ double eps_at_upd(const UpdParams& p, const double* e, int orb) {
  return __ldcg(p.rank1 == 2 ? e + int64_t(orb) + int64_t(orb) * p.ld1 : e + orb);
}

// x / 2 without the FP64 pipe where that is an exponent decrement (normal x
// whose half is normal); the FP64 multiply otherwise (the same bits either way)
__device__ __forceinline__ double half_of(double x) {
  const unsigned long long b = bits_of(x);
  const unsigned f = unsigned(b >> 52) & 0x7FFu;
  return f >= 2u && f != 0x7FFu ? double_of(b - (1ull << 52)) : __dmul_rn(x, 0.5);
}

__global__ void __launch_bounds__(kUpdThreads, 6) update_t2_kernel(UpdParams p, const double* __restrict__ xn,
                                                           const double* __restrict__ xnp,
                                                           const double* __restrict__ xo,
                                                           const double* __restrict__ xop, double* __restrict__ err,
                                                           double* __restrict__ next, const double* __restrict__ e,
                                                           double* norm2, double* partial, unsigned* counter) {
  __shared__ double pn[kUpdA][kUpdB + 1], po[kUpdA][kUpdB + 1];  // [a][b] of the partner tiles
  __shared__ double sa[kUpdA], sb[kUpdB];  // (e_i + e_j) - e_a of the tile's a, e_b of its b
  // The next update's CTAs may take their places as this one's leave; they wait
  // here until it has completed before they read anything.  All its inputs are
  // read from L2 (__ldcg): the update before may have written them while this
  // grid was already there, so they are not read-only for its lifetime, as the
  // non-coherent loads (__ldg) require, and a line of this
  // SM's L1 may be from before that write.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  double acc = 0.0;
  for (int64_t u = blockIdx.x; u < p.units; u += gridDim.x) {
    int64_t r = u;
    const int at = int(r % p.tiles_a);
    r /= p.tiles_a;
    const int bt = int(r % p.tiles_b);
    r /= p.tiles_b;
    const int i = int(r % p.ei), j = int(r / p.ei);
    const int a0 = at * p.ta, b0 = bt * p.tb;
    const int na = min(p.ta, p.ea - a0), nb = min(p.tb, p.eb - b0), n = p.ta * p.tb;
    __syncthreads();  // the previous unit's tiles are read
    if (threadIdx.x < kUpdA) {
      const int k = threadIdx.x;
      if (k < na)
        sa[k] = __dsub_rn(__dadd_rn(eps_at_upd(p, e, p.oi + i), eps_at_upd(p, e, p.oj + j)),
                          eps_at_upd(p, e, p.oa + a0 + k));
      if (k < nb) sb[k] = eps_at_upd(p, e, p.ob + b0 + k);
    }
    const int64_t qb = a0 + int64_t(p.ea) * (i + int64_t(p.ei) * (b0 + int64_t(p.eb) * j));
    const int64_t qsb = int64_t(p.ea) * p.ei;
    double t[kUpdGroup], t1[kUpdGroup];
    auto load_own = [&](int e0) {
#pragma unroll
      for (int g = 0; g < kUpdGroup; ++g) {
        const int el = e0 + kUpdThreads * g, b = int((uint32_t(el) * p.mul_a) >> 20), a = el - b * p.ta;
        const bool live = el < n && a < na && b < nb;
        t[g] = live ? __ldcg(xn + qb + a + qsb * b) : 1.0;
        t1[g] = live ? __ldcg(xo + qb + a + qsb * b) : 0.0;
      }
    };
    load_own(threadIdx.x);
    // partner block (b,j,a,i): element (b, j, a, i) at b + eb*(j + ej*(a + ea*i))
    const int64_t pb = b0 + int64_t(p.eb) * (j + int64_t(p.ej) * (a0 + int64_t(p.ea) * i));
    const int64_t psa = int64_t(p.eb) * p.ej;
#pragma unroll 1
    for (int e0 = threadIdx.x; e0 < n; e0 += kUpdThreads * kUpdGroup) {
      double vn[kUpdGroup], vo[kUpdGroup];
#pragma unroll
      for (int g = 0; g < kUpdGroup; ++g) {
        const int el = e0 + kUpdThreads * g, a = int((uint32_t(el) * p.mul_b) >> 20), b = el - a * p.tb;
        const bool live = el < n && a < na && b < nb;
        vn[g] = live ? __ldcg(xnp + pb + b + psa * a) : 0.0;
        vo[g] = live ? __ldcg(xop + pb + b + psa * a) : 0.0;
      }
#pragma unroll
      for (int g = 0; g < kUpdGroup; ++g) {
        const int el = e0 + kUpdThreads * g, a = int((uint32_t(el) * p.mul_b) >> 20), b = el - a * p.tb;
        if (el < n) pn[a][b] = vn[g], po[a][b] = vo[g];
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int e0 = threadIdx.x; e0 < n; e0 += kUpdThreads * kUpdGroup) {
      if (e0 != int(threadIdx.x)) load_own(e0);
      int64_t q[kUpdGroup];
      double eps[kUpdGroup], td[kUpdGroup];
      bool live[kUpdGroup];
#pragma unroll
      for (int g = 0; g < kUpdGroup; ++g) {
        const int el = e0 + kUpdThreads * g, b = int((uint32_t(el) * p.mul_a) >> 20), a = el - b * p.ta;
        live[g] = el < n && a < na && b < nb;
        q[g] = qb + a + qsb * b;
        eps[g] = 1.0;  // outside the tile: 1 / 1, dropped
        if (live[g]) {
          t[g] = __dadd_rn(pn[a][b], t[g]);
          t1[g] = __dadd_rn(po[a][b], t1[g]);
          eps[g] = __dsub_rn(sa[a], sb[b]);
        }
      }
      div_rn_n<kUpdGroup>(t, eps, td);
      // -0.5 (t1 - td) and 0.5 td by their exponent fields where both halves
      // are normal numbers (a multiplication or a comparison would take the
      // FP64 pipe, 16 clocks a warp)
      double ev[kUpdGroup], nx[kUpdGroup];
      bool all = true;
      uint32_t least = ~0u;  // of |t|'s exponent and upper fraction: below 2^-1021, t loses a bit when it is halved
#pragma unroll
      for (int g = 0; g < kUpdGroup; ++g) {
        const unsigned long long x = bits_of(__dsub_rn(t1[g], td[g])), y = bits_of(td[g]);
        least = min(least, uint32_t(bits_of(t[g]) >> 32) << 1);
        ev[g] = double_of((x - (1ull << 52)) ^ (1ull << 63));
        nx[g] = double_of(y - (1ull << 52));
        t1[g] = double_of(x);
        all = all && (uint32_t(x >> 52) & 0x7FFu) - 2u < 2045u && (uint32_t(y >> 52) & 0x7FFu) - 2u < 2045u;
      }
      if (!all || least < kHalvable) {
#pragma unroll 1
        for (int g = 0; g < kUpdGroup; ++g) {
          double x = 0.0, y = 0.0, tg = 0.0, eg = 0.0;
#pragma unroll
          for (int k = 0; k < kUpdGroup; ++k)
            if (k == g) x = t1[k], y = td[k], tg = t[k], eg = eps[k];
          const unsigned f = uint32_t(bits_of(y) >> 52) & 0x7FFu;
          x = double_of(bits_of(half_of(x)) ^ (1ull << 63));
          y = f - 2u < 2045u && (uint32_t(bits_of(tg) >> 32) << 1) >= kHalvable ? half_of(y)
                                                                                : __ddiv_rn(__dmul_rn(tg, 0.5), eg);
#pragma unroll
          for (int k = 0; k < kUpdGroup; ++k)
            if (k == g) ev[k] = x, nx[k] = y;
        }
      }
#pragma unroll
      for (int g = 0; g < kUpdGroup; ++g) {
        if (!live[g]) continue;
        if (err) err[q[g]] = ev[g];
        next[q[g]] = nx[g];
        if (norm2) acc = fma(ev[g], ev[g], acc);
      }
    }
  }
  if (!norm2) return;
  double total;
  if (grid_sum(acc, partial, counter, &total)) *norm2 = __dadd_rn(*norm2, total);
}

// ---------------------------------------------------------------- scalar cases
// tensor_block_contract_ with a rank-0 operand (tensor_dil_omp.F90:770-778):
// the zeroed destination receives tensor*scalar through tensor_block_add_,
// whose factor rule (|s-1| <= 1e-13 means 1) applies; scalar*scalar is a plain
// product.  Results land in D through the destination offsets.
__global__ void __launch_bounds__(kThreads) scalar_case_kernel(
    const double* __restrict__ t, const double* __restrict__ sc, const int64_t* __restrict__ offT,
    const int64_t* __restrict__ offD, double* D, int64_t n, int beta) {
  const double s = *sc;
  const bool unit = fabs(s - 1.0) <= 1e-13;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    const double x = t[offT[i]];
    const double v = __dadd_rn(0.0, unit ? x : __dmul_rn(x, s));
    const int64_t o = offD[i];
    D[o] = beta ? __dadd_rn(D[o], v) : v;
  }
}

__global__ void scalar_scalar_kernel(const double* l, const double* r, double* d, int beta) {
  const double v = __dmul_rn(*l, *r);
  *d = beta ? __dadd_rn(*d, v) : v;
}

// Two blocks copied side by side, each thread with four loads in flight: the
// blocks are in host memory and the link's latency, not its rate, is to cover.
__global__ void __launch_bounds__(256) copy_two_kernel(const double* __restrict__ a, double* __restrict__ da, int64_t na,
                                                       const double* __restrict__ b, double* __restrict__ db, int64_t nb) {
  constexpr int kLoads = 4;
  const int64_t threads = int64_t(gridDim.x) * blockDim.x, n = na + nb;
  for (int64_t i0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i0 < n; i0 += kLoads * threads) {
    double x[kLoads];
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int64_t i = i0 + q * threads;
      if (i < n) x[q] = i < na ? a[i] : b[i - na];
    }
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int64_t i = i0 + q * threads;
      if (i < n) (i < na ? da[i] : db[i - na]) = x[q];
    }
  }
}

}  // namespace

// ============================================================== launchers
int launch_fill(double* d, int64_t n, double v, cudaStream_t s) {
  return launch_ew<EwOp::kFill>(d, nullptr, n, v, s);
}
int launch_copy_two(const double* a, double* da, int64_t na, const double* b, double* db, int64_t nb, cudaStream_t s) {
  const int64_t want = (na + nb + 1023) / 1024, most = int64_t(ctx()->num_sms > 0 ? ctx()->num_sms : 152) * 8;
  copy_two_kernel<<<unsigned(std::max<int64_t>(1, std::min(want, most))), 256, 0, s>>>(a, da, na, b, db, nb);
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}
int launch_scale(double* d, int64_t n, double f, cudaStream_t s) {
  return launch_ew<EwOp::kScale>(d, nullptr, n, f, s);
}
int launch_scale_copy(double* d, const double* src, int64_t n, double f, cudaStream_t s) {
  if (!src) return fail(A4G_ERR_ARG, "null source block");
  return launch_ew<EwOp::kScaleCopy>(d, src, n, f, s);
}
int launch_increment(double* d, int64_t n, double delta, cudaStream_t s) {
  return launch_ew<EwOp::kIncrement>(d, nullptr, n, delta, s);
}
int launch_add_scaled(double* t0, const double* t1, int64_t n, double scale, cudaStream_t s) {
  if (!t1) return fail(A4G_ERR_ARG, "null source block");
  if (fabs(scale - 1.0) > 1e-13) return launch_ew<EwOp::kAddScaled>(t0, t1, n, scale, s);
  return launch_ew<EwOp::kAdd>(t0, t1, n, 1.0, s);
}
int launch_axpy(double* y, const double* x, int64_t n, double alpha, cudaStream_t s) {
  if (!x) return fail(A4G_ERR_ARG, "null source block");
  return launch_ew<EwOp::kAxpy>(y, x, n, alpha, s);
}

int launch_permute(int rank, const int* ext, const int* o2n_1based, const double* in, double* out,
                   cudaStream_t s) {
  if (rank < 0 || rank > kMaxRank) return fail(A4G_ERR_ARG, "rank out of range");
  if (!in || !out) return fail(A4G_ERR_ARG, "null block pointer");
  if (rank == 0) {
    A4G_CUDA(cudaMemcpyAsync(out, in, sizeof(double), cudaMemcpyDeviceToDevice, s));
    return A4G_OK;
  }
  int o2n[kPermMax];
  bool seen[kPermMax] = {false};
  int64_t total = 1;
  for (int i = 0; i < rank; ++i) {
    o2n[i] = o2n_1based[i] - 1;
    if (o2n[i] < 0 || o2n[i] >= rank || seen[o2n[i]]) return fail(A4G_ERR_ARG, "invalid permutation");
    seen[o2n[i]] = true;
    if (ext[i] <= 0) return fail(A4G_ERR_ARG, "non-positive extent");
    total *= ext[i];
  }
  PermParams p;
  make_perm(rank, ext, o2n, &p);
  if (p.rank <= 1) {
    A4G_CUDA(cudaMemcpyAsync(out, in, total * sizeof(double), cudaMemcpyDeviceToDevice, s));
    return A4G_OK;
  }
  return launch_perm_op<0>(p, in, out, nullptr, total, s);
}

int launch_add_sub_permuted(int subtract, int rank, const int* r_ext, const int* o2n_1based,
                            double* d, const double* l, const double* r, cudaStream_t s) {
  if (rank < 0 || rank > kMaxRank) return fail(A4G_ERR_ARG, "rank out of range");
  if (!d || !l || !r) return fail(A4G_ERR_ARG, "null block pointer");
  int64_t total = 1;
  int o2n[kPermMax];
  for (int i = 0; i < rank; ++i) {
    total *= r_ext[i];
    o2n[i] = o2n_1based[i] - 1;
  }
  if (total == 0) return A4G_OK;
  PermParams p{};
  if (rank == 0) {
    p.rank = 1;
    p.ext[0] = 1;
    p.sin[0] = p.sout[0] = 1;
  } else {
    make_perm(rank, r_ext, o2n, &p);
  }
  if (p.rank == 0) {  // every extent is 1
    p.rank = 1;
    p.ext[0] = 1;
    p.sin[0] = p.sout[0] = 1;
  }
  return subtract ? launch_perm_op<2>(p, r, d, l, total, s) : launch_perm_op<1>(p, r, d, l, total, s);
}

int launch_dot(const double* a, const double* b, const int64_t* offA, const int64_t* offB, int64_t n, double* d_out,
               const ReductionSlot& slot, int beta, cudaStream_t s) {
  const int g = std::min<int>(kDotBlocks, grid_for(n, 8));
  dot_kernel<<<g, kThreads, 0, s>>>(a, b, offA, offB, n, d_out, beta, slot.partial, slot.counter);
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

int launch_norm2(const double* a, int64_t n, double* d_out, const ReductionSlot& slot, cudaStream_t s) {
  // 6 CTAs per SM: one resident wave
  const int sms = ctx()->num_sms > 0 ? ctx()->num_sms : 152;
  const int g = std::min<int>({kDotBlocks, 6 * sms, grid_for(n, 8)});
  norm2_kernel<<<g, kThreads, 0, s>>>(a, n, aligned16(a) ? 1 : 0, d_out, slot.partial, slot.counter);
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

int launch_slice_insert(int insert, int rank, double* tens, const int* tens_ext, double* slice,
                        const int* slice_ext, const int* ext_beg, cudaStream_t s) {
  if (rank < 0 || rank > kMaxRank) return fail(A4G_ERR_ARG, "rank out of range");
  if (!tens || !slice) return fail(A4G_ERR_ARG, "null block pointer");
  SliceParams p{};
  p.rank = rank;
  int64_t n = 1, st = 1;
  p.tbase = 0;
  for (int q = 0; q < rank; ++q) {
    if (ext_beg[q] < 0 || slice_ext[q] <= 0 || ext_beg[q] + slice_ext[q] > tens_ext[q])
      return fail(A4G_ERR_ARG, "slice outside the block");
    p.sext[q] = slice_ext[q];
    p.tstride[q] = st;
    p.tbase += int64_t(ext_beg[q]) * st;
    st *= tens_ext[q];
    n *= slice_ext[q];
  }
  if (n > 0x7fffffff - kThreads * kSliceLoads) {
    slice_insert_kernel<<<grid_for(n), kThreads, 0, s>>>(p, insert, tens, slice, n);
    A4G_CUDA(cudaGetLastError());
    return A4G_OK;
  }
  // dims that are whole in the slice join their outer neighbour; unit dims go
  SliceParams m{};
  m.tbase = p.tbase;
  bool whole = false;  // the last kept dim covers its extent of the block
  for (int q = 0; q < rank; ++q) {
    if (whole) m.sext[m.rank - 1] *= p.sext[q];
    else if (p.sext[q] != 1 || m.rank == 0) m.sext[m.rank] = p.sext[q], m.tstride[m.rank++] = p.tstride[q];
    else continue;
    whole = p.sext[q] == tens_ext[q];
  }
  if (m.rank == 0) m.rank = 1, m.sext[0] = 1, m.tstride[0] = 1;
  bool pairs = aligned16(tens) && aligned16(slice) && m.tstride[0] == 1 && (m.sext[0] & 1) == 0 && (m.tbase & 1) == 0;
  for (int q = 1; q < m.rank; ++q) pairs = pairs && (m.tstride[q] & 1) == 0;
  if (pairs) {
    n /= 2, m.sext[0] /= 2, m.tbase /= 2;
    for (int q = 1; q < m.rank; ++q) m.tstride[q] /= 2;
  }
  for (int q = 0; q < m.rank; ++q) m.div[q] = fast_div(unsigned(m.sext[q]));
  const unsigned grid = unsigned((n + kThreads * kSliceLoads - 1) / (kThreads * kSliceLoads));
  if (pairs && insert) slice_runs_kernel<1><<<grid, kThreads, 0, s>>>(m, reinterpret_cast<double2*>(tens), reinterpret_cast<double2*>(slice), unsigned(n));
  else if (pairs) slice_runs_kernel<0><<<grid, kThreads, 0, s>>>(m, reinterpret_cast<double2*>(tens), reinterpret_cast<double2*>(slice), unsigned(n));
  else if (insert) slice_runs_kernel<1><<<grid, kThreads, 0, s>>>(m, tens, slice, unsigned(n));
  else slice_runs_kernel<0><<<grid, kThreads, 0, s>>>(m, tens, slice, unsigned(n));
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

static DenParams den_params(int rank0, const int* off, const int* ext0, const int* pos, int rank1, int ld1,
                            int64_t* n) {
  DenParams p{};
  p.rank0 = rank0;
  p.rank1 = rank1;
  p.ld1 = ld1;
  *n = 1;
  for (int q = 0; q < rank0; ++q) {
    p.ext[q] = ext0[q];
    p.off[q] = off[q];
    p.pos[q] = pos ? pos[q] : q;
    *n *= ext0[q];
  }
  for (int q = 0; q < rank0; ++q) p.poff[q] = p.off[p.pos[q]];
  return p;
}

// Grid of the chain walk (rank 4 or 6 in the denominator's order): a thread
// per (x0, x1) position (the positions split evenly over gx CTAs of at most
// kEnThreads threads); units (x3 [x5], an x2 range) spread over one resident
// wave of CTAs (2 per SM), at most max_ctas in all.  The x2 ranges are cut so
// that a CTA gets 16 units or more where the block has them (the last round is
// then nearly full), at rank 4 in multiples of the elements a thread divides
// together (a 48 x 42 x 53 x 42 block in ranges of 6 left 2 of 6 elements to
// the one-by-one tail).
struct ChainGrid {
  int64_t gx = 0, gy = 0, nunits = 0;
  int threads = 0, per = 0;
  size_t smem = 0;
};
ChainGrid chain_grid(int rank0, const int* ext0, int64_t max_ctas) {
  ChainGrid g;
  const int sms = ctx()->num_sms > 0 ? ctx()->num_sms : 152;
  const int64_t n01 = int64_t(ext0[0]) * ext0[1];
  g.gx = (n01 + kEnThreads - 1) / kEnThreads;
  g.threads = int(((n01 + g.gx - 1) / g.gx + 31) / 32 * 32);
  const int64_t nocc = rank0 == 6 ? int64_t(ext0[3]) * ext0[5] : ext0[3];
  const int64_t wave = std::max<int64_t>(1, std::min<int64_t>(2LL * sms / g.gx, max_ctas / g.gx));
  const int64_t chunks = std::max<int64_t>(1, std::min<int64_t>(ext0[2], (16 * wave + nocc - 1) / nocc));
  g.per = int((ext0[2] + chunks - 1) / chunks);
  if (rank0 == 4) g.per = (g.per + kEnLoads - 1) / kEnLoads * kEnLoads;
  g.nunits = nocc * ((ext0[2] + g.per - 1) / g.per);
  g.gy = std::min(g.nunits, wave);
  g.smem = size_t(ext0[2] + (rank0 == 6 ? ext0[4] : 0)) * sizeof(double);
  return g;
}

int launch_denominator(int rank0, const int* off, const int* ext0, double* data, int rank1,
                       int ld1, const double* e_or_fock, cudaStream_t s) {
  int64_t n = 0;
  const DenParams p = den_params(rank0, off, ext0, nullptr, rank1, ld1, &n);
  if (n == 0) return A4G_OK;
  if (rank0 == 4 || rank0 == 6) {
    // the chain's prefix formed once per unit: one FP64 subtraction per element
    const ChainGrid g = chain_grid(rank0, ext0, 0x7fffffffLL);
    if (g.smem <= 48 * 1024 && g.gx <= 0x7fffffffLL && g.gy <= 65535) {
      energy_chain_kernel<true><<<dim3(unsigned(g.gx), unsigned(g.gy)), g.threads, g.smem, s>>>(
          p, data, e_or_fock, g.per, g.nunits, 0.0, nullptr, nullptr, nullptr);
      A4G_CUDA(cudaGetLastError());
      return A4G_OK;
    }
  }
  denominator_kernel<<<grid_for((n + kDenRun - 1) / kDenRun), kThreads, 0, s>>>(p, data, e_or_fock, n);
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

int launch_update_t2(const int* off, const int* ext, const double* t2new, const double* t2new_pair,
                     const double* t2old, const double* t2old_pair, double* err, double* next, int rank1, int ld1,
                     const double* e_or_fock, double* norm2, const ReductionSlot& slot, cudaStream_t s) {
  UpdParams p{};
  p.ea = ext[0], p.ei = ext[1], p.eb = ext[2], p.ej = ext[3];
  p.oa = off[0], p.oi = off[1], p.ob = off[2], p.oj = off[3];
  p.rank1 = rank1, p.ld1 = ld1;
  if (int64_t(p.ei) * p.ej > 65535) return fail(A4G_ERR_RANGE, "amplitude update: block too large");
  // the cut of the plane with the fewest passes over a tile (kUpdGroup x
  // kUpdThreads elements a pass), a quarter of a pass for each tile's ends;
  // tiles of 8 and more a side where the plane has them
  int64_t best = 0;
  for (int na = (p.ea + kUpdA - 1) / kUpdA, a_end = std::max(na, std::min(na + 3, p.ea / 8)); na <= a_end; ++na)
    for (int nb = (p.eb + kUpdB - 1) / kUpdB, b_end = std::max(nb, std::min(nb + 3, p.eb / 8)); nb <= b_end; ++nb) {
      const int ta = (p.ea + na - 1) / na, tb = (p.eb + nb - 1) / nb;
      const int64_t passes = (ta * tb + kUpdGroup * kUpdThreads - 1) / (kUpdGroup * kUpdThreads);
      const int64_t cost = int64_t(na) * nb * (4 * passes + 1);
      if (!best || cost < best) best = cost, p.tiles_a = na, p.tiles_b = nb, p.ta = ta, p.tb = tb;
    }
  p.mul_a = ((1u << 20) + p.ta - 1) / p.ta, p.mul_b = ((1u << 20) + p.tb - 1) / p.tb;
  p.units = int64_t(p.tiles_a) * p.tiles_b * p.ei * p.ej;
  if (p.units == 0) return A4G_OK;
  // one resident wave (6 CTAs of 128 threads per SM): its CTAs share the units evenly
  const int sms = ctx()->num_sms > 0 ? ctx()->num_sms : 152;
  const int64_t wave = std::min<int64_t>(kDotBlocks, 6 * int64_t(sms));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(std::min(p.units, wave))), cfg.blockDim = dim3(kUpdThreads), cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at, cfg.numAttrs = 1;
  A4G_CUDA(cudaLaunchKernelEx(&cfg, update_t2_kernel, p, t2new, t2new_pair, t2old, t2old_pair, err, next, e_or_fock, norm2,
                              slot.partial, slot.counter));
  return A4G_OK;
}

int launch_energy_contract(int rank0, const int* off, const int* ext0, const int* pos, const double* w,
                           int rank1, int ld1, const double* e_or_fock, double efact, double* esum,
                           const ReductionSlot& slot, cudaStream_t s) {
  int64_t n = 0;
  const DenParams p = den_params(rank0, off, ext0, pos, rank1, ld1, &n);
  if (n == 0) return A4G_OK;
  bool identity = true;
  for (int q = 0; q < rank0; ++q) identity &= p.pos[q] == q;
  const int sms = ctx()->num_sms > 0 ? ctx()->num_sms : 152;
  const int64_t n01 = rank0 >= 2 ? int64_t(ext0[0]) * ext0[1] : n;
  if (identity && (rank0 == 4 || rank0 == 6) && n01 <= kEnThreads * int64_t(kDotBlocks)) {
    // at most kDotBlocks partials (one per CTA)
    const ChainGrid g = chain_grid(rank0, ext0, kDotBlocks);
    if (g.smem > 48 * 1024) return fail(A4G_ERR_RANGE, "energy contraction: segments too large");
    energy_chain_kernel<false><<<dim3(unsigned(g.gx), unsigned(g.gy)), g.threads, g.smem, s>>>(
        p, const_cast<double*>(w), e_or_fock, g.per, g.nunits, efact, esum, slot.partial, slot.counter);
  } else {
    const int g = int(std::min<int64_t>({int64_t(kDotBlocks), 8LL * sms,
                                         std::max<int64_t>(1, (n + kThreads * kDenRun - 1) / (kThreads * kDenRun))}));
    energy_generic_kernel<<<g, kThreads, 0, s>>>(p, w, e_or_fock, n, efact, esum, slot.partial, slot.counter);
  }
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

int launch_scalar_cases(const DevPlan* p, const double* L, const double* R, double* D, int beta,
                        const ReductionSlot& slot, cudaStream_t s) {
  const GemmPlan& h = p->host;
  switch (h.kind) {
    case ContractKind::kFull:
      return launch_dot(L, R, p->offLk, p->offRk, h.K, D, slot, beta, s);
    case ContractKind::kRightScalar:
      scalar_case_kernel<<<grid_for(h.M), kThreads, 0, s>>>(L, R, p->offLm, p->offDm, D, h.M, beta);
      break;
    case ContractKind::kLeftScalar:
      scalar_case_kernel<<<grid_for(h.N), kThreads, 0, s>>>(R, L, p->offRn, p->offDn, D, h.N, beta);
      break;
    case ContractKind::kScalarScalar:
      scalar_scalar_kernel<<<1, 1, 0, s>>>(L, R, D, beta);
      break;
    default:
      return fail(A4G_ERR_ARG, "not a scalar contraction");
  }
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

}  // namespace a4g
