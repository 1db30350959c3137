// Plain FP64 block contraction on the FP64 tensor path (DMMA, mma.sync f64),
// with the operand and result permutes folded into the tile loads/stores.
//
// Matrix view (planner):  D[offDm[m]+offDn[n]] (=|+=) sum_k L[offLm[m]+offLk[k]] * R[offRk[k]+offRn[n]]
// so no transposed copy of L, R or D is ever written (the reference allocates
// and fills transposed temporaries, tensor_dil_omp.F90:729-751, 782-785).
//
// The FP64 pipes bound both forms (1.046 TFLOP/s of m8n8k4 and 1.005 of FMAs
// measured with all four of an SM's quarters busy, a quarter of that from one
// warp), the gathers are small beside them.  So a tile pays for what lives in
// it and no more, and every SM gets the same share:
//   - a CTA holds at most 32 x 32 results as 8 x 8 DMMA tiles and runs only the
//     live ones; up to 4 columns beyond the last whole 8 run as FMAs, a row per
//     lane, where that is less than another DMMA column (25 columns cost 25);
//   - its four warps share every k step (16 k, 4 each) and not the tile, so
//     they stay equal whatever the tile's shape, and add up once at the end;
//   - a cluster of 1, 2, 4 or 8 CTAs divides a tile's k steps and adds its
//     partial tiles through distributed shared memory in rank order: one
//     launch, no workspace, the same bits on every run.
// Rows, columns and cluster size come from a model of the makespan (f64_form).
// Against 64 x 64 (48, 32) tiles padded to their edges, 2 x 2 warps a tile, and
// partial tiles through a workspace and a second launch: a 660 x 580 x 580 pair
// 715 -> 497 us (425 at the pipes' rate), the o=10/v=48 step 1488 -> 1120 us
// (1013), 108 x 96 x 96 pairs 43 -> 12 us.
//
// The grouped form runs a whole pardo step: one cluster owns one tile of one
// destination block and sums the products of every block pair that feeds that
// block (the contract-accumulate the interpreter lacks), then writes D once.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "a4g_internal.h"
#include "grouped.h"

namespace a4g {
namespace {

namespace cg = cooperative_groups;

constexpr int BK = kF64Step;  // a k step: 4 k for each of the four warps
constexpr int kStage = 32;  // k staged at a time
constexpr int kThreadsF64 = 128;
constexpr int kTile = 32;  // rows and columns of the largest tile

__device__ __forceinline__ void dmma_8x8x4(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// Element e = threadIdx.x + 128 i of a 32 x kStage operand tile: with the
// operand unit-stride along k (kfast) threads walk k fastest, else the rows.
__device__ __forceinline__ void tile_coord(bool kfast, int e, int& r, int& kk) {
  if (kfast) kk = e % kStage, r = e / kStage;
  else r = e & 31, kk = e >> 5;
}

// Gathers one 32 x kStage operand tile (rows x the first `left` of the k that
// offK starts at).
__device__ __forceinline__ void gather_tile(bool kfast, double (&reg)[kStage / 4], const double* __restrict__ X,
                                            const int64_t* __restrict__ offRow,  // smem, per row
                                            const int64_t* __restrict__ offK,    // global, per k
                                            int rows, int left) {
#pragma unroll
  for (int i = 0; i < kStage / 4; ++i) {
    int r, kk;
    tile_coord(kfast, int(threadIdx.x) + kThreadsF64 * i, r, kk);
    reg[i] = (r < rows && kk < left) ? __ldg(&X[offRow[r] + __ldg(&offK[kk])]) : 0.0;
  }
}

__device__ __forceinline__ void store_tile(bool kfast, double (*S)[kTile + 4], const double (&reg)[kStage / 4]) {
#pragma unroll
  for (int i = 0; i < kStage / 4; ++i) {
    int r, kk;
    tile_coord(kfast, int(threadIdx.x) + kThreadsF64 * i, r, kk);
    S[kk][r] = reg[i];
  }
}

// FMA columns that `part` live columns beyond a tile's whole 8s run as (1, 2 or
// 4), or 0 where another DMMA column costs less.
__host__ __device__ inline int f64_fma_cols(int part, int mi) {
  const int c = part == 3 ? 4 : part;
  return c <= 4 && c < 2 * mi ? c : 0;
}

struct F64Smem {
  union {
    struct {
      double As[2][kStage][kTile + 4];  // +4 doubles: conflict-free fragment reads
      double Bs[2][kStage][kTile + 4];
    };
    double part[kThreadsF64 / 32][kTile][kTile + 2];  // each warp's share of the tile, column-major
  };
  int64_t sLm[kTile], sRn[kTile];
};

// The first MI rows of 8 of a tile, one k4.  A body of its own per MI: a DMMA
// that is predicated off takes its slot in the pipe all the same.
template <int MI, int NJ>
__device__ __forceinline__ void mma_rows(double (&acc)[kTile / 8][NJ][2], const double* a, const double* b) {
  double bf[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) bf[j] = b[8 * j];
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const double af = a[8 * i];
#pragma unroll
    for (int j = 0; j < NJ; ++j) dmma_8x8x4(acc[i][j], af, bf[j]);
  }
}

// part = sum over the k steps [ks0 of pair pb, ks1 of pair pe - 1) of the
// tile's rows m0.. (mi DMMA tiles) and columns n0.. (NJ DMMA tiles, then up to
// NREM columns of FMAs, nrem of them live).  Warp w takes k = 4w..4w+3 of each
// step.  NREM is a template parameter for the same reason.
template <int NJ, int NREM>
__device__ void accumulate_tile(F64Smem& sm, const GroupedPair* __restrict__ pairs, const PlanRef* __restrict__ plans,
                                int pb, int pe, int ks0, int ks1, int m0, int n0, int mi, int nrem) {
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int g = lane >> 2, tig = lane & 3;
  double acc[kTile / 8][NJ ? NJ : 1][2];
  double rem[NREM ? NREM : 1];
#pragma unroll
  for (int i = 0; i < kTile / 8; ++i)
#pragma unroll
    for (int j = 0; j < (NJ ? NJ : 1); ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
  for (int c = 0; c < (NREM ? NREM : 1); ++c) rem[c] = 0.0;

  for (int q = pb; q < pe; ++q) {
    const GroupedPair pr = pairs[q];
    const PlanRef pl = plans[pr.plan];
    const int first = q == pb ? f64_step_start(ks0, pl.K) : 0, end = q == pe - 1 ? f64_step_start(ks1, pl.K) : pl.K;
    const int rows = min(pl.M - m0, 8 * mi), cols = min(pl.N - n0, 8 * NJ + nrem);
    const int64_t *offLk = pl.offLk + first, *offRk = pl.offRk + first;
    int left = end - first;  // k to do, from offLk and offRk on
    __syncthreads();  // previous pair done with the tables / tiles
    if (t < kTile) sm.sLm[t] = t < rows ? pl.offLm[m0 + t] : 0;
    else if (t < 2 * kTile) sm.sRn[t - kTile] = t - kTile < cols ? pl.offRn[n0 + t - kTile] : 0;
    __syncthreads();
    if (left <= 0) continue;
    double ra[kStage / 4], rb[kStage / 4];
    gather_tile(pl.a_kfast, ra, pr.l, sm.sLm, offLk, rows, left);
    gather_tile(pl.b_kfast, rb, pr.r, sm.sRn, offRk, cols, left);
    store_tile(pl.a_kfast, sm.As[0], ra);
    store_tile(pl.b_kfast, sm.Bs[0], rb);
    __syncthreads();
    for (int cur = 0; left > 0; left -= kStage, cur ^= 1) {
      const bool more = left > kStage;
      if (more) {
        offLk += kStage, offRk += kStage;
        gather_tile(pl.a_kfast, ra, pr.l, sm.sLm, offLk, rows, left - kStage);
        gather_tile(pl.b_kfast, rb, pr.r, sm.sRn, offRk, cols, left - kStage);
      }
#pragma unroll
      for (int h = 0; h < kStage / BK; ++h) {
        if (h && h * BK >= left) break;
        const int k4 = h * BK + 4 * warp;
        if constexpr (NJ > 0) {
          const double *ak = &sm.As[cur][k4 + tig][g], *bk = &sm.Bs[cur][k4 + tig][g];
          switch (mi) {
            case 1: mma_rows<1>(acc, ak, bk); break;
            case 2: mma_rows<2>(acc, ak, bk); break;
            case 3: mma_rows<3>(acc, ak, bk); break;
            default: mma_rows<4>(acc, ak, bk); break;
          }
        }
        if constexpr (NREM > 0) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const double a0 = sm.As[cur][k4 + kk][lane];
#pragma unroll
            for (int c = 0; c < NREM; ++c) rem[c] = fma(a0, sm.Bs[cur][k4 + kk][8 * NJ + c], rem[c]);
          }
        }
      }
      if (more) {
        store_tile(pl.a_kfast, sm.As[cur ^ 1], ra);
        store_tile(pl.b_kfast, sm.Bs[cur ^ 1], rb);
      }
      __syncthreads();
    }
  }
  __syncthreads();  // the staged operands are done with
  if constexpr (NJ > 0)
#pragma unroll
    for (int i = 0; i < kTile / 8; ++i)
      if (i < mi)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) sm.part[warp][8 * j + 2 * tig + h][8 * i + g] = acc[i][j][h];
  if constexpr (NREM > 0)
#pragma unroll
    for (int c = 0; c < NREM; ++c) sm.part[warp][8 * NJ + c][lane] = rem[c];
}

template <int NREM, class... A>
__device__ __forceinline__ void accumulate_cols(int nj, A&&... args) {
  if constexpr (NREM > 0) {
    switch (nj) {
      case 0: return accumulate_tile<0, NREM>(args...);
      case 1: return accumulate_tile<1, NREM>(args...);
      case 2: return accumulate_tile<2, NREM>(args...);
      default: return accumulate_tile<3, NREM>(args...);
    }
  } else {
    switch (nj) {
      case 1: return accumulate_tile<1, 0>(args...);
      case 2: return accumulate_tile<2, 0>(args...);
      case 3: return accumulate_tile<3, 0>(args...);
      default: return accumulate_tile<4, 0>(args...);
    }
  }
}

// One CTA's share of one tile (nu columns of 8, the last one perhaps partial),
// then the sum over the cluster's CTAs and their warps into D.  mode bit 0: accumulate into D (beta = 1),
// bit 1: store the negated sum.
__device__ void f64_tile(F64Smem& sm, const GroupedPair* pairs, const PlanRef* plans, int pb, int pe, int ks0, int ks1,
                         const PlanRef& dp, double* __restrict__ D, int m0, int n0, int mi, int nu, int mode) {
  const int rows = min(dp.M - m0, 8 * mi), cols = min(dp.N - n0, 8 * nu);
  // columns beyond the last whole 8: up to four as FMAs (64 clk a column of 32
  // rows and k on a quarter's pipe), else one more DMMA column (512 clk a tile
  // of 8 rows and 4 k)
  const int part = cols & 7, fma_cols = f64_fma_cols(part, mi);
  if (fma_cols == 1) accumulate_cols<1>(nu - 1, sm, pairs, plans, pb, pe, ks0, ks1, m0, n0, mi, part);
  else if (fma_cols == 2) accumulate_cols<2>(nu - 1, sm, pairs, plans, pb, pe, ks0, ks1, m0, n0, mi, part);
  else if (fma_cols == 4) accumulate_cols<4>(nu - 1, sm, pairs, plans, pb, pe, ks0, ks1, m0, n0, mi, part);
  else accumulate_cols<0>(nu, sm, pairs, plans, pb, pe, ks0, ks1, m0, n0, mi, 0);
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = int(cluster.num_blocks()), rank = int(cluster.block_rank());
  if (ranks > 1) cluster.sync();
  else __syncthreads();
  const bool col_fast = dp.N > 1 && dp.offDn[1] - dp.offDn[0] == 1;
  const int total = rows * cols, lo = total * rank / ranks, hi = total * (rank + 1) / ranks;
  for (int e = lo + int(threadIdx.x); e < hi; e += kThreadsF64) {
    const int m = col_fast ? e / cols : e % rows, n = col_fast ? e % cols : e / rows;
    double v = 0.0;
    for (int q = 0; q < ranks; ++q)
#pragma unroll
      for (int w = 0; w < kThreadsF64 / 32; ++w) {
        double* x = &sm.part[w][n][m];
        v += ranks > 1 ? *cluster.map_shared_rank(x, q) : *x;
      }
    if (mode & 2) v = -v;
    double* p = D + dp.offDm[m0 + m] + dp.offDn[n0 + n];
    *p = (mode & 1) ? *p + v : v;
  }
  if (ranks > 1) cluster.sync();  // no CTA leaves while its partial tile is read
}

// One block pair: cluster x = tile, its CTAs share the tile's k steps.
struct F64PairArgs {
  GroupedPair pair;
  PlanRef plan;
  double* d;
  int tiles_m, tiles_n, mode;
};
__global__ void __launch_bounds__(kThreadsF64, 4) contract_f64_kernel(const __grid_constant__ F64PairArgs a) {
  __shared__ __align__(16) F64Smem sm;
  const int ranks = int(cg::this_cluster().num_blocks()), rank = int(cg::this_cluster().block_rank());
  const int tile = int(blockIdx.x) / ranks, tm = tile % a.tiles_m, tn = tile / a.tiles_m;
  const int um = ceil_div(a.plan.M, 8), un = ceil_div(a.plan.N, 8), steps = ceil_div(a.plan.K, BK);
  const int u0 = int(int64_t(um) * tm / a.tiles_m), u1 = int(int64_t(um) * (tm + 1) / a.tiles_m);
  const int v0 = int(int64_t(un) * tn / a.tiles_n), v1 = int(int64_t(un) * (tn + 1) / a.tiles_n);
  f64_tile(sm, &a.pair, &a.plan, 0, 1, int(int64_t(steps) * rank / ranks), int(int64_t(steps) * (rank + 1) / ranks),
           a.plan, a.d, 8 * u0, 8 * v0, u1 - u0, v1 - v0, a.mode);
}

// A pardo step: one CTA per (destination block, tile, share of its pairs' k
// steps), a tile's shares in one cluster.
__global__ void __launch_bounds__(kThreadsF64, 4) grouped_f64_kernel(const GroupedF64Tile* __restrict__ tiles,
                                                                     const GroupedPair* __restrict__ pairs,
                                                                     const PlanRef* __restrict__ plans, int mode) {
  __shared__ __align__(16) F64Smem sm;
  const GroupedF64Tile tl = tiles[blockIdx.x];
  f64_tile(sm, pairs, plans, tl.pair_begin, tl.pair_end, tl.ks0, tl.ks1, plans[tl.dplan], tl.d, tl.m0, tl.n0, tl.mi,
           tl.nu, mode);
}

template <class... P, class... A>
int launch_clusters(void (*kernel)(P...), int64_t ctas, int cluster, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(ctas));
  cfg.blockDim = dim3(kThreadsF64);
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = unsigned(cluster), at.val.clusterDim.y = 1, at.val.clusterDim.z = 1;
  cfg.attrs = &at, cfg.numAttrs = 1;
  A4G_CUDA(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
  return A4G_OK;
}

}  // namespace

// Tile rows and columns (in 8s) and the cluster size with the least estimated
// time.  A CTA's cost on a quarter's pipe: 578 clk a DMMA, 300 for the FMAs of a
// column and 16 k, 300 to add the shares of an 8 x 8 tile, 250 a step and 3000 at
// its ends.  An SM runs up to four CTAs at once and needs them to fill the pipe;
// up to that many the fullest SM decides, beyond it half a CTA more than the mean.
// Over 12 shapes from 32^3 to 1024 x 256 x 1024, all 64 forms measured of each,
// the forms it picks take 5.6 % more than the best ones (and up to 9x less than the worst).
F64Form f64_form(const std::vector<F64Shape>& shapes, int sms) {
  F64Form best;
  double best_t = 0.0;
  int64_t hm = 1, hn = 1;
  for (const F64Shape& x : shapes) hm = std::max(hm, (x.M + 7) / 8), hn = std::max(hn, (x.N + 7) / 8);
  for (int h = 1; h <= int(std::min<int64_t>(4, hm)); ++h)
    for (int w = 1; w <= int(std::min<int64_t>(4, hn)); ++w) {
      double tiles = 0.0, cost[4] = {0.0, 0.0, 0.0, 0.0}, largest[4] = {0.0, 0.0, 0.0, 0.0};
      for (const F64Shape& x : shapes) {
        const int64_t um = (x.M + 7) / 8, un = (x.N + 7) / 8, tm = (um + h - 1) / h, tn = (un + w - 1) / w;
        const int mi = int((um + tm - 1) / tm), nu = int((un + tn - 1) / tn);  // the largest tile
        const double n = double(x.count) * double(tm * tn), rows = double(um) / double(tm), cols = double(un) / double(tn);
        const int fma_cols = f64_fma_cols(int(x.N & 7), mi);
        const double saved = fma_cols ? (578.0 * rows - 300.0 * fma_cols) / double(tn) : 0.0;
        tiles += n;
        for (int c = 0; c < 4; ++c) {
          const double steps = double((x.steps + (1 << c) - 1) >> c);  // the longest share's
          cost[c] += n * (steps * (578.0 * rows * cols - saved + 250.0) + 300.0 * rows * cols + 3000.0);
          largest[c] = std::max(largest[c], steps * (578.0 * mi * nu + 250.0) + 300.0 * mi * nu + 3000.0);
        }
      }
      for (int c = 0; c < 4; ++c) {
        const double ctas = tiles * double(1 << c), mean = ctas / sms;
        if (ctas > double(0x7fffffff)) break;
        const double per_sm = mean <= 4.0 ? std::ceil(mean) : mean + 0.5, own = cost[c] / tiles;
        const double full = per_sm <= 1.0 ? 0.4 : per_sm <= 2.0 ? 0.7 : per_sm <= 3.0 ? 0.9 : 1.0;
        const double t = per_sm * own / full + 0.5 * largest[c] + 0.01 * ((1 << c) - 1) * own + (c ? 3000.0 : 0.0);
        if (best_t == 0.0 || t < best_t) best_t = t, best.h = h, best.w = w, best.cluster = 1 << c;
      }
    }
  return best;
}

int launch_contract_f64(const DevPlan* p, const double* L, const double* R, double* D, int mode,
                        cudaStream_t s) {
  const GemmPlan& h = p->host;
  if (h.M > 0x7fffffff || h.N > 0x7fffffff || h.K > 0x7fffffff)
    return fail(A4G_ERR_RANGE, "matrix dimension exceeds 2^31");
  const F64Form& f = p->f64;
  const int64_t um = (h.M + 7) / 8, un = (h.N + 7) / 8, tm = (um + f.h - 1) / f.h, tn = (un + f.w - 1) / f.w;
  if (tm * tn * f.cluster > 0x7fffffffLL) return fail(A4G_ERR_RANGE, "contraction grid too large");
  F64PairArgs a{};
  a.pair = {L, R, 0, 0};
  a.plan = plan_ref(*p);
  a.d = D;
  a.tiles_m = int(tm), a.tiles_n = int(tn), a.mode = mode;
  return launch_clusters(contract_f64_kernel, tm * tn * f.cluster, f.cluster, s, a);
}

int launch_grouped_f64(const GroupedF64Tile* tiles, int ntiles, int cluster, const GroupedPair* pairs,
                       const PlanRef* plans, int mode, cudaStream_t s) {
  if (ntiles <= 0) return A4G_OK;
  return launch_clusters(grouped_f64_kernel, ntiles, cluster, s, tiles, pairs, plans, mode);
}

}  // namespace a4g
