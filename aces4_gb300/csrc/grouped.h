// Device-visible descriptors of a planned pardo step (batched contraction):
// the FP64 grouped kernel and the split-precision (Ozaki) pipeline.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

#include "a4g_internal.h"

namespace a4g {

// Device copy of one contraction plan's address tables (see GemmPlan).
struct PlanRef {
  const int64_t *offLm, *offLk, *offRk, *offRn, *offDm, *offDn;
  int M, N, K;
  int a_kfast, b_kfast;
};

inline PlanRef plan_ref(const DevPlan& p) {
  PlanRef r;
  r.offLm = p.offLm, r.offLk = p.offLk, r.offRk = p.offRk, r.offRn = p.offRn;
  r.offDm = p.offDm, r.offDn = p.offDn;
  r.M = int(p.host.M), r.N = int(p.host.N), r.K = int(p.host.K);
  r.a_kfast = p.host.a_kfast, r.b_kfast = p.host.b_kfast;
  return r;
}

// ------------------------------------------------------------ FP64 grouped
constexpr int kF64Step = 16;  // k of one step
// n / d rounded up, 1 <= n <= 2^31 - 1.
__host__ __device__ constexpr int ceil_div(int n, int d) { return (n - 1) / d + 1; }
// The k at which step `step` of K starts (K beyond the last one); step * 16
// may pass 2^31 where K is within 16 of it.
__host__ __device__ constexpr int f64_step_start(int step, int K) {
  return step <= (K - 1) / kF64Step ? step * kF64Step : K;
}
struct GroupedPair {
  const double* l;
  const double* r;
  int plan;
  int pad;
};
// One CTA's share of a destination tile: rows m0.. (mi 8s), columns n0.. (nu
// 8s), the k steps (of 16) from ks0 of pair pair_begin to ks1 of pair
// pair_end - 1.  A tile's shares follow each other and make a cluster.
struct GroupedF64Tile {
  double* d;
  int m0, n0, mi, nu;
  int pair_begin, pair_end, ks0, ks1;
  int dplan;  // plan giving D's tables and M, N
  int pad;
};
// mode: bit 0 accumulate, bit 1 negate
int launch_grouped_f64(const GroupedF64Tile* tiles, int ntiles, int cluster, const GroupedPair* pairs,
                       const PlanRef* plans, int mode, cudaStream_t s);

// ------------------------------------------------------------ split precision
// A panel holds the BF16 slices of every left block that feeds one group of
// destination rows, K-major: slice i, row m, column k at
//   base[(i * rows_pad + m) * kpad + k];
// the same layout with n for right-operand (B) panels.  Row exponents E (|x| <
// 2^E over the whole row of the panel) are kept per row.
struct OzPanel {
  __nv_bfloat16* base;
  int* exps;   // biased max exponent per row (atomicMax target)
  int rows;    // live rows
  int rows_pad;
  int64_t kpad;
};

// One operand block to slice into a panel (left blocks into A panels, right
// blocks into B panels).  Element (row, k) of the block is
//   src[offRow[row] + offK[k]].
struct OzSplitJob {
  const double* src;
  const int64_t* offRow;
  const int64_t* offK;
  int rows, K;
  int kfast;  // src is unit-stride along k
  int panel;
  int64_t koff;  // first k column of this block inside the panel (multiple of 16)
  int negate;    // slice -x instead of x (a term subtracted in a fused two-term step); generic layout only
  int pad;
};

// What CTA t of an exponent or split pass works on: piece `tile` of job `job`
// (one 8-byte load; a search in the jobs' prefix sums took one dependent load
// per halving, a microsecond at 256 jobs, before the first element was read).
struct OzTileRef {
  int job, tile;
};

// Memory layout of a split job's source block, detected on the host from the
// address tables: a plain column-major [rows x K] matrix (rows contiguous), a
// [K x rows] matrix (k contiguous), or anything else (gathered through the
// tables).
enum OzLayout { kOzGeneric = 0, kOzRowsMajor = 1, kOzKMajor = 2 };

// The job sets (one per operand side and layout) that one launch of a pass
// covers, one after another in the grid: a set that follows the first starts
// while that one drains, and a small step pays for one launch, not for three.
struct OzJobSetRef {
  const OzSplitJob* jobs;
  const OzTileRef* refs;
  const OzPanel* panels;
  int layout;
  unsigned end;  // first CTA after this set
};
constexpr int kOzMaxJobSets = 16;  // 3 layouts a side, the right k-major set once per pipeline part
struct OzJobSetRefs {
  int n = 0;
  int64_t total = 0;  // CTAs
  OzJobSetRef s[kOzMaxJobSets];
  void add(const OzSplitJob* jobs, const OzTileRef* refs, int64_t tiles, const OzPanel* panels, int layout) {
    if (tiles <= 0) return;
    total += tiles;
    if (n < kOzMaxJobSets) s[n] = {jobs, refs, panels, layout, unsigned(total)};
    ++n;
  }
  bool fits() const { return n <= kOzMaxJobSets && total <= 0x7fffffff; }
};

// One output tile (the GEMM form's tile_rows x tile_cols) of one destination block.
struct OzTile {
  int dblock;
  int m0, n0;
  int panel_a, panel_b;
  int trip_begin, trip_end;  // range of OzTrip (one per block pair feeding the tile)
  int kb_total;              // sum of the pairs' 64-wide k blocks
};
// k position of one stretch of block pairs (back to back in both panels)
// inside the A and B panels.
struct OzTrip {
  int64_t koff_a, koff_b;
  int nkb;
  int pad;
};
// Destination of a tile grid: one destination block, or a stack of blocks
// that share the rows (the same left blocks, the same row addressing) laid
// side by side along n.  Element (m, n) lives at colptr[n] + rowoff[m].
struct OzDBlock {
  double* d;
  int plan;  // PlanRef index of the (first) block
  int panel_a, panel_b;
  int col_fast;  // D is unit-stride along n, not along m: store by columns
  int M, N;      // rows; columns of all stacked blocks
  const int64_t* rowoff;  // [M] row offsets (the blocks' common offDm)
  double* const* colptr;  // [N] column bases (block + offDn of its column)
};

constexpr int kOzBM = 128, kOzBN = 128, kOzBK = 64, kOzK16 = 16, kOzMaxSlices = 8;
constexpr int kOzMaxPipelineParts = 8;  // GEMM launches per pardo step when the right split pipelines

// Work unit of the tensor-core kernel: one level of one tile over a range of
// its k blocks (split-K).  Units are ordered (level, split, tile) so that the
// CTAs running at the same time stream the same k window of the panels; in
// the direct form (no split-K) they are ordered (tile, level) and one CTA (or
// CTA pair) runs all levels of a tile in a row.
struct OzUnit {
  int tile, level, split;
  int kb_begin, kb_end;  // range in the tile's concatenated k-block list
  int trip_first;        // first trip overlapping kb_begin
  int kb_in_trip;        // k-block offset inside that trip
  int pad;
};

// Energy form of the direct GEMM (fused two-term step): per destination
// sub-block, what the epilogue needs to form the orbital-energy denominator of
// element (m, n) in the reference's order of additions: the chain without its
// last term, precomputed per sub-block as ptab[rk[m] * ckn + ck[n]], then the
// last term (a row or a column index) subtracted:
//     eps(m, n) = ptab[rk[m] * ckn + ck[n]] - elast[last_row ? m : n]
struct OzEnergyBlock {
  const double* ptab;
  const int* rk;        // [M]
  const int* ck;        // [N]
  const double* elast;  // [M] or [N]
  int ckn;
  int last_row;
};

// Residue form (residue.cu): what the operand side and the GEMM need of the
// moduli, and what the reconstruction needs.
constexpr int kOzMaxResidues = 15;
constexpr int kOzResidueChunkKb = 4;  // 64-wide k blocks per exact FP32 chunk (256 k, |residues| <= 255)
constexpr int kOzResidueBias = 256;     // added to a residue stored in the workspace (0 .. 512)
struct OzResidues {
  int L, slices;
  // each twice, as the packed FP32 instructions take them: -p, the FP32
  // reciprocal of p, and 2^14, 2^28, 2^42 modulo p
  float2 np[kOzMaxResidues], inv[kOzMaxResidues], c[3][kOzMaxResidues];
};
struct OzCrt {
  int L, slices;
  int words;  // 32-bit words of the reconstruction: 3 when |sum| < 2^95, 4 when |sum| < 2^127, else 5
  // each twice, as the packed FP32 instructions take them: -p, the FP32
  // nearest 1/p, (P / p)^-1 modulo p, P the product of the moduli
  float2 np[kOzMaxResidues], inv[kOzMaxResidues], cinv[kOzMaxResidues];
  int m[kOzMaxResidues][5];    // P / p modulo 2^160, signed 32-bit words
  int prod[5];                 // P modulo 2^160
  long long base[5];           // -0x4B400000 sum_i m[i][w]: the integers come with the bits of 1.5 2^23
};

struct OzGemmArgs {
  const void* maps_a;  // CUtensorMap[n_panels_a], 64-byte aligned, device memory
  const void* maps_b;
  const OzPanel* panels_a;
  const OzPanel* panels_b;
  const OzTile* tiles;
  const OzTrip* trips;
  const OzUnit* units;
  int n_units;
  int n_tiles;
  int slices;
  int nsplit;
  int chunk_kb[kOzMaxResidues];  // k blocks per exact flush at each level (or modulus)
  int* ws;                     // [tile][level][split][col 128][row 128] exact integer level sums
  int* err_flag;
  // Direct form (128-column tiles, one split): the levels of a tile are folded
  // exactly in TMEM (64-bit Horner sum over levels) and the epilogue rounds
  // once and stores D; no workspace, no recombine kernel.
  int direct;
  int mode;  // direct: bit 0 accumulate into D, bit 1 negate
  int dry;   // direct: compute everything but store nothing (timing)
  const OzDBlock* dblocks;
  // Residue form: slices = the number of moduli; "level" t of a unit is the
  // product of slice t of A with slice t of B, reduced modulo res_p[t] in the
  // epilogue and stored as int16 plus kOzResidueBias (ws: [tile][modulus][split][col][row] int16).
  int residue;
  float res_p[kOzMaxResidues], res_inv[kOzMaxResidues];
  // Energy form (direct, one SM per tile): nothing is stored; each epilogue
  // thread accumulates sum D(x) * fl(D(x) / eps(x)) over its elements in FP64
  // and writes it to epart[(blockIdx.x * 16 + epilogue warp) * 32 + lane].
  int energy;
  const OzEnergyBlock* eblocks;  // one per destination sub-block (tile.dblock)
  double* epart;
};

}  // namespace a4g
