// Host launchers of the split-precision (Ozaki) contraction kernels.
#pragma once

#include <vector>

#include "grouped.h"

namespace a4g {

constexpr int kOzMaxUsableSlices = 7;  // 7 digits x 7 bits = 49 bits <= the 53-bit FP64 mantissa

int oz_prepare();  // one-time kernel attributes (call outside stream capture)
int oz_chunk_kb(int level);  // 64-wide k blocks per exact FP32 flush at a level
int oz_make_tensor_map(void* map128, const void* base, int64_t kpad, int64_t rows, int64_t rows_pad, int planes,
                       int box_rows);
// the all-levels form's map of a panel: boxes of 32 k x box_rows rows x every slice (64-byte swizzle)
int oz_make_levels_map(void* map128, const void* base, int64_t kpad, int64_t rows, int64_t rows_pad, int slices,
                       int box_rows);
int oz_max_pairs(int* pairs);  // CTA pairs of the 2-SM kernel that fit on the GPU at once
// CTA counts of the exponent / split kernels for one job of a given layout, and
// the list of pieces of a job set's CTAs.
int64_t oz_exp_tiles(int layout, int rows, int K);
int64_t oz_split_tiles(int layout, int rows, int K);
inline void oz_add_refs(std::vector<OzTileRef>* refs, int job, int64_t tiles) {
  for (int64_t t = 0; t < tiles; ++t) refs->push_back({job, int(t)});
}
int oz_launch_exp(const OzJobSetRefs& sets, cudaStream_t s);
int oz_launch_split(const OzJobSetRefs& sets, int slices, cudaStream_t s);
// pair = false: 1-SM kernel, 128 x tile_cols tiles; pair = true: CTA-pair
// kernel (cluster of 2, cta_group::2), 256 x tile_cols tiles, grid even.
// tile_cols: 128 (exact sums kept in TMEM) or 256 (exact sums in registers).
int oz_launch_gemm(const OzGemmArgs& args, int grid, bool pair, int tile_cols, cudaStream_t s);
// All-levels form of the direct GEMM (128 x 64 tiles, every level accumulator
// in TMEM at once; oz_make_levels_map maps): fits when slices <= 5 and every
// tile's k range is at most 5 blocks of 64.
constexpr int kOzLevelsTileCols = 64;
bool oz_levels_fit(int slices, int kb_total);
int oz_launch_levels(const OzGemmArgs& args, int grid, cudaStream_t s);
// Residue form (residue.cu): the number of products for K columns at `slices`
// slices (0: not possible), its tables, the operand side and the
// reconstruction (ws as int16, see OzGemmArgs).
int oz_residue_count(int slices, int64_t K);
void oz_residue_tables(int slices, int L, int64_t K, OzResidues* r, OzCrt* t);
int oz_residue_prepare();  // kernel attributes (oz_prepare calls it)
int oz_launch_residues(const OzJobSetRefs& sets, const OzResidues& r, cudaStream_t s);
// residue pieces of one job (the digits': oz_split_tiles)
int64_t oz_residue_tiles(int layout, int rows, int K);
int oz_launch_residue_recombine(const OzTile* tiles, int ntiles, int tile_rows, int tile_cols,
                                const OzDBlock* dblocks, const OzPanel* pa, const OzPanel* pb, const void* ws,
                                const OzCrt& t, int nsplit, int mode, cudaStream_t s);
int oz_wait_timeout_selftest(int limit_ms, int* waited_ms, cudaStream_t s);
// device runs of the one-rounding helpers (exact_fp.h) over device arrays
int oz_round_selftest(int n, const long long* v, const int* e2, const int* neg, double* out, cudaStream_t s);
int oz_div_selftest(int n, const double* a, const double* b, double* out, cudaStream_t s);
// esum (device) += efact * the sum of the energy form's n partials, in a fixed order.
int oz_launch_energy_reduce(const double* part, int n, double efact, double* esum, cudaStream_t s);
int oz_launch_recombine(const OzTile* tiles, int ntiles, int tile_rows, int tile_cols, const OzDBlock* dblocks,
                        const OzPanel* pa, const OzPanel* pb, const int* ws, int slices,
                        int nsplit, int mode, cudaStream_t s);  // mode: bit 0 accumulate, bit 1 negate

}  // namespace a4g
