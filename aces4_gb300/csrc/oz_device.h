// Device helpers shared by the split-precision kernels (digits in ozaki.cu,
// residues in residue.cu): locating a split job, loading its tile, the
// fixed-point value of an element.
#pragma once

#include "grouped.h"

namespace a4g {
namespace {

constexpr int kDigitBits = 8;

// A row or column exponent of 2047 (the field of Inf and NaN) marks a panel
// row that holds a non-finite value: digits cannot carry it, so every result
// that row or column feeds is stored as NaN (in FP64 a NaN or an infinity in
// an operand makes the whole row or column of the product NaN or infinite).
constexpr int kNonFiniteExp = 2047;

// What this CTA works on.
struct JobPiece {
  OzSplitJob jb;
  OzPanel pn;
  int layout, tile;
};
__device__ __forceinline__ JobPiece job_piece(const OzJobSetRefs& sets) {
  int q = 0;
  unsigned base = 0;
  while (q + 1 < sets.n && blockIdx.x >= sets.s[q].end) base = sets.s[q++].end;
  const OzTileRef ref = sets.s[q].refs[blockIdx.x - base];
  JobPiece p;
  p.jb = sets.s[q].jobs[ref.job];
  p.pn = sets.s[q].panels[p.jb.panel];
  p.layout = sets.s[q].layout;
  p.tile = ref.tile;
  return p;
}

constexpr int kSplitT = 64;

// Loads one 64x64 (row, k) tile of a job into shared memory as raw bits: a
// thread keeps its k (operands unit-stride along k) or its row and walks the
// other, eight addresses and then eight loads in flight (one at a time, each
// load waited for its address: the o=40/v=300 ring step's exponents 0.86 ms
// instead of 0.78, its residues 1.98 instead of 1.79).
__device__ __forceinline__ void load_job_tile(const OzSplitJob& jb, int r0, int k0,
                                              unsigned long long (*tile)[kSplitT + 1]) {
  constexpr int kBatch = 8;
  const int own = threadIdx.x & 63, first = threadIdx.x >> 6;  // 256 threads
  const bool kfast = jb.kfast != 0;
  const int64_t* walk = kfast ? jb.offRow + r0 : jb.offK + k0;
  const int limit = kfast ? jb.rows - r0 : jb.K - k0;
  const bool live = own < (kfast ? jb.K - k0 : jb.rows - r0);
  const double* src = jb.src + (live ? __ldg(kfast ? jb.offK + k0 + own : jb.offRow + r0 + own) : 0);
  const unsigned long long flip = jb.negate ? (1ull << 63) : 0ull;  // -x: the sign bit (exponents unchanged)
#pragma unroll 1
  for (int p0 = 0; p0 < 16; p0 += kBatch) {
    int64_t off[kBatch];
    unsigned long long v[kBatch];
#pragma unroll
    for (int p = 0; p < kBatch; ++p) {
      const int q = first + 4 * (p0 + p);
      off[p] = live && q < limit ? __ldg(walk + q) : -1;
    }
#pragma unroll
    for (int p = 0; p < kBatch; ++p) v[p] = off[p] >= 0 ? __double_as_longlong(__ldg(src + off[p])) : 0ull;
#pragma unroll
    for (int p = 0; p < kBatch; ++p) {
      const int q = first + 4 * (p0 + p);
      (kfast ? tile[q][own] : tile[own][q]) = v[p] ^ flip;
    }
  }
}

// Signed fixed-point value of one double against its row exponent (biased
// max exponent mx, |x| < 2^E with E = mx - 1022):
//     n = round_half_away(x * 2^(8*slices - E - 1)),   |n| <= 2^(8*slices - 1).
__device__ __forceinline__ long long quantize(unsigned long long bits, int mx, int slices) {
  const int be = int((bits >> 52) & 0x7FF);
  const unsigned long long frac = bits & ((1ull << 52) - 1);
  const unsigned long long mant = be ? (frac | (1ull << 52)) : frac;
  const int ex = be ? be : 1;
  const int E = (mx ? mx : 1) - 1022;
  const int sh = ex - 1076 + kDigitBits * slices - E;  // |x| * 2^(8s-E-1) = mant * 2^sh
  unsigned long long m;
  if (sh >= 0) m = mant << sh;  // only for 7 slices: sh <= 2, mant << 2 < 2^55
  else if (-sh >= 63) m = 0ull;
  else m = (mant + (1ull << (-sh - 1))) >> (-sh);
  return (bits >> 63) ? -static_cast<long long>(m) : static_cast<long long>(m);
}

}  // namespace
}  // namespace a4g
