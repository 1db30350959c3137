// Residue form of the split-precision contraction: the product of the two
// fixed-point operands computed exactly through residues modulo small coprime
// numbers, instead of the digit products of the levels 0..S-1.
//
// At S slices an operand element is the integer n = round(x 2^(8S - E - 1)),
// |n| <= 2^(8S-1), as in the digit form (same row scales; both round to the
// nearest integer, ties here to even up to 6 slices, there away from zero).  The
// digit form multiplies S (S + 1) / 2 pairs of 8-bit digits and drops the
// levels i + j >= S.  Here n is reduced modulo L coprime moduli p <= 511 to
// residues |r| <= 255 (exact BF16 values); one tensor-core product per modulus
// gives the contraction modulo p, and the Chinese remainder theorem gives the
// integer sum_k n_L n_R itself, rounded once to FP64: no level is dropped, so
// the error is that of rounding the operands alone.  What it needs is
// prod p > 2 |sum| >= 2 K 4^(8S-1): L = 11 products at 5 slices instead of 15,
// 13 instead of 21 at 6, 15 instead of 28 at 7 (at 4 slices 10 against 10).
//
// Method: residue-number ("Ozaki scheme II") matrix products, Ozaki, Uchino,
// Imamura, "Ozaki Scheme II: A GEMM-oriented emulation of floating-point
// matrix multiplication using an integer modular technique" (2025), with
// BF16 residues instead of INT8 ones: 9-bit moduli, because every integer up
// to 256 is a BF16 value, and FP32 accumulation over 256 k at a time:
// 256 * 255^2 + 256 < 2^24, so every partial sum is an exact FP32 integer and
// the GEMM's epilogue reduces it modulo p before the next 256 (ozaki.cu).
// Longer chunks would want smaller moduli (k of 960 for p <= 257) and with
// them 13 products instead of 11.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "a4g_internal.h"
#include "exact_fp.h"
#include "f32x2.h"
#include "oz_device.h"
#include "ozaki.h"

namespace a4g {
namespace {

// Pairwise coprime (511 = 7 73, 508 = 4 127, 507 = 3 13^2, 505 = 5 101,
// 493 = 17 29, 473 = 11 43, the others prime), the largest products first.
constexpr int kModuli[kOzMaxResidues] = {511, 509, 508, 507, 505, 503, 499, 493,
                                         491, 487, 479, 473, 467, 463, 461};

int symmetric(long long v, int p) {  // v mod p in (-p/2, p/2]
  long long r = v % p;
  if (r < 0) r += p;
  return int(2 * r > p ? r - p : r);
}

int inverse_mod(int a, int p) {
  for (int x = 1; x < p; ++x)
    if (symmetric((long long)a * x, p) == 1) return x;
  return 0;
}

// A number modulo 2^160.
struct Words160 {
  uint32_t w[5] = {1, 0, 0, 0, 0};
  void times(uint32_t f) {
    uint64_t carry = 0;
    for (uint32_t& x : w) carry += uint64_t(x) * f, x = uint32_t(carry), carry >>= 32;
  }
};
// Its words in base 2^32 with digits in [-2^31, 2^31), modulo 2^160.
void signed_words(const Words160& v, int (&w)[5]) {
  uint64_t carry = 0;
  for (int j = 0; j < 5; ++j) {
    const uint64_t t = v.w[j] + carry;
    w[j] = int(uint32_t(t));
    carry = (t >> 32) + (w[j] < 0 ? 1 : 0);
  }
}

// ------------------------------------------------------------------ operand side
// n of an element: one FP64 multiply-add against 1.5 2^52, whose low bits are
// the integer x 2^(8S - E - 1) rounded to nearest (|n| <= 2^47 up to 6
// slices); 7 slices, and rows whose scale is no double (E below -980), take the
// integer path.  The FP64 pipe runs one such operation per element in the time
// the other pipes take for the residues; the integer path's two 64-bit shifts
// and the rest cost about 25 instructions.
constexpr double kFixMagic = 6755399441055744.0;  // 1.5 2^52
struct RowScale {
  double scale;  // 2^(8S - E - 1); 0: the integer path
  int mx, slices;
};
__device__ __forceinline__ RowScale row_scale(int mx, int slices) {
  RowScale r{0.0, mx, slices};
  const int e = kDigitBits * slices - 1 - ((mx ? mx : 1) - 1022) + 1023;  // biased exponent of the scale
  if (slices <= 6 && e >= 1 && e <= 2046) r.scale = __longlong_as_double((long long)e << 52);
  return r;
}
__device__ __forceinline__ long long fixed_point(unsigned long long bits, const RowScale& r) {
  if (r.scale != 0.0)
    return __double_as_longlong(__fma_rn(__longlong_as_double((long long)bits), r.scale, kFixMagic)) -
           0x4338000000000000ll;
  return quantize(bits, r.mx, r.slices);
}

// The 14-bit pieces of n, balanced (|f| <= 2^13, the top one what is left), as
// FP32: n = f[0] + f[1] 2^14 + f[2] 2^28 (+ f[3] 2^42).  Three pieces hold
// |n| <= 2^39 (5 slices), four |n| <= 2^55.
template <int NP>
__device__ __forceinline__ void pieces(long long n, float (&f)[NP]) {
  constexpr long long bias = NP == 3 ? (8192ll << 14) + 8192ll : (8192ll << 28) + (8192ll << 14) + 8192ll;
  const long long m = n + bias;
#pragma unroll
  for (int q = 0; q < NP - 1; ++q)
    f[q] = __uint_as_float(0x4B000000u + (uint32_t(m >> (14 * q)) & 0x3FFFu)) - (8388608.0f + 8192.0f);
  // masked: a NaN's bits may be anything, and must stay a finite float
  f[NP - 1] = __uint_as_float(0x4B000000u + (uint32_t(int(m >> (14 * (NP - 1))) + 0x4000) & 0x7FFFu)) -
              (8388608.0f + 16384.0f);
}

__device__ __forceinline__ F32x2 packed(const float2& c) { return *reinterpret_cast<const F32x2*>(&c); }

// Residues of eight elements modulo every modulus, eight BF16 per 16-byte
// store.  r = f0 + c1 f1 + c2 f2 (+ c3 f3) is exact in FP32 (|c| <= 255:
// |r| < 6.3e6), q = rint(r / p) through a reciprocal of relative error below
// 2^-24 (the error of r / p, below 2^-10.2, is less than the distance
// 1 / (2 p) of a residue class from a tie), r - q p exact.  Packed FP32: two
// elements per instruction.
template <int NP>
__device__ __forceinline__ void store_residues(const OzResidues& R, const unsigned long long (&b)[8],
                                               const RowScale& rs, uint4* dst, size_t plane) {
  F32x2 f[NP][4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    float x[NP], y[NP];
    pieces<NP>(fixed_point(b[2 * u], rs), x);
    pieces<NP>(fixed_point(b[2 * u + 1], rs), y);
#pragma unroll
    for (int q = 0; q < NP; ++q) f[q][u] = pack2(x[q], y[q]);
  }
  const F32x2 magic = pack2(kRintMagic, kRintMagic), unmagic = pack2(-kRintMagic, -kRintMagic);
#pragma unroll 1
  for (int i = 0; i < R.L; ++i) {
    const F32x2 inv = packed(R.inv[i]), np = packed(R.np[i]);
    uint32_t o[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      F32x2 r = f[0][u];
#pragma unroll
      for (int q = 1; q < NP; ++q) r = fma2(f[q][u], packed(R.c[q - 1][i]), r);
      r = fma2(np, add2(fma2(r, inv, magic), unmagic), r);
      o[u] = bf16x2_of(r);
    }
    *dst = make_uint4(o[0], o[1], o[2], o[3]);
    dst += plane;
  }
}

// Any source layout: 64 x 64 tiles gathered through the address tables.
template <int NP>
__device__ __forceinline__ void residues_generic(const OzResidues& R, const OzSplitJob& jb, const OzPanel& pn, int t,
                                                 unsigned long long (*tile)[kSplitT + 1]) {
  const int ktiles = (jb.K + kSplitT - 1) / kSplitT;
  const int r0 = (t / ktiles) * kSplitT, k0 = (t % ktiles) * kSplitT;
  load_job_tile(jb, r0, k0, tile);
  __syncthreads();
  const size_t plane = size_t(pn.rows_pad) * pn.kpad / 8;
#pragma unroll 1
  for (int p = 0; p < 2; ++p) {
    const int k = 8 * (threadIdx.x & 7), r = (threadIdx.x >> 3) + 32 * p;
    if (r0 + r >= jb.rows || k0 + k >= jb.K) continue;
    unsigned long long b[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) b[u] = tile[r][k + u];  // zero beyond K
    store_residues<NP>(R, b, row_scale(pn.exps[r0 + r], R.slices),
                       reinterpret_cast<uint4*>(pn.base + (size_t(r0 + r) * pn.kpad + jb.koff + k0 + k)), plane);
  }
}

// A [K x rows] block (k contiguous): eight rows per CTA, eight consecutive k
// per thread, threads over the rows' k octets in turn (a row of 144 k has 18).
template <int NP>
__device__ __forceinline__ void residues_kmaj(const OzResidues& R, const OzSplitJob& jb, const OzPanel& pn, int t) {
  const int r0 = t * 8;
  const size_t plane = size_t(pn.rows_pad) * pn.kpad / 8;
  const int octs = (jb.K + 7) / 8, rows = min(8, jb.rows - r0);
  const bool vec = (jb.K & 1) == 0;
  for (int e = threadIdx.x; e < octs * rows; e += 256) {
    const int r = r0 + e / octs, k = 8 * (e % octs);
    const double* src = jb.src + size_t(r) * jb.K + k;
    unsigned long long b[8];
    if (vec) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        double2 v = make_double2(0.0, 0.0);
        if (k + 2 * u < jb.K) v = __ldg(reinterpret_cast<const double2*>(src + 2 * u));
        b[2 * u] = __double_as_longlong(v.x), b[2 * u + 1] = __double_as_longlong(v.y);
      }
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u) b[u] = k + u < jb.K ? __double_as_longlong(__ldg(src + u)) : 0ull;
    }
    store_residues<NP>(R, b, row_scale(pn.exps[r], R.slices),
                       reinterpret_cast<uint4*>(pn.base + (size_t(r) * pn.kpad + jb.koff + k)), plane);
  }
}

// A column-major [rows x K] block (rows contiguous), transposed through shared
// memory: 32 rows and up to eight tiles of 64 k per CTA, two tiles copied
// asynchronously (16 or 8 bytes at a time) while a third is reduced; one tile
// per CTA, loaded, then reduced, ran at 57 % of the memory bandwidth.  Element
// (k, row) of a tile lies at [k][(row + 2 (k / 8)) mod 32]: the copies' 16-byte
// pieces stay whole, and the eight octets of two rows that a half warp reads
// fall into 16 different banks.
constexpr int kRowTiles = 8, kRowStages = 3, kRowRows = 32;
__device__ __forceinline__ void copy_async(uint32_t dst, const double* src, int bytes, bool live) {
  const int n = live ? bytes : 0;  // what is left out is zero
  if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
template <int NP>
__device__ __forceinline__ void residues_rows(const OzResidues& R, const OzSplitJob& jb, const OzPanel& pn, int t,
                                              unsigned long long (*tiles)[64][kRowRows]) {
  const int kchunks = (jb.K + 64 * kRowTiles - 1) / (64 * kRowTiles);
  const int r0 = (t / kchunks) * kRowRows, kfirst = (t % kchunks) * 64 * kRowTiles;
  const int n = min(kRowTiles, (jb.K - kfirst + 63) / 64);
  const size_t plane = size_t(pn.rows_pad) * pn.kpad / 8;
  const bool vec = (jb.rows & 1) == 0;
  auto load = [&](int i, int stage) {
    if (i < n) {
      const int k0 = kfirst + 64 * i;
      const uint32_t dst = uint32_t(__cvta_generic_to_shared(tiles[stage]));
      const int rp = threadIdx.x & 15, r = r0 + 2 * rp;
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const int k = (threadIdx.x >> 4) + 16 * p;
        const bool live = k0 + k < jb.K && r < jb.rows;
        const double* src = live ? jb.src + size_t(k0 + k) * jb.rows + r : jb.src;
        const uint32_t at = dst + 8u * uint32_t(kRowRows * k + ((2 * rp + 2 * (k >> 3)) & (kRowRows - 1)));
        if (vec) {
          copy_async(at, src, 16, live);
        } else {
          copy_async(at, src, 8, live);
          copy_async(at + 8, live && r + 1 < jb.rows ? src + 1 : jb.src, 8, live && r + 1 < jb.rows);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");  // one group per tile, empty ones too
  };
  for (int i = 0; i < kRowStages - 1; ++i) load(i, i);
  const int o = threadIdx.x & 7, row = threadIdx.x >> 3;  // this thread's octet and row
  const bool live = r0 + row < jb.rows;
  const RowScale rs = row_scale(live ? pn.exps[r0 + row] : 0, R.slices);
  uint4* dst = reinterpret_cast<uint4*>(pn.base + (size_t(r0 + row) * pn.kpad + jb.koff + kfirst + 8 * o));
  int stage = 0, next = kRowStages - 1;
  for (int i = 0; i < n; ++i) {
    load(i + kRowStages - 1, next);
    next = next + 1 == kRowStages ? 0 : next + 1;
    asm volatile("cp.async.wait_group %0;" ::"n"(kRowStages - 1) : "memory");
    __syncthreads();
    if (live && kfirst + 64 * i + 8 * o < jb.K) {
      unsigned long long b[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) b[u] = tiles[stage][8 * o + u][(row + 2 * o) & (kRowRows - 1)];  // zero beyond K
      store_residues<NP>(R, b, rs, dst + 8 * i, plane);
    }
    __syncthreads();  // the tile is read before a later one lands in it
    stage = stage + 1 == kRowStages ? 0 : stage + 1;
  }
}

template <int NP>
__global__ void __launch_bounds__(256, 4) oz_residue_kernel(const __grid_constant__ OzResidues R,
                                                            const __grid_constant__ OzJobSetRefs sets) {
  extern __shared__ __align__(16) unsigned long long residue_smem[];
  const JobPiece p = job_piece(sets);
  if (p.layout == kOzRowsMajor)
    residues_rows<NP>(R, p.jb, p.pn, p.tile, reinterpret_cast<unsigned long long(*)[64][kRowRows]>(residue_smem));
  else if (p.layout == kOzKMajor)
    residues_kmaj<NP>(R, p.jb, p.pn, p.tile);
  else
    residues_generic<NP>(R, p.jb, p.pn, p.tile, reinterpret_cast<unsigned long long(*)[kSplitT + 1]>(residue_smem));
}
constexpr size_t kRowsSmem = kRowStages * 64 * kRowRows * sizeof(unsigned long long);
constexpr size_t kGenericSmem = kSplitT * (kSplitT + 1) * sizeof(unsigned long long);

// ------------------------------------------------------------------ result side
// The integer X with X = s_i (mod p_i), |X| < prod p / 2 (the host admits only
// sums below 0.49 prod p), scaled by 2^e2 and rounded once:
//     X = sum_i y_i (P / p_i) - k P,   y_i = s_i (P / p_i)^-1 mod p_i,
//     k = rint(sum_i y_i / p_i)
// in W signed 32-bit word columns of 64-bit sums, modulo 2^(32 W): three words
// hold |X| < 2^95, four |X| < 2^127, five any sum that 15 moduli hold (2^133).
// Two sums at a time: the residue arithmetic in packed FP32.
template <int W>
struct CrtPair {
  long long col[2][W];
  F32x2 turns;
  __device__ __forceinline__ void clear(const OzCrt& T) {
    turns = 0ull;  // two +0
#pragma unroll
    for (int w = 0; w < W; ++w) col[0][w] = col[1][w] = T.base[w];
  }
  // two biased residues (16-bit halves of s, below 2^15 + 2^8) less the bias
  // in `unbias` = -2^23 - bias; |s| < 2^14, |cinv| < 2^8: the product is an exact
  // FP32 integer.  The integers enter the columns with the bits of 1.5 2^23 and
  // T.base takes them out again (modulo 2^64, like every step of a column).
  __device__ __forceinline__ void add(const OzCrt& T, int i, int s, F32x2 unbias, F32x2 magic, F32x2 unmagic) {
    const F32x2 x = add2(pack2(__uint_as_float(__byte_perm(uint32_t(s), 0x4B000000u, 0x7610)),
                               __uint_as_float(__byte_perm(uint32_t(s), 0x4B000000u, 0x7632))),
                         unbias);
    const F32x2 v = fma2(x, packed(T.cinv[i]), 0ull);
    const F32x2 y = fma2(packed(T.np[i]), add2(fma2(v, packed(T.inv[i]), magic), unmagic), v);
    turns = fma2(y, packed(T.inv[i]), turns);
    float y0, y1;
    unpack2(add2(y, magic), y0, y1);
#pragma unroll
    for (int w = 0; w < W; ++w) {
      col[0][w] = mad_wide(int(__float_as_uint(y0)), T.m[i][w], col[0][w]);
      col[1][w] = mad_wide(int(__float_as_uint(y1)), T.m[i][w], col[1][w]);
    }
  }
  __device__ __forceinline__ void value(const OzCrt& T, const int (&e2)[2], bool neg, double (&out)[2]) {
    float t0, t1;
    unpack2(turns, t0, t1);
    out[0] = one(T, col[0], t0, e2[0], neg);
    out[1] = one(T, col[1], t1, e2[1], neg);
  }
  static __device__ __forceinline__ double one(const OzCrt& T, long long (&c)[W], float turns, int e2, bool neg) {
    const int k = 0x4B400000 - int(__float_as_uint(__fadd_rn(turns, kRintMagic)));
#pragma unroll
    for (int w = 0; w < W; ++w) c[w] = mad_wide(k, T.prod[w], c[w]);
    if constexpr (W == 5) {
      uint32_t w[5];
      long long t = 0;
#pragma unroll
      for (int j = 0; j < 5; ++j) t += c[j], w[j] = uint32_t(t), t >>= 32;
      const bool minus = int(w[4]) < 0;
      if (minus) {
        unsigned long long carry = 1;
#pragma unroll
        for (int j = 0; j < 5; ++j) carry += uint32_t(~w[j]), w[j] = uint32_t(carry), carry >>= 32;
      }
      const unsigned long long a = (unsigned long long)w[4] << 32 | w[3], b = (unsigned long long)w[2] << 32 | w[1];
      if (a) {  // from 2^96 on: the top 62 bits, the last one sticky
        const int n = clz64(a);
        const unsigned long long top = n ? a << n | b >> (64 - n) : a, rest = b << n | w[0];
        const long long v = (long long)(top >> 2 | ((top & 3u) || rest ? 1ull : 0ull));
        return i64_scaled_to_double(minus ? -v : v, e2 + 98 - n, neg);
      }
      return small((unsigned long long)w[2], (unsigned long long)w[1] << 32 | w[0], minus, e2, neg);
    }
    unsigned __int128 x = (unsigned __int128)(__int128)c[0] + ((unsigned __int128)(__int128)c[1] << 32);
    if constexpr (W == 4) {
      x += ((unsigned __int128)(__int128)c[2] << 64) + ((unsigned __int128)(unsigned long long)c[3] << 96);
    } else {
      const long long hi = (long long)(unsigned long long)(x >> 64) + c[2];
      x = ((unsigned __int128)(unsigned long long)(long long)int(hi) << 64) | (unsigned long long)x;  // 96 bits, signed
    }
    const bool minus = (__int128)x < 0;
    const unsigned __int128 u = minus ? -x : x;
    const unsigned long long hi = (unsigned long long)(u >> 64), lo = (unsigned long long)u;
    if constexpr (W == 3) {
      // |X| in [2^64, 2^95) without a branch: its top 62 bits, the last one sticky
      const uint32_t h = uint32_t(hi), m = uint32_t(lo >> 32), l = uint32_t(lo);
      const int n = __clz(int(h | 1u));
      const uint32_t top = __funnelshift_l(m, h, n), low = __funnelshift_l(l, m, n), rest = l << n;
      const unsigned long long kept = ((unsigned long long)top << 32 | low) >> 2;
      const long long v = (long long)(kept | ((low & 3u) | rest ? 1ull : 0ull));
      double r;
      if (i64_scaled_normal(v, e2 + 34 - n, &r) && h) return minus != neg ? -r : r;
    }
    return small(hi, lo, minus, e2, neg);
  }
  // (minus ? -1 : 1) (hi 2^64 + lo) 2^e2: the top 62 bits, what is below them
  // folded into the last (a sticky bit: the rounding position lies above it)
  static __device__ __forceinline__ double small(unsigned long long hi, unsigned long long lo, bool minus, int e2,
                                                 bool neg) {
    const int sh = (hi ? 64 - clz64(hi) : -clz64(lo | 1ull)) + 2;
    long long v = (long long)lo;
    if (sh > 0) {
      const unsigned long long kept = sh >= 64 ? hi >> (sh - 64) : (hi << (64 - sh)) | (lo >> sh);
      const unsigned long long below = sh >= 64 ? lo | (hi & ((1ull << (sh - 64)) - 1)) : lo & ((1ull << sh) - 1);
      v = (long long)(kept | (below ? 1ull : 0ull));
      e2 += sh;
    }
    return i64_scaled_to_double(minus ? -v : v, e2, neg);
  }
};

// One CTA per 64 rows x 8 columns of a tile (a small step has few tiles, so
// the pieces are small): a thread reads two rows of one column (one 4-byte
// load per modulus and split, all moduli's in flight), sums the splits'
// residues (two non-negative 16-bit sums in one 32-bit one: at most 64 splits
// of at most 512), reconstructs, scales and
// stores along D's unit-stride dimension (through shared memory when that is
// n).  About 200 instructions an element and the loads' latency bound it, not
// HBM: four CTAs per SM (up to 12 moduli; more spill) and packed residue
// arithmetic took the o=40/v=300 ring step's reconstruction from 2.57 to 2.02 ms.
constexpr int kRecThreads = 256;
template <int L, int W>
__global__ void __launch_bounds__(kRecThreads, L <= 12 && W == 3 ? 4 : 3) oz_residue_recombine_kernel(
    const __grid_constant__ OzCrt T, const OzTile* __restrict__ tiles, const OzDBlock* __restrict__ dblocks,
    const OzPanel* __restrict__ pa, const OzPanel* __restrict__ pb, const int16_t* __restrict__ ws, int log_rows,
    int log_cols, int nsplit, int mode) {
  __shared__ double sm[64][9];
  const int log_rp = log_rows - 6, log_cp = log_cols - 3;  // 64-row pieces, 8-column pieces
  const int tile = blockIdx.x >> (log_rp + log_cp);
  const int piece = blockIdx.x & ((1 << (log_rp + log_cp)) - 1);
  const int sr = (piece & ((1 << log_rp) - 1)) * 64, sc = (piece >> log_rp) * 8;
  const int rp = 2 * (threadIdx.x & 31), cl = threadIdx.x >> 5;
  const size_t plane = size_t(1) << (log_rows + log_cols);  // one split's [cols][rows]
  const int* q = reinterpret_cast<const int*>(ws + size_t(tile) * L * nsplit * plane +
                                              (size_t(sc + cl) << log_rows) + sr + rp);
  const size_t step = size_t(nsplit) * plane / 2;
  // the first split's loads leave before the tile's tables are known (a tile's
  // workspace is whole, whatever of it lies in D)
  int s[L];
#pragma unroll
  for (int i = 0; i < L; ++i) s[i] = __ldg(q + size_t(i) * step);
  const OzTile tl = tiles[tile];
  const OzDBlock db = dblocks[tl.dblock];
  if (tl.n0 + sc >= db.N || tl.m0 + sr >= db.M) return;  // the piece lies beyond D
  const int m = tl.m0 + sr + rp, n = tl.n0 + sc + cl;
  double v[2] = {0.0, 0.0};
  if (m < db.M && n < db.N) {
    for (int sp = 1; sp < nsplit; ++sp)
#pragma unroll
      for (int i = 0; i < L; ++i) s[i] += __ldg(q + size_t(i) * step + size_t(sp) * (plane / 2));
    const int bias = kOzResidueBias * nsplit;
    const int e0 = pa[tl.panel_a].exps[m], f = pb[tl.panel_b].exps[n];
    const int e1 = m + 1 < db.M ? pa[tl.panel_a].exps[m + 1] : 0;
    const int F = (f ? f : 1) - 1022 + 2 - 2 * kDigitBits * T.slices;
    CrtPair<W> crt;
    crt.clear(T);
    const float off = -8388608.0f - float(bias);
    const F32x2 unbias = pack2(off, off), magic = pack2(kRintMagic, kRintMagic), unmagic = pack2(-kRintMagic, -kRintMagic);
#pragma unroll
    for (int i = 0; i < L; ++i) crt.add(T, i, s[i], unbias, magic, unmagic);
    const int e2[2] = {(e0 ? e0 : 1) - 1022 + F, (e1 ? e1 : 1) - 1022 + F};
    crt.value(T, e2, mode & 2, v);
    if (e0 == kNonFiniteExp || f == kNonFiniteExp) v[0] = __longlong_as_double(0x7FF8000000000000ll);
    if (e1 == kNonFiniteExp || f == kNonFiniteExp) v[1] = __longlong_as_double(0x7FF8000000000000ll);
  }
  if (!db.col_fast) {
    if (n >= db.N) return;
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (m + h < db.M) {
        double* dst = db.colptr[n] + db.rowoff[m + h];
        *dst = (mode & 1) ? *dst + v[h] : v[h];
      }
    return;
  }
  sm[rp][cl] = v[0], sm[rp + 1][cl] = v[1];
  __syncthreads();
  for (int e = threadIdx.x; e < 64 * 8; e += kRecThreads) {
    const int c = e & 7, row = e >> 3;
    const int mm = tl.m0 + sr + row, nn = tl.n0 + sc + c;
    if (mm < db.M && nn < db.N) {
      double* dst = db.colptr[nn] + db.rowoff[mm];
      *dst = (mode & 1) ? *dst + sm[row][c] : sm[row][c];
    }
  }
}

}  // namespace

// Products the residue form needs for K columns at `slices` slices: the
// smallest count whose moduli hold every sum |sum| <= K 4^(8 slices - 1) below
// 0.49 of their product; 0 when none does (15 hold sums below 2^133).  At 5
// slices or more and k ranges worth it (batch.cu), 10 to 15.
int oz_residue_count(int slices, int64_t K) {
  if (K < 1) return 0;
  const double need = 2.0 * (8.0 * slices - 1.0) + std::log2(double(K));
  double have = std::log2(0.49);
  for (int i = 0; i < kOzMaxResidues; ++i) {
    have += std::log2(double(kModuli[i]));
    if (i >= 9 && have > need + 1e-6) return i + 1;  // at least the 10 the kernels are built for
  }
  return 0;
}

void oz_residue_tables(int slices, int L, int64_t K, OzResidues* r, OzCrt* t) {
  *r = OzResidues{};
  *t = OzCrt{};
  r->L = t->L = L;
  r->slices = t->slices = slices;
  const double bits = 2.0 * (8.0 * slices - 1.0) + std::log2(double(K));
  t->words = bits < 94.9 ? 3 : bits < 126.9 ? 4 : 5;
  Words160 prod;
  for (int i = 0; i < L; ++i) prod.times(unsigned(kModuli[i]));
  signed_words(prod, t->prod);
  for (int i = 0; i < L; ++i) {
    const int p = kModuli[i];
    r->np[i] = t->np[i] = make_float2(-float(p), -float(p));
    r->inv[i] = t->inv[i] = make_float2(1.0f / float(p), 1.0f / float(p));
    for (int q = 0; q < 3; ++q) {
      const float c = float(symmetric(1ll << (14 * (q + 1)), p));
      r->c[q][i] = make_float2(c, c);
    }
    Words160 m;
    long long mp = 1;
    for (int j = 0; j < L; ++j)
      if (j != i) m.times(unsigned(kModuli[j])), mp = mp * kModuli[j] % p;
    signed_words(m, t->m[i]);
    const float c = float(symmetric(inverse_mod(int(mp), p), p));
    t->cinv[i] = make_float2(c, c);
    for (int w = 0; w < 5; ++w)
      t->base[w] = (long long)((unsigned long long)t->base[w] - 0x4B400000ull * (unsigned long long)(long long)t->m[i][w]);
  }
}

int64_t oz_residue_tiles(int layout, int rows, int K) {
  if (layout == kOzRowsMajor) return int64_t((rows + kRowRows - 1) / kRowRows) * ((K + 64 * kRowTiles - 1) / (64 * kRowTiles));
  return oz_split_tiles(layout, rows, K);
}

int oz_launch_residues(const OzJobSetRefs& sets, const OzResidues& r, cudaStream_t s) {
  if (!sets.total) return A4G_OK;
  if (!sets.fits()) return fail(A4G_ERR_RANGE, "too many split tiles");
  size_t smem = 0;  // what the layouts at hand need: it bounds the CTAs per SM
  for (int q = 0; q < sets.n; ++q) {
    if (sets.s[q].layout == kOzRowsMajor) smem = std::max(smem, kRowsSmem);
    if (sets.s[q].layout == kOzGeneric) smem = std::max(smem, kGenericSmem);
  }
  if (r.slices <= 5) oz_residue_kernel<3><<<unsigned(sets.total), 256, smem, s>>>(r, sets);
  else oz_residue_kernel<4><<<unsigned(sets.total), 256, smem, s>>>(r, sets);
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

int oz_residue_prepare() {
  A4G_CUDA(cudaFuncSetAttribute(oz_residue_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(std::max(kRowsSmem, kGenericSmem))));
  A4G_CUDA(cudaFuncSetAttribute(oz_residue_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(std::max(kRowsSmem, kGenericSmem))));
  return A4G_OK;
}

int oz_launch_residue_recombine(const OzTile* tiles, int ntiles, int tile_rows, int tile_cols,
                                const OzDBlock* dblocks, const OzPanel* pa, const OzPanel* pb, const void* ws,
                                const OzCrt& t, int nsplit, int mode, cudaStream_t s) {
  if (ntiles <= 0) return A4G_OK;
  const int lr = tile_rows == 256 ? 8 : 7, lc = tile_cols == 256 ? 8 : 7;
  const int64_t pieces = int64_t(ntiles) * (tile_rows / 64) * (tile_cols / 8);
  if (nsplit > 64 || pieces > 0x7fffffffLL) return fail(A4G_ERR_RANGE, "too many tiles");
  auto go = [&](auto l, auto w) {
    oz_residue_recombine_kernel<decltype(l)::value, decltype(w)::value><<<unsigned(pieces), kRecThreads, 0, s>>>(
        t, tiles, dblocks, pa, pb, static_cast<const int16_t*>(ws), lr, lc, nsplit, mode);
  };
  const std::integral_constant<int, 3> w3;
  const std::integral_constant<int, 4> w4;
  switch (t.L) {
    case 10: go(std::integral_constant<int, 10>(), w3); break;  // 10 moduli hold sums below 2^89
    case 11:
      if (t.words == 3) go(std::integral_constant<int, 11>(), w3);
      else go(std::integral_constant<int, 11>(), w4);
      break;
    case 12: go(std::integral_constant<int, 12>(), w4); break;
    case 13: go(std::integral_constant<int, 13>(), w4); break;
    case 14: go(std::integral_constant<int, 14>(), w4); break;
    case 15:
      if (t.words == 5) go(std::integral_constant<int, 15>(), std::integral_constant<int, 5>());
      else go(std::integral_constant<int, 15>(), w4);
      break;
    default: return fail(A4G_ERR_ARG, "residue form: 10 to 15 moduli");
  }
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

}  // namespace a4g
