// Split-precision (Ozaki scheme) block contraction on the tcgen05 tensor cores.
//
// Each FP64 operand row (left blocks) / column (right blocks) is scaled by a
// power of two with |x| < 2^E over the whole row of the pardo step, rounded to
// the integer n = round(x * 2^(8*slices - E - 1)) (|n| <= 2^(8*slices-1)) and
// cut into `slices` balanced base-256 digits:
//     x ~= sum_i d_i * 2^(E + 1 - 8(i+1)),   d_0 in [-128, 128], d_i in [-128, 127].
// Digits are exact BF16 values and every digit product is at most 2^14.  The
// product of two slices is an integer matrix, so
//     L*R ~= sum_t 2^(E_m + F_n + 2 - 8(t+2)) * S_t,   S_t = sum_{i+j=t} A_i B_j
// over levels t < slices (triangular truncation).  Each S_t is computed on the
// tensor cores (kind::f16, BF16 x BF16 -> FP32) in chunks of k short enough
// that every FP32 partial sum is an integer below 2^24 and therefore exact;
// the epilogue warps fold each chunk into an exact running sum (an FP32 (hi,
// lo) TwoSum pair kept in TMEM for 128-column tiles, int32 registers for
// 256-column tiles).  A final FP64 kernel applies the powers of two and
// writes D.
//
// Published method: Ozaki, Ogita, Oishi, Rump, "Error-free transformations of
// matrix multiplication by using fast routines of matrix multiplication and
// its applications", Numer. Algorithms 59 (2012); Mukunoki, Ozaki, Ogita,
// Imamura, "DGEMM using Tensor Cores, and Its Accurate and Reproducible
// Versions", ISC 2020 (slices on tensor cores with exact FP32 accumulation).
//
// Kernels:
//   oz_exp_kernel       max exponent per panel row          (HBM: 8 B/elem read)
//   oz_split_kernel     FP64 -> BF16 digit slices, K-major   (HBM: 8 B read + 2*slices B write)
//                       with the block's index permute folded into the gather; both take every
//                       operand side and source layout of a step in one launch
//   oz_gemm_kernel<PAIR, BN, DIRECT, ENERGY>
//                       persistent warp-specialised tcgen05 GEMM: TMA (SW128)
//                       -> smem ring -> tcgen05.mma into TMEM (2 accumulators)
//                       -> epilogue warps fold each exact chunk into the level
//                       sum.  Four forms: one SM or a CTA pair (cta_group::2)
//                       per tile, 128 or 256 columns per MMA; the batch
//                       autotunes among them.
//   oz_recombine_kernel int64 sum over split-K units, FP64 combination of the
//                       levels, scaled store into D
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "a4g_internal.h"
#include "exact_fp.h"
#include "f32x2.h"
#include "grouped.h"
#include "oz_device.h"
#include "ozaki.h"

namespace a4g {
namespace {

constexpr int kThreadsOz = 320;  // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue
// Direct forms: warps 2..17 epilogue (four per TMEM lane quadrant, 32 columns
// each): their epilogue also rounds and stores every result.
constexpr int kThreadsOzDirect = 576;
constexpr uint32_t kTileBytes = kOzBM * kOzBK * 2;  // 16 KB per operand tile
// TMEM columns, 128-column forms: [0,128) and [128,256) are the two FP32 MMA
// accumulators; [256,384) and [384,512) hold the running exact (hi, lo) sums of
// the current level.  256-column forms: [0,256) and [256,512) are the two
// accumulators; the level sums live in the epilogue threads' registers.
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kTmemHi = 256, kTmemLo = 384;
// Direct form: the same two regions hold the low and high 32-bit words of the
// exact 64-bit running sum over levels.
constexpr uint32_t kTmemW0 = 256, kTmemW1 = 384;
constexpr unsigned long long kWaitLimitNs = 20ull * 1000 * 1000 * 1000;  // 20 s

// tcgen05 instruction descriptor, kind::f16: D F32 (bits 4-5 = 1), A BF16
// (bits 7-9 = 1), B BF16 (bits 10-12 = 1), both K-major (bits 15/16 = 0),
// N>>3 at bits 17-22, M>>4 at bits 24-28.
template <int M, int N>
constexpr uint32_t idesc_bf16() {
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(N >> 3) << 17) | (uint32_t(M >> 4) << 24);
}

// Shared memory of the tensor-core kernel, per form (PAIR: a CTA pair computes
// one tile with cta_group::2; BN: tile columns).  Each CTA stages its 128 rows
// of A and its BN (1-SM) or BN/2 (pair) rows of B per 64-wide k block:
//   1-SM BN=128: 32 KB x 6 stages   pair BN=128: 24 KB x 9
//   1-SM BN=256: 48 KB x 4 stages   pair BN=256: 32 KB x 6
template <bool PAIR, int BN>
struct __align__(1024) OzSmemT {
  static constexpr uint32_t kBBytes = uint32_t(PAIR ? BN / 2 : BN) * kOzBK * 2;
  static constexpr int kSt = int((216u * 1024u) / (kTileBytes + kBBytes)) > 9 ? 9
                                                                               : int((216u * 1024u) / (kTileBytes + kBBytes));
  uint8_t a[kSt][kTileBytes];
  uint8_t b[kSt][kBBytes];
  uint64_t full[kSt], empty[kSt];
  uint64_t acc_full[2], acc_empty[2];
  uint64_t drain;
  uint32_t tmem_base;
  volatile int abort;
};

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) { mbar_expect_tx(smem_u32(bar), bytes); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after kWaitLimitNs or when another role aborted.
template <class SM>
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, SM& sm, int* err, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = now_ns();
#pragma unroll 1
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255) == 0) {
      if (sm.abort) return false;
      if (now_ns() - t0 > kWaitLimitNs) {
        sm.abort = 1;
        atomicExch(err, code);
        return false;
      }
    }
  }
}
// The same wait by a whole warp (shared-memory address of the barrier): every
// lane returns the same answer, so the warp stays converged around the
// single-thread issues that follow.
template <class SM>
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, SM& sm, int* err, int code) {
  auto done = [&]() {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return __all_sync(0xffffffffu, ok != 0) != 0;
  };
  if (done()) return true;
  const unsigned long long t0 = now_ns();
#pragma unroll 1
  for (uint32_t it = 1;; ++it) {
    if (done()) return true;
    if ((it & 255) == 0) {
      const bool late = now_ns() - t0 > kWaitLimitNs;
      if (__any_sync(0xffffffffu, sm.abort || late)) {
        if (!sm.abort) {
          sm.abort = 1;
          atomicExch(err, code);
        }
        __syncwarp();
        return false;
      }
    }
  }
}
// One lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const void* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          dst),
      "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) { tc_commit(smem_u32(bar)); }
template <int N>
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc_bf16<128, N>()), "r"(accum));
}
// --- CTA-pair (cta_group::2) forms
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared variable in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_shared(const void* p, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(smem_u32(p)), "r"(rank));
  return out;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_cluster(uint32_t bar_cluster, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(bar_cluster), "r"(bytes)
               : "memory");
}
// TMA load into this CTA's shared memory that signals an mbarrier which may
// live in either CTA of the pair
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const void* map, uint32_t bar_cluster, int c0, int c1,
                                                 int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          dst),
      "l"(map), "r"(bar_cluster), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
template <int N>
__device__ __forceinline__ void tc_mma_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc_bf16<256, N>()), "r"(accum));
}
// arrive on the mbarrier at the same offset in both CTAs of the pair once
// this thread's tcgen05 operations complete
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          bar),
      "h"(uint16_t(3))
      : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) { tc_commit_pair(smem_u32(bar)); }

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, rows of 128 B,
// 8-row core groups 1024 B apart (SBO), descriptor version 1 (bits 46-48).
// The low word holds the tile's address (in 16-byte units) and the leading
// byte offset (unused for SW128 K-major); the high word is the same for all.
__device__ __forceinline__ uint32_t sw128_desc_lo(const void* tile) {
  return ((smem_u32(tile) & 0x3FFFF) >> 4) | (1u << 16);
}
__device__ __forceinline__ uint64_t sw128_desc(uint32_t lo) {
  constexpr uint32_t hi = uint32_t(1024 >> 4) | (1u << 14) | (2u << 29);  // SBO, version 1, SWIZZLE_128B
  return (uint64_t(hi) << 32) | lo;
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 32 consecutive TMEM columns of this thread's lane; completes at tc_wait_ld().
__device__ __forceinline__ void tc_ld32_nowait(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tc_ld16_nowait(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// Exact accumulation of an integer-valued float x (|x| < 2^24) into hi + lo.
__device__ __forceinline__ void two_sum_acc(float& hi, float& lo, float x) {
  const float s = __fadd_rn(hi, x);
  const float bp = __fsub_rn(s, hi);
  const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(x, bp));
  hi = s;
  lo = __fadd_rn(lo, e);
}

// ------------------------------------------------------------------ roles
// Walks the k blocks of one unit: calls f(koff_a, koff_b, kb) per 64-wide
// block (the panels are zero beyond the end of every stretch of pairs up to
// the next 64-column boundary, so whole blocks are always multiplied).
template <class F>
__device__ __forceinline__ void for_unit_kblocks(const OzGemmArgs& a, const OzUnit& un, const OzTile& tl,
                                                 F&& f) {
  int kb = un.kb_begin;
  int q = un.trip_first, j = un.kb_in_trip;
  while (kb < un.kb_end && q < tl.trip_end) {
    const OzTrip tr = a.trips[q];
    for (; j < tr.nkb && kb < un.kb_end; ++j, ++kb)
      if (!f(int(tr.koff_a) + j * kOzBK, int(tr.koff_b) + j * kOzBK, kb)) return;
    ++q;
    j = 0;
  }
}

// Units are distributed over CTAs (1-SM form) or over CTA pairs (2-SM form:
// both CTAs of a pair walk the same units).
template <bool PAIR>
__device__ __forceinline__ int unit_first() { return PAIR ? int(blockIdx.x >> 1) : int(blockIdx.x); }
template <bool PAIR>
__device__ __forceinline__ int unit_stride() { return PAIR ? int(gridDim.x >> 1) : int(gridDim.x); }

// This CTA's (pair's) units in run order; f(u) returns false to stop.  The
// direct form hands out whole tiles: units (tile, 0..slices-1) in a row.
template <bool PAIR, class F>
__device__ __forceinline__ void for_units(const OzGemmArgs& a, F&& f) {
  if (a.direct) {
    const int groups = a.n_units / a.slices;
    for (int g = unit_first<PAIR>(); g < groups; g += unit_stride<PAIR>())
      for (int lv = 0; lv < a.slices; ++lv)
        if (!f(g * a.slices + lv)) return;
  } else {
    for (int u = unit_first<PAIR>(); u < a.n_units; u += unit_stride<PAIR>())
      if (!f(u)) return;
  }
}

// Both single-issuer roles run as whole, converged warps: every lane keeps the
// loop's counters and waits, one elected lane issues.  Stage addresses,
// barriers and descriptors are the first stage's plus a multiple of the stage
// index, with no division and no address conversion in the loop: a role whose
// instructions for one stage (64 k: 512 clocks of MMAs for a 256-column tile)
// take longer than the stage itself starves the tensor cores.
template <bool PAIR, int BN, bool RES>
__device__ void producer(const OzGemmArgs& a, OzSmemT<PAIR, BN>& sm, uint32_t rank) {
  using SM = OzSmemT<PAIR, BN>;
  constexpr uint32_t kBytes = kTileBytes + SM::kBBytes;
  const bool leader = elect_one();
  const uint32_t a0 = smem_u32(sm.a[0]), b0 = smem_u32(sm.b[0]), empty0 = smem_u32(&sm.empty[0]);
  const uint32_t full0 = PAIR ? mapa_shared(&sm.full[0], 0) : smem_u32(&sm.full[0]);  // pair: the leader CTA's
  uint32_t s = 0, free_parity = 1;
  for_units<PAIR>(a, [&](int u) {
    const OzUnit un = a.units[u];
    const OzTile tl = a.tiles[un.tile];
    const int level = un.level;
    const void* ma = static_cast<const uint8_t*>(a.maps_a) + size_t(tl.panel_a) * 128;
    const void* mb = static_cast<const uint8_t*>(a.maps_b) + size_t(tl.panel_b) * 128;
    const int first = RES ? level : 0;
    const int ar = tl.m0 + int(rank) * kOzBM;                       // this CTA's 128 rows of A
    const int br = tl.n0 + (PAIR ? int(rank) * (BN / 2) : 0);  // and of B (pair form: half of them)
    bool ok = true;
    for_unit_kblocks(a, un, tl, [&](int ka, int kb, int) {
      for (int i = first; i <= level; ++i) {
        const int j = RES ? level : level - i;  // the B slice, or the modulus' own
        if (!warp_wait(empty0 + 8 * s, free_parity, sm, a.err_flag, 1)) return ok = false;
        if (leader) {
          const uint32_t fb = full0 + 8 * s;
          if constexpr (PAIR) {
            mbar_expect_tx_cluster(fb, kBytes);
            tma_load_3d_pair(a0 + s * kTileBytes, ma, fb, ka, ar, i);
            tma_load_3d_pair(b0 + s * SM::kBBytes, mb, fb, kb, br, j);
          } else {
            mbar_expect_tx(fb, kBytes);
            tma_load_3d(a0 + s * kTileBytes, ma, fb, ka, ar, i);
            tma_load_3d(b0 + s * SM::kBBytes, mb, fb, kb, br, j);
          }
        }
        __syncwarp();
        if (++s == uint32_t(SM::kSt)) s = 0, free_parity ^= 1;
      }
      return true;
    });
    return ok;
  });
}

// One lane issues every MMA (in the leader CTA's warp in the pair form).
template <bool PAIR, int BN, bool RES>
__device__ void mma_issuer(const OzGemmArgs& a, OzSmemT<PAIR, BN>& sm, uint32_t tmem) {
  using SM = OzSmemT<PAIR, BN>;
  const bool leader = elect_one();
  const uint32_t full0 = smem_u32(&sm.full[0]), empty0 = smem_u32(&sm.empty[0]);
  const uint32_t acc_full0 = smem_u32(&sm.acc_full[0]), acc_empty0 = smem_u32(&sm.acc_empty[0]);
  const uint32_t ad0 = sw128_desc_lo(sm.a[0]), bd0 = sw128_desc_lo(sm.b[0]);
  uint32_t s = 0, full_parity = 0, chunk = 0;
  for_units<PAIR>(a, [&](int u) {
    const OzUnit un = a.units[u];
    const OzTile tl = a.tiles[un.tile];
    const int ckb = a.chunk_kb[un.level];
    const int products = RES ? 1 : un.level + 1;
    int left = 0;  // k blocks left in the chunk (0: a new chunk)
    uint32_t buf = 0;
    bool ok = true;
    for_unit_kblocks(a, un, tl, [&](int, int, int kb) {
      uint32_t acc = 1;
      if (left == 0) {
        buf = chunk & 1;
        if (!warp_wait(acc_empty0 + 8 * buf, ((chunk >> 1) & 1) ^ 1, sm, a.err_flag, 2)) return ok = false;
        tc_fence_after();
        left = min(ckb, un.kb_end - kb);
        acc = 0;
      }
      const uint32_t d_tmem = tmem + buf * BN;
      --left;
      for (int i = 0; i < products; ++i) {
        if (!warp_wait(full0 + 8 * s, full_parity, sm, a.err_flag, 3)) return ok = false;
        tc_fence_after();
        if (leader) {
          const uint32_t ad = ad0 + s * (kTileBytes >> 4), bd = bd0 + s * (SM::kBBytes >> 4);
#pragma unroll
          for (int kk = 0; kk < kOzBK / 16; ++kk) {
            const uint32_t ac = kk == 0 ? acc : 1u;
            if constexpr (PAIR) tc_mma_pair<BN>(d_tmem, sw128_desc(ad + 2 * kk), sw128_desc(bd + 2 * kk), ac);
            else tc_mma<BN>(d_tmem, sw128_desc(ad + 2 * kk), sw128_desc(bd + 2 * kk), ac);
          }
          if constexpr (PAIR) tc_commit_pair(empty0 + 8 * s);
          else tc_commit(empty0 + 8 * s);
          if (left == 0 && i == products - 1) {
            if constexpr (PAIR) tc_commit_pair(acc_full0 + 8 * buf);
            else tc_commit(acc_full0 + 8 * buf);
          }
        }
        __syncwarp();
        acc = 1;
        if (++s == uint32_t(SM::kSt)) s = 0, full_parity ^= 1;
      }
      if (left == 0) ++chunk;
      return true;
    });
    return ok;
  });
}

__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
      "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tc_ld8_nowait(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

// Direct form: what a thread needs to store its part of a tile (its row,
// columns col0..col0+31), gathered once when the tile starts (while the
// tensor cores work on the tile's first level): the row's D offset and
// scale; the 32 columns' D bases and scales go to the warp's table in shared
// memory (read back as broadcasts).
struct DirectCol {
  double* colp;  // column base in D; null: column outside D
  int F;         // biased column exponent (at least 1)
  int pad;
};
// Energy form: a second per-warp table (only that kernel declares it, so the
// store forms keep their shared memory).
struct EnergyCol {
  double ec;  // the column's last-term orbital energy (when the last term is a column index)
  int ck;     // the column's index into the prefix table (-1: outside D)
  int pad;
};
struct DirectTile {
  long long roff;   // the row's offset from a column base
  DirectCol* cols;  // this warp's 32 entries
  int ebase;        // row scale and constant part of the result's exponent
  bool mlive;
  bool nonfinite;   // the row holds a non-finite operand value
  // energy form
  EnergyCol* ecols;    // this warp's 32 entries
  const double* prow;  // the row's prefix-table row
  double er;           // the row's last-term orbital energy (when the last term is a row index)
  bool last_row;
};

template <bool ENERGY>
__device__ __forceinline__ void direct_tile(DirectTile& t, const OzGemmArgs& a, const OzTile& tl, int row,
                                            int col0, int lane) {
  const OzDBlock db = a.dblocks[tl.dblock];
  const int m = tl.m0 + row, n = tl.n0 + col0 + lane;
  t.mlive = m < db.M;
  int Em = 1;
  t.roff = 0;
  t.nonfinite = false;
  [[maybe_unused]] OzEnergyBlock eb{};
  if constexpr (ENERGY) {
    eb = a.eblocks[tl.dblock];
    t.last_row = eb.last_row != 0;
    t.prow = eb.ptab;
    t.er = 0.0;
  }
  if (t.mlive) {
    const int e = a.panels_a[tl.panel_a].exps[m];
    Em = e ? e : 1;
    t.nonfinite = e == kNonFiniteExp;
    if constexpr (ENERGY) {
      t.prow = eb.ptab + int64_t(eb.rk[m]) * eb.ckn;
      if (t.last_row) t.er = eb.elast[m];
    } else {
      t.roff = db.rowoff[m];
    }
  }
  t.ebase = Em - 1022 - 1022 + 2 - kDigitBits * (a.slices + 1);
  DirectCol c{nullptr, 1, 0};
  [[maybe_unused]] EnergyCol ec{0.0, -1, 0};
  if (n < db.N) {
    const int f = a.panels_b[tl.panel_b].exps[n];
    c.F = f ? f : 1;
    if constexpr (ENERGY) {
      ec.ck = eb.ck[n];
      if (!eb.last_row) ec.ec = eb.elast[n];
    } else {
      c.colp = db.colptr[n];
    }
  }
  __syncwarp();  // the previous tile's entries are read
  t.cols[lane] = c;
  if constexpr (ENERGY) t.ecols[lane] = ec;
  __syncwarp();
}

// Accumulate mode: asks L2 for the thread's 32 D elements when the tile
// starts, so that the loads after its last chunk find them there.
__device__ __forceinline__ void prefetch_direct(const DirectTile& t) {
  if (!t.mlive) return;
#pragma unroll 8
  for (int j = 0; j < 32; ++j) {
    double* cp = t.cols[j].colp;
    if (cp) asm volatile("prefetch.global.L2 [%0];" ::"l"(cp + t.roff));
  }
}

__device__ __forceinline__ void load_d8(const DirectTile& t, int c0, bool acc, double (&d)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    double* cp = t.cols[c0 + j].colp;
    d[j] = 0.0;
    if (acc && t.mlive && cp) d[j] = cp[t.roff];
  }
}

// Direct form, after the last chunk of a tile's last level: rounds the 32
// exact 64-bit sums of this thread's row held in TMEM (low words at w0addr,
// high words kTmemW1 - kTmemW0 columns further) to FP64 with the row and
// column scales and stores (or adds) them into D, 8 columns at a time; in the
// accumulate mode the next 8 D loads are in flight while 8 are added.
__device__ __forceinline__ void store_direct(const OzGemmArgs& a, const DirectTile& t, uint32_t w0addr) {
  if (a.dry) return;
  const bool acc = a.mode & 1;
  double dn[8];
  load_d8(t, 0, acc, dn);
#pragma unroll 1
  for (int p = 0; p < 4; ++p) {
    double dc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) dc[j] = dn[j];
    if (p < 3) load_d8(t, 8 * (p + 1), acc, dn);
    uint32_t w0[8], w1[8];
    tc_ld8_nowait(w0addr + 8 * p, w0);
    tc_ld8_nowait(w0addr + (kTmemW1 - kTmemW0) + 8 * p, w1);
    tc_wait_ld();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const DirectCol c = t.cols[8 * p + j];
      const long long v = (long long)(((unsigned long long)w1[j] << 32) | w0[j]);
      double x = i64_scaled_to_double(v, t.ebase + c.F, a.mode & 2);
      if (t.nonfinite || c.F == kNonFiniteExp) x = __longlong_as_double(0x7FF8000000000000ll);
      if (t.mlive && c.colp) c.colp[t.roff] = acc ? dc[j] + x : x;
    }
  }
}

// Energy form, after the last chunk of a tile's last level: the same rounding
// of the 32 exact sums as store_direct, then per element (nothing stored)
//     acc += x * fl(x / eps),   eps = fl(prefix - e_last)
// in FP64: the prefix is the denominator chain without its last term, formed
// on the host in the reference's order; the quotient is the exactly rounded
// FP64 quotient (div_rn); zeros add nothing and skip the division.  A
// non-finite operand value in the row or column makes x (and the sum) NaN.
// Every lane of the warp runs the TMEM loads (.sync.aligned: the whole warp
// together); rows outside the block are skipped per element.
__device__ __forceinline__ void energy_direct(const OzGemmArgs& a, const DirectTile& t, uint32_t w0addr,
                                              double& acc) {
#pragma unroll 1
  for (int p = 0; p < 4; ++p) {
    uint32_t w0[8], w1[8];
    tc_ld8_nowait(w0addr + 8 * p, w0);
    tc_ld8_nowait(w0addr + (kTmemW1 - kTmemW0) + 8 * p, w1);
    tc_wait_ld();
#pragma unroll
    for (int j0 = 0; j0 < 8; j0 += 2) {  // two elements at a time without a branch between them
      double x[2], qv[2];
      bool ok[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int j = j0 + i, F = t.cols[8 * p + j].F;
        const EnergyCol ec = t.ecols[8 * p + j];
        const long long v = (long long)(((unsigned long long)w1[j] << 32) | w0[j]);
        ok[i] = i64_scaled_normal(v, t.ebase + F, &x[i]);
        const double eps = __dsub_rn(t.prow[max(ec.ck, 0)], t.last_row ? t.er : ec.ec);
        ok[i] = div_rn_int(x[i], eps, &qv[i]) && ok[i] && t.mlive && ec.ck >= 0 && !t.nonfinite && F != kNonFiniteExp;
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (ok[i]) {
          acc = fma(x[i], qv[i], acc);
          continue;
        }
        const int j = j0 + i, F = t.cols[8 * p + j].F;
        const EnergyCol ec = t.ecols[8 * p + j];
        if (!t.mlive || ec.ck < 0) continue;
        double y = i64_scaled_to_double((long long)(((unsigned long long)w1[j] << 32) | w0[j]), t.ebase + F, false);
        if (t.nonfinite || F == kNonFiniteExp) y = __longlong_as_double(0x7FF8000000000000ll);
        if (!nonzero(y)) continue;
        acc = fma(y, div_rn(y, __dsub_rn(t.prow[ec.ck], t.last_row ? t.er : ec.ec)), acc);
      }
    }
  }
}

// Eight warps, two per TMEM lane quadrant (warp % 4); each thread owns one
// accumulator row and 64 of its 128 columns, in two groups of 32.  The three
// TMEM loads of a group (chunk, hi, lo) are issued before one wait.  In the
// pair form each CTA drains its own 128 rows and signals the leader.
//
// Direct form: the running sum of a tile is the exact integer
//     sum_t S_t * 256^(slices-1-t)
// (Horner over the levels t, which arrive in order), kept as two 32-bit
// TMEM words per element; the host admits a batch to this form only when the
// sum stays below 2^63.  The last chunk of the last level is rounded once and
// stored into D.
template <bool PAIR, bool DIRECT, bool ENERGY = false>
__device__ void epilogue(const OzGemmArgs& a, OzSmemT<PAIR, 128>& sm, uint32_t tmem, int warp, int lane,
                         uint32_t rank) {
  constexpr int kRows = PAIR ? 2 * kOzBM : kOzBM;  // rows of a tile
  constexpr int kCols = DIRECT ? 32 : 64;          // columns of a thread
  const int q = warp & 3, h = (warp - 2) >> 2;
  const int row = int(rank) * kOzBM + 32 * q + lane;
  const uint32_t lane_addr = tmem + (uint32_t(32 * q) << 16) + uint32_t(kCols * h);
  uint32_t empty_bar[2];
  for (int b = 0; b < 2; ++b) empty_bar[b] = PAIR ? mapa_shared(&sm.acc_empty[b], 0) : smem_u32(&sm.acc_empty[b]);
  uint32_t chunk = 0;
  [[maybe_unused]] DirectTile dt{};
  [[maybe_unused]] double eacc = 0.0;
  if constexpr (DIRECT) {
    __shared__ DirectCol direct_cols[kThreadsOzDirect / 32 - 2][32];  // one table per epilogue warp
    dt.cols = direct_cols[warp - 2];
    if constexpr (ENERGY) {
      __shared__ EnergyCol energy_cols[kThreadsOzDirect / 32 - 2][32];
      dt.ecols = energy_cols[warp - 2];
    }
  }
  auto release = [&](uint32_t buf) {
    tc_fence_before();
    __syncwarp();
    if (lane == 0) {
      if constexpr (PAIR) mbar_arrive_cluster(empty_bar[buf]);
      else mbar_arrive(&sm.acc_empty[buf]);
    }
  };
  for_units<PAIR>(a, [&](int u) {
    const OzUnit un = a.units[u];
    const int ckb = a.chunk_kb[un.level];
    const int nchunks = (un.kb_end - un.kb_begin + ckb - 1) / ckb;
    if constexpr (DIRECT) {
      const bool last_level = un.level == a.slices - 1;
      if (un.level == 0) {
        direct_tile<ENERGY>(dt, a, a.tiles[un.tile], row, kCols * h, lane);
        if constexpr (!ENERGY)
          if ((a.mode & 1) && !a.dry) prefetch_direct(dt);
      }
      for (int c = 0; c < nchunks; ++c) {
        const uint32_t buf = chunk & 1;
        if (!mbar_wait(&sm.acc_full[buf], (chunk >> 1) & 1, sm, a.err_flag, 4)) return false;
        tc_fence_after();
        const bool fresh = c == 0 && un.level == 0;  // no running sum yet
        const uint32_t mul = c == 0 ? 256u : 1u;     // a new level: running sum * 256
        const bool final = last_level && c == nchunks - 1;
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {
          uint32_t x[8], w0[8], w1[8];
          tc_ld8_nowait(lane_addr + buf * kOzBN + 8 * g, x);
          if (!fresh) {
            tc_ld8_nowait(lane_addr + kTmemW0 + 8 * g, w0);
            tc_ld8_nowait(lane_addr + kTmemW1 + 8 * g, w1);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) w0[j] = w1[j] = 0u;
          }
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            // (w1:w0) * mul + x modulo 2^64 in 32-bit multiply-adds (x is an
            // integer below 2^24, exact in FP32): low word with its carry, then
            // the high word
            const unsigned long long lo =
                (unsigned long long)w0[j] * mul + (unsigned long long)(long long)__float2int_rz(__uint_as_float(x[j]));
            w0[j] = uint32_t(lo);
            w1[j] = w1[j] * mul + uint32_t(lo >> 32);
          }
          tc_st8(lane_addr + kTmemW0 + 8 * g, w0);
          tc_st8(lane_addr + kTmemW1 + 8 * g, w1);
        }
        tc_wait_st();
        release(buf);  // the next MMAs may start while this thread stores D
        ++chunk;
        if (final) {
          if constexpr (ENERGY) energy_direct(a, dt, lane_addr + kTmemW0, eacc);
          else store_direct(a, dt, lane_addr + kTmemW0);
        }
      }
      return true;
    } else {
    int* w = a.ws + ((size_t(un.tile) * a.slices + un.level) * a.nsplit + un.split) * kOzBN * kRows +
             size_t(64 * h) * kRows + row;
    if (nchunks == 0) {  // empty k range: its partial sum is zero
#pragma unroll 8
      for (int j = 0; j < 64; ++j) w[size_t(j) * kRows] = 0;
      return true;
    }
    for (int c = 0; c < nchunks; ++c) {
      const uint32_t buf = chunk & 1;
      if (!mbar_wait(&sm.acc_full[buf], (chunk >> 1) & 1, sm, a.err_flag, 4)) return false;
      tc_fence_after();
      const bool first = c == 0, last = c == nchunks - 1;
#pragma unroll 1
      for (int g = 0; g < 2; ++g) {
        uint32_t x[32], hi[32], lo[32];
        tc_ld32_nowait(lane_addr + buf * kOzBN + 32 * g, x);
        if (!first) {
          tc_ld32_nowait(lane_addr + kTmemHi + 32 * g, hi);
          tc_ld32_nowait(lane_addr + kTmemLo + 32 * g, lo);
        }
        tc_wait_ld();
        if (first) {
#pragma unroll
          for (int j = 0; j < 32; ++j) hi[j] = x[j], lo[j] = 0u;
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            float hv = __uint_as_float(hi[j]), lv = __uint_as_float(lo[j]);
            two_sum_acc(hv, lv, __uint_as_float(x[j]));
            hi[j] = __float_as_uint(hv), lo[j] = __float_as_uint(lv);
          }
        }
        if (!last) {
          tc_st32(lane_addr + kTmemHi + 32 * g, hi);
          tc_st32(lane_addr + kTmemLo + 32 * g, lo);
        } else {
          // hi + lo is the unit's exact level sum, an integer below 2^31 (the
          // host sizes units for that), stored as int32
#pragma unroll
          for (int j = 0; j < 32; ++j)
            w[size_t(32 * g + j) * kRows] =
                int(static_cast<long long>(__uint_as_float(hi[j])) + static_cast<long long>(__uint_as_float(lo[j])));
        }
      }
      if (!last) tc_wait_st();
      release(buf);
      ++chunk;
    }
    return true;
    }
  });
  if constexpr (ENERGY) a.epart[(size_t(blockIdx.x) * 16 + size_t(warp - 2)) * 32 + lane] = eacc;
}

// 256-column tiles: the two FP32 accumulators use all 512 TMEM columns, so the
// exact running level sum of a unit lives in registers as int32 (a unit's
// level sum is an integer below 2^31 and every chunk value below 2^24, so the
// conversion and the additions are exact).  Eight warps, two per lane
// quadrant; each thread owns one row and 128 columns, read 16 at a time.
template <bool PAIR>
__device__ void epilogue_int(const OzGemmArgs& a, OzSmemT<PAIR, 256>& sm, uint32_t tmem, int warp, int lane,
                             uint32_t rank) {
  constexpr int BN = 256;
  constexpr int kRows = PAIR ? 2 * kOzBM : kOzBM;
  const int q = warp & 3, h = (warp - 2) >> 2;
  const int row = int(rank) * kOzBM + 32 * q + lane;
  const uint32_t lane_addr = tmem + (uint32_t(32 * q) << 16) + uint32_t(128 * h);
  uint32_t empty_bar[2];
  for (int b = 0; b < 2; ++b) empty_bar[b] = PAIR ? mapa_shared(&sm.acc_empty[b], 0) : smem_u32(&sm.acc_empty[b]);
  uint32_t chunk = 0;
  for_units<PAIR>(a, [&](int u) {
    const OzUnit un = a.units[u];
    const int ckb = a.chunk_kb[un.level];
    const int nchunks = (un.kb_end - un.kb_begin + ckb - 1) / ckb;
    int* w = a.ws + ((size_t(un.tile) * a.slices + un.level) * a.nsplit + un.split) * BN * kRows +
             size_t(128 * h) * kRows + row;
    int sum[128];
#pragma unroll
    for (int j = 0; j < 128; ++j) sum[j] = 0;
    for (int c = 0; c < nchunks; ++c) {
      const uint32_t buf = chunk & 1;
      if (!mbar_wait(&sm.acc_full[buf], (chunk >> 1) & 1, sm, a.err_flag, 4)) return false;
      tc_fence_after();
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        uint32_t x[16];
        tc_ld16_nowait(lane_addr + buf * BN + 16 * g, x);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) sum[16 * g + j] += __float2int_rz(__uint_as_float(x[j]));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) mbar_arrive_cluster(empty_bar[buf]);
        else mbar_arrive(&sm.acc_empty[buf]);
      }
      ++chunk;
    }
#pragma unroll
    for (int j = 0; j < 128; ++j) w[size_t(j) * kRows] = sum[j];
    return true;
  });
}

// Residue form, every tile shape: a chunk (256 k) of the modulus' product is an
// exact FP32 integer below 2^24 - 256; the thread's running residue (at most 256
// in magnitude: p / 2, or one multiple of p off where the reciprocal's error
// meets a tie; one FP32 register per column) is added to it, exactly, and the
// sum reduced modulo p again: four packed FP32 instructions per two
// columns.  (The conversion to int32 that the level form uses runs at a
// quarter of the FP32 rate's 128 per clock and would take as long as the
// chunk's MMAs: 2048 clocks for a 128 x 256 accumulator.)  A chunk has to be
// drained within the next one's MMAs: the pair 256 x 256 form keeps its tensor
// pipe 90 % busy (95 % with the drain left out; sixteen epilogue warps instead
// of eight, with loads of eight columns in flight, measured the same).  Stored
// as the non-negative int16 r + kOzResidueBias.
template <bool PAIR, int BN>
__device__ void epilogue_residue(const OzGemmArgs& a, OzSmemT<PAIR, BN>& sm, uint32_t tmem, int warp, int lane,
                                 uint32_t rank) {
  constexpr int kRows = PAIR ? 2 * kOzBM : kOzBM;
  constexpr int kCols = BN / 2;  // columns of a thread
  const int q = warp & 3, h = (warp - 2) >> 2;
  const int row = int(rank) * kOzBM + 32 * q + lane;
  const uint32_t lane_addr = tmem + (uint32_t(32 * q) << 16) + uint32_t(kCols * h);
  uint32_t empty_bar[2];
  for (int b = 0; b < 2; ++b) empty_bar[b] = PAIR ? mapa_shared(&sm.acc_empty[b], 0) : smem_u32(&sm.acc_empty[b]);
  const F32x2 magic = pack2(kRintMagic, kRintMagic), unmagic = pack2(-kRintMagic, -kRintMagic);
  const F32x2 biased = pack2(kRintMagic + kOzResidueBias, kRintMagic + kOzResidueBias);
  uint32_t chunk = 0;
  for_units<PAIR>(a, [&](int u) {
    const OzUnit un = a.units[u];
    const int nchunks = (un.kb_end - un.kb_begin + kOzResidueChunkKb - 1) / kOzResidueChunkKb;
    const float p = a.res_p[un.level], ip = a.res_inv[un.level];
    const F32x2 inv = pack2(ip, ip), np = pack2(-p, -p);
    int16_t* w = reinterpret_cast<int16_t*>(a.ws) +
                 ((size_t(un.tile) * a.slices + un.level) * a.nsplit + un.split) * BN * kRows +
                 size_t(kCols * h) * kRows + row;
    F32x2 r[kCols / 2];
#pragma unroll
    for (int j = 0; j < kCols / 2; ++j) r[j] = 0ull;  // two +0
    for (int c = 0; c < nchunks; ++c) {
      const uint32_t buf = chunk & 1;
      if (!mbar_wait(&sm.acc_full[buf], (chunk >> 1) & 1, sm, a.err_flag, 4)) return false;
      tc_fence_after();
      uint32_t xg[16];
#pragma unroll
      for (int g = 0; g < kCols / 16; ++g) {
        tc_ld16_nowait(lane_addr + buf * BN + 16 * g, xg);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const F32x2 y = add2(pack2(__uint_as_float(xg[2 * j]), __uint_as_float(xg[2 * j + 1])), r[8 * g + j]);
          r[8 * g + j] = fma2(np, add2(fma2(y, inv, magic), unmagic), y);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) mbar_arrive_cluster(empty_bar[buf]);
        else mbar_arrive(&sm.acc_empty[buf]);
      }
      ++chunk;
    }
#pragma unroll
    for (int j = 0; j < kCols / 2; ++j) {
      float lo, hi;
      unpack2(add2(r[j], biased), lo, hi);  // the low 16 bits of 1.5 2^23 + x are x
      w[size_t(2 * j) * kRows] = int16_t(__float_as_uint(lo));
      w[size_t(2 * j + 1) * kRows] = int16_t(__float_as_uint(hi));
    }
    return true;
  });
}

template <bool PAIR, int BN, bool DIRECT = false, bool ENERGY = false, bool RES = false>
__global__ void __launch_bounds__(DIRECT ? kThreadsOzDirect : kThreadsOz, 1)
    oz_gemm_kernel(const __grid_constant__ OzGemmArgs a) {
  using SM = OzSmemT<PAIR, BN>;
  extern __shared__ uint8_t smem_raw[];
  SM& sm = *reinterpret_cast<SM*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_rank() : 0u;
  if (threadIdx.x == 0) {
    for (int s = 0; s < SM::kSt; ++s) {
      mbar_init(&sm.full[s], PAIR ? 2 : 1);  // pair form: one expect_tx arrive from each CTA
      mbar_init(&sm.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.acc_full[b], 1);
      // one arrive per epilogue warp (of both CTAs)
      mbar_init(&sm.acc_empty[b], (DIRECT ? 16 : 8) * (PAIR ? 2 : 1));
    }
    mbar_init(&sm.drain, 1);
    sm.abort = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(&sm.tmem_base)),
                   "r"(kTmemCols));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(&sm.tmem_base)),
                   "r"(kTmemCols));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync();  // the peer's barriers exist before anyone signals them
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp == 0) {
    producer<PAIR, BN, RES>(a, sm, rank);
  } else if (warp == 1) {
    if (rank == 0) {
      mma_issuer<PAIR, BN, RES>(a, sm, tmem);
      // all MMAs this warp issued have completed before TMEM is released
      if (elect_one()) {
        if constexpr (PAIR) tc_commit_pair(&sm.drain);
        else tc_commit(&sm.drain);
      }
      __syncwarp();
      warp_wait(smem_u32(&sm.drain), 0, sm, a.err_flag, 5);
    }
  } else {
    if constexpr (RES) epilogue_residue<PAIR, BN>(a, sm, tmem, warp, lane, rank);
    else if constexpr (BN == 256) epilogue_int<PAIR>(a, sm, tmem, warp, lane, rank);
    else epilogue<PAIR, DIRECT, ENERGY>(a, sm, tmem, warp, lane, rank);
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync();  // the leader's MMAs have read this CTA's smem and TMEM
  if (warp == 1) {
    tc_fence_after();
    if constexpr (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
  }
}

// ------------------------------------------------------------------ all levels at once
// Form of the direct GEMM for sub-problems whose k range fits one exact FP32
// flush per level (at most 5 slices, k at most 320): every level accumulator
// of a 128 x 64 tile lives in TMEM at once (levels 0-2 one each; levels 3 and
// 4, whose sums over 320 k could pass 2^24, one per half of the k range:
// 7 x 64 = 448 columns).  Each 32-wide k block of the tile's S A-slices and S
// B-slices is loaded once (one 3-D copy per operand) for all S (S + 1) / 2
// slice pairs, where the level-by-level form loads two tiles per pair.
// A slice i multiplies B slices 0, 1, ... into levels i, i + 1, ...: B slices
// lie one after another in shared memory (rows of one taller operand) and the
// levels' accumulators side by side in TMEM, so one MMA of up to 256 columns
// covers up to four slice pairs and reads A slice i from shared memory once
// for all of them: 6 MMAs (8 in the second half of the k range) and 54 KB (62)
// of operand reads per 16 k instead of 15 MMAs of 64 columns and 90 KB.  When
// the tile's MMAs complete, the epilogue reads each accumulator once, forms
// the exact sum over levels (the same 64-bit integer as the level-by-level
// Horner sum) in registers and releases TMEM before it rounds and divides,
// sums or stores: the tensor cores run the next tile meanwhile.
constexpr int kLvBN = 64, kLvBK = 32, kLvMaxS = 5, kLvSt = 3, kLvAcc = 7;
constexpr uint32_t kLvATile = kOzBM * kLvBK * 2;  // 8 KB: 128 rows x 32 k
constexpr uint32_t kLvBTile = kLvBN * kLvBK * 2;  // 4 KB: 64 columns x 32 k
// What the epilogue needs of a tile's rows and columns, laid out by the
// producer warp while the tensor cores work on the tile: the chain of loads to
// it (tile, panel and block, tables) is not in the sixteen epilogue warps' way.
// (In their way it took, per step: o=24/v=240 with energy 17.8 ms instead of
// 17.0, o=12/v=63 stored 459 us instead of 410, a third of that from rounding
// eight results without a branch.)
struct LvTab {
  double rx[kOzBM];      // energy form: the row's last-term orbital energy
  long long rp[kOzBM];   // energy: the row's line of the prefix table; store: its offset in D
  double cx[kLvBN];      // energy form: the column's last-term orbital energy
  long long cp[kLvBN];   // energy: the column in that line (-1: outside D); store: its base in D (0: outside)
  int re[kOzBM];         // biased row exponent (at least 1; 0: outside D)
  int cf[kLvBN];         // biased column exponent (at least 1)
  int flag;              // energy: the last term runs over the rows; store: D is unit-stride along the columns
};
struct __align__(1024) LvSmem {
  uint8_t a[kLvSt][kLvMaxS][kLvATile];
  uint8_t b[kLvSt][kLvMaxS][kLvBTile];
  uint64_t full[kLvSt], empty[kLvSt];
  uint64_t acc_full, acc_empty, drain;
  uint64_t tab_full[2], tab_empty[2];
  LvTab tab[2];
  uint32_t tmem_base;
  volatile int abort;
  double out[kThreadsOzDirect / 32 - 2][32][9];  // per epilogue warp: 32 rows x 8 columns on their way to D
};
static_assert(sizeof(LvSmem) + 1024 <= 232448, "one CTA's shared memory");
static_assert(kLvBN == kOzLevelsTileCols, "tile columns of the all-levels form");
// TMEM accumulator (in 64-column units) of level t; levels 3 and 4: of k half
// h.  The levels of each half lie side by side: 0 1 2 3 4 | 3' 4'.
__device__ __forceinline__ int lv_acc(int t, int h) { return t + (t >= 3 && h ? 2 : 0); }

// Shared-memory matrix descriptor: K-major, 64-byte swizzle, rows of 64 B,
// 8-row core groups 512 B apart; `lo` as sw128_desc_lo.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t lo) {
  constexpr uint32_t hi = uint32_t(512 >> 4) | (1u << 14) | (4u << 29);  // SBO, version 1, SWIZZLE_64B
  return (uint64_t(hi) << 32) | lo;
}

// Per 32-wide k block of a tile, one stage: the S A-slices (rows m0..m0+127)
// and the S B-slices (columns n0..n0+63).  Converged warp, one lane issues.
// Then the tile's tables.
template <bool ENERGY>
__device__ void lv_producer(const OzGemmArgs& a, LvSmem& sm, int lane) {
  const uint32_t bytes = uint32_t(a.slices) * (kLvATile + kLvBTile);
  const bool leader = elect_one();
  const uint32_t a0 = smem_u32(sm.a[0][0]), b0 = smem_u32(sm.b[0][0]);
  const uint32_t full0 = smem_u32(&sm.full[0]), empty0 = smem_u32(&sm.empty[0]);
  uint32_t s = 0, free_parity = 1, nt = 0;
  for (int g = int(blockIdx.x); g < a.n_tiles; g += int(gridDim.x), ++nt) {
    const OzTile tl = a.tiles[g];
    const void* ma = static_cast<const uint8_t*>(a.maps_a) + size_t(tl.panel_a) * 128;
    const void* mb = static_cast<const uint8_t*>(a.maps_b) + size_t(tl.panel_b) * 128;
    const int *exps_a = a.panels_a[tl.panel_a].exps, *exps_b = a.panels_b[tl.panel_b].exps;
    const OzDBlock db = a.dblocks[tl.dblock];
    [[maybe_unused]] OzEnergyBlock eb{};
    if constexpr (ENERGY) eb = a.eblocks[tl.dblock];
    for (int q = tl.trip_begin; q < tl.trip_end; ++q) {
      const OzTrip tr = a.trips[q];
      int ka = int(tr.koff_a), kb = int(tr.koff_b);
      for (int j = 0; j < 2 * tr.nkb; ++j, ka += kLvBK, kb += kLvBK) {
        if (!warp_wait(empty0 + 8 * s, free_parity, sm, a.err_flag, 1)) return;
        if (leader) {
          const uint32_t fb = full0 + 8 * s;
          mbar_expect_tx(fb, bytes);
          tma_load_3d(a0 + s * (kLvMaxS * kLvATile), ma, fb, ka, tl.m0, 0);
          tma_load_3d(b0 + s * (kLvMaxS * kLvBTile), mb, fb, kb, tl.n0, 0);
        }
        __syncwarp();
        if (++s == uint32_t(kLvSt)) s = 0, free_parity ^= 1;
      }
    }
    const uint32_t slot = nt & 1;
    if (!warp_wait(smem_u32(&sm.tab_empty[slot]), ((nt >> 1) & 1) ^ 1, sm, a.err_flag, 1)) return;
    LvTab& t = sm.tab[slot];
#pragma unroll
    for (int i = 0; i < kOzBM / 32; ++i) {
      const int row = 32 * i + lane, m = tl.m0 + row;
      int e = 0;
      long long p = ENERGY ? reinterpret_cast<long long>(eb.ptab) : 0;  // rows outside read (and drop) the first line
      double x = 0.0;
      if (m < db.M) {
        e = max(exps_a[m], 1);
        if constexpr (ENERGY) {
          p = reinterpret_cast<long long>(eb.ptab + int64_t(eb.rk[m]) * eb.ckn);
          if (eb.last_row) x = eb.elast[m];
        } else {
          p = db.rowoff[m];
        }
      }
      t.re[row] = e, t.rp[row] = p, t.rx[row] = x;
    }
#pragma unroll
    for (int i = 0; i < kLvBN / 32; ++i) {
      const int col = 32 * i + lane, n = tl.n0 + col;
      int f = 1;
      long long p = ENERGY ? -1 : 0;
      double x = 0.0;
      if (n < db.N) {
        f = max(exps_b[n], 1);
        if constexpr (ENERGY) {
          p = eb.ck[n];
          if (!eb.last_row) x = eb.elast[n];
        } else {
          p = reinterpret_cast<long long>(db.colptr[n]);
        }
      }
      t.cf[col] = f, t.cp[col] = p, t.cx[col] = x;
    }
    if (lane == 0) t.flag = ENERGY ? eb.last_row : db.col_fast;
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.tab_full[slot]);
  }
}

// One MMA (16 k) of 64 * levels columns.
__device__ __forceinline__ void lv_mma_one(uint32_t d, uint32_t ad, uint32_t bd, int levels, uint32_t acc) {
  const uint32_t idesc = idesc_bf16<128, 0>() | (uint32_t(levels) << 20);  // N >> 3 = 8 * levels at bit 17
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(sw64_desc(ad)), "l"(sw64_desc(bd)), "r"(idesc), "r"(acc));
}

// The MMAs of one 16-k step of S slices: A slice i against B slices j into
// levels i + j < S, as few and as wide as the accumulators' order allows
// (second half of the k range: levels 3 and 4 have accumulators of their own).
// acc_lo / acc_hi: 0 where the first MMA into levels 0-2 / 3-4 overwrites.
template <int S, bool SECOND>
__device__ __forceinline__ void lv_step(uint32_t tmem, uint32_t ad, uint32_t bd, uint32_t acc_lo, uint32_t acc_hi) {
  constexpr uint32_t kA = kLvATile >> 4, kB = kLvBTile >> 4;
#pragma unroll
  for (int i = 0; i < S; ++i) {
    const uint32_t ai = ad + uint32_t(i) * kA;
    if constexpr (!SECOND) {
      const int n = S - i < 4 ? S - i : 4;  // levels i .. i + n - 1: at most 256 columns
      lv_mma_one(tmem + uint32_t(kLvBN * i), ai, bd, n, i == 0 ? acc_lo : 1u);
      if (n < S - i) lv_mma_one(tmem + uint32_t(kLvBN * (i + n)), ai, bd + uint32_t(n) * kB, S - i - n, i == 0 ? acc_hi : 1u);
    } else {
      const int lo = (S < 3 ? S : 3) - i;  // levels i .. 2
      if (lo > 0) lv_mma_one(tmem + uint32_t(kLvBN * i), ai, bd, lo, i == 0 ? acc_lo : 1u);
      const int t = i > 3 ? i : 3;         // levels t .. S - 1
      if (S - t > 0)
        lv_mma_one(tmem + uint32_t(kLvBN * (t + 2)), ai, bd + uint32_t(t - i) * kB, S - t, i == 0 ? acc_hi : 1u);
    }
  }
}

// The tile's 2 kb_total 32-wide k blocks in two equal halves (at most 160 k
// each); the first MMA into an accumulator overwrites it.  Converged warp, one
// lane issues.
template <int S>
__device__ void lv_mma(const OzGemmArgs& a, LvSmem& sm, uint32_t tmem) {
  const bool leader = elect_one();
  const uint32_t full0 = smem_u32(&sm.full[0]), empty0 = smem_u32(&sm.empty[0]);
  const uint32_t acc_full = smem_u32(&sm.acc_full), acc_empty = smem_u32(&sm.acc_empty);
  const uint32_t ad0 = sw128_desc_lo(sm.a[0][0]), bd0 = sw128_desc_lo(sm.b[0][0]);
  uint32_t s = 0, full_parity = 0, free_parity = 1;
  for (int g = int(blockIdx.x); g < a.n_tiles; g += int(gridDim.x)) {
    const int half = a.tiles[g].kb_total;
    if (!warp_wait(acc_empty, free_parity, sm, a.err_flag, 2)) return;
    free_parity ^= 1;
    tc_fence_after();
    for (int kb = 0; kb < 2 * half; ++kb) {
      if (!warp_wait(full0 + 8 * s, full_parity, sm, a.err_flag, 3)) return;
      tc_fence_after();
      if (leader) {
        const uint32_t ad = ad0 + s * (kLvMaxS * kLvATile >> 4), bd = bd0 + s * (kLvMaxS * kLvBTile >> 4);
        if (kb < half) {
          const uint32_t acc = kb == 0 ? 0u : 1u;
          lv_step<S, false>(tmem, ad, bd, acc, acc);
          lv_step<S, false>(tmem, ad + 2, bd + 2, 1u, 1u);  // the block's second 16 k: 32 B further
        } else {
          lv_step<S, true>(tmem, ad, bd, 1u, kb == half ? 0u : 1u);
          lv_step<S, true>(tmem, ad + 2, bd + 2, 1u, 1u);
        }
        tc_commit(empty0 + 8 * s);
        if (kb + 1 == 2 * half) tc_commit(acc_full);
      }
      __syncwarp();
      if (++s == uint32_t(kLvSt)) s = 0, full_parity ^= 1;
    }
  }
}

constexpr int kLvGroup = 4;  // elements whose energy work overlaps

// Sixteen warps, four per TMEM lane quadrant; a thread owns one row and 16
// columns.  Per tile: the wait for the tile's tables and MMAs, the exact sums (two groups of 8 columns, each
// accumulator read once), TMEM released, then per element the rounding to
// FP64 with the row and column scales and
//   energy form: acc += x * fl(x / eps), eps = fl(prefix - e_last)
//   (the chain without its last term tabulated in the reference's order; the
//   quotient exactly rounded; zeros add nothing);
//   store form: D = x or D += x.
// A non-finite operand value in the row or column makes x NaN.
template <bool ENERGY, int S>
__device__ void lv_epilogue(const OzGemmArgs& a, LvSmem& sm, uint32_t tmem, int warp, int lane) {
  const int q = warp & 3, h = (warp - 2) >> 2;
  const int row = 32 * q + lane;
  const uint32_t lane_addr = tmem + (uint32_t(32 * q) << 16) + uint32_t(16 * h);
  // 256^t, hidden from the compiler: a level joins the sum with one 32 x 32 + 64
  // bit multiply-add instead of five shifts and additions
  int weight[4];
  asm volatile("mov.b32 %0, 1;\n\tmov.b32 %1, 256;\n\tmov.b32 %2, 65536;\n\tmov.b32 %3, 16777216;"
               : "=r"(weight[0]), "=r"(weight[1]), "=r"(weight[2]), "=r"(weight[3]));
  [[maybe_unused]] double eacc = 0.0;
  uint32_t nt = 0;
  for (int g = int(blockIdx.x); g < a.n_tiles; g += int(gridDim.x), ++nt) {
    const uint32_t slot = nt & 1;
    if (!mbar_wait(&sm.tab_full[slot], (nt >> 1) & 1, sm, a.err_flag, 4)) break;
    const LvTab& t = sm.tab[slot];
    const int re = t.re[row];
    const bool mlive = re != 0, nonfinite = re == kNonFiniteExp, flag = t.flag != 0;
    const int ebase = max(re, 1) - 1022 - 1022 + 2 - kDigitBits * (S + 1);
    const int* cf = t.cf + 16 * h;
    const long long* cp = t.cp + 16 * h;
    if (!mbar_wait(&sm.acc_full, nt & 1, sm, a.err_flag, 4)) break;
    tc_fence_after();
    long long sum[16];
#pragma unroll
    for (int gg = 0; gg < 2; ++gg) {
      uint32_t v[kLvAcc][8];
#pragma unroll
      for (int c = 0; c < kLvAcc; ++c) tc_ld8_nowait(lane_addr + uint32_t(kLvBN * c + 8 * gg), v[c]);
      tc_wait_ld();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        // sum_t S_t 256^(S-1-t), S_t an integer below 2^24 in FP32 (levels
        // 3 and 4: the sum of the two halves)
        long long r = 0;
#pragma unroll
        for (int t = 0; t < S; ++t) {
          int st = __float2int_rz(__uint_as_float(v[lv_acc(t, 0)][j]));
          if (t >= 3) st += __float2int_rz(__uint_as_float(v[lv_acc(t, 1)][j]));
          if (S - 1 - t == 4) r = (long long)((unsigned long long)uint32_t(st) << 32);
          else asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(r) : "r"(st), "r"(weight[S - 1 - t]));
        }
        sum[8 * gg + j] = r;
      }
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.acc_empty);  // the next tile's MMAs may start
    if constexpr (ENERGY) {
      // groups of kLvGroup elements without a branch between them, so that
      // their conversions, denominators and divisions overlap; zeros, dead rows
      // and columns, non-finite rows and results beyond the normal range are
      // done one by one afterwards
      const double* prow = reinterpret_cast<const double*>(t.rp[row]);
      const double er = t.rx[row];
      const double* ec = t.cx + 16 * h;
#pragma unroll
      for (int j0 = 0; j0 < 16; j0 += kLvGroup) {
        double x[kLvGroup], qv[kLvGroup];
        bool ok[kLvGroup], all = mlive && !nonfinite;
#pragma unroll
        for (int i = 0; i < kLvGroup; ++i) {
          const int F = cf[j0 + i], ck = int(cp[j0 + i]);
          ok[i] = i64_scaled_normal(sum[j0 + i], ebase + F, &x[i]);
          const double eps = __dsub_rn(prow[max(ck, 0)], flag ? er : ec[j0 + i]);
          ok[i] = div_rn_int(x[i], eps, &qv[i]) && ok[i] && ck >= 0 && F != kNonFiniteExp;
          all = all && ok[i];
        }
        if (all) {
#pragma unroll
          for (int i = 0; i < kLvGroup; ++i) eacc = fma(x[i], qv[i], eacc);
        } else if (mlive) {
#pragma unroll
          for (int i = 0; i < kLvGroup; ++i) {
            if (ok[i] && !nonfinite) {
              eacc = fma(x[i], qv[i], eacc);
              continue;
            }
            const int F = cf[j0 + i], ck = int(cp[j0 + i]);
            if (ck < 0) continue;
            double y = i64_scaled_to_double(sum[j0 + i], ebase + F, false);
            if (nonfinite || F == kNonFiniteExp) y = __longlong_as_double(0x7FF8000000000000ll);
            if (!nonzero(y)) continue;
            eacc = fma(y, div_rn(y, __dsub_rn(prow[ck], flag ? er : ec[j0 + i])), eacc);
          }
        }
      }
    } else {
      const bool acc = a.mode & 1, neg = a.mode & 2;
      const long long roff = t.rp[row];
      double(*buf)[9] = sm.out[warp - 2];
#pragma unroll
      for (int h8 = 0; h8 < 2; ++h8) {
        // eight roundings without a branch between them; results beyond the
        // normal range one by one afterwards
        double x[8];
        uint32_t slow = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const long long v = sum[8 * h8 + j];
          const int F = cf[8 * h8 + j];
          const bool ok = i64_scaled_normal(v, ebase + F, &x[j]) || v == 0;
          if (v == 0) x[j] = 0.0;
          x[j] = __longlong_as_double(__double_as_longlong(x[j]) ^ (neg ? (1ll << 63) : 0ll));
          if (nonfinite || F == kNonFiniteExp) x[j] = __longlong_as_double(0x7FF8000000000000ll);
          else if (!ok) slow |= 1u << j;
        }
        if (slow) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (slow >> j & 1) x[j] = i64_scaled_to_double(sum[8 * h8 + j], ebase + cf[8 * h8 + j], neg);
        }
        if (!flag) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            double* p = reinterpret_cast<double*>(cp[8 * h8 + j]);
            if (mlive && p) p[roff] = acc ? p[roff] + x[j] : x[j];
          }
          continue;
        }
        // D runs along the columns: the warp's 32 x 8 results turn in shared
        // memory, so that a store covers four rows of 64 contiguous bytes
        // instead of 32 rows of one element each, 32 cycles of the load / store
        // unit per instruction (o=12/v=63 step, 413 MB of W: 666 -> 459 us;
        // rows that are contiguous already store directly)
#pragma unroll
        for (int j = 0; j < 8; ++j) buf[lane][j] = x[j];
        __syncwarp();
        const int c = lane & 7;
        double* base = reinterpret_cast<double*>(cp[8 * h8 + c]);
        double* p[8];
        double old[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int rr = 32 * q + 4 * i + (lane >> 3);
          p[i] = base && t.re[rr] ? base + t.rp[rr] : nullptr;
          old[i] = acc && p[i] ? *p[i] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const double y = buf[4 * i + (lane >> 3)][c];
          if (p[i]) *p[i] = acc ? old[i] + y : y;
        }
        __syncwarp();
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.tab_empty[slot]);
  }
  if constexpr (ENERGY) a.epart[(size_t(blockIdx.x) * 16 + size_t(warp - 2)) * 32 + lane] = eacc;
}

template <bool ENERGY, int S>
__global__ void __launch_bounds__(kThreadsOzDirect, 1) oz_levels_kernel(const __grid_constant__ OzGemmArgs a) {
  extern __shared__ uint8_t smem_raw[];
  LvSmem& sm = *reinterpret_cast<LvSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kLvSt; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    mbar_init(&sm.acc_full, 1);
    mbar_init(&sm.acc_empty, 16);  // one arrive per epilogue warp
    mbar_init(&sm.drain, 1);
    for (int s = 0; s < 2; ++s) mbar_init(&sm.tab_full[s], 1), mbar_init(&sm.tab_empty[s], 16);
    sm.abort = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  if (warp == 0) {
    lv_producer<ENERGY>(a, sm, lane);
  } else if (warp == 1) {
    lv_mma<S>(a, sm, tmem);
    if (elect_one()) tc_commit(&sm.drain);  // all MMAs of this warp have completed before TMEM is released
    __syncwarp();
    warp_wait(smem_u32(&sm.drain), 0, sm, a.err_flag, 5);
  } else {
    lv_epilogue<ENERGY, S>(a, sm, tmem, warp, lane);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
  }
}

// ------------------------------------------------------------------ split side
// Row maxima of any source layout: 64 x 64 tiles gathered through the tables.
__device__ __forceinline__ void exp_generic(const OzSplitJob& jb, const OzPanel& pn, int t,
                                            unsigned long long (*tile)[kSplitT + 1]) {
  const int ktiles = (jb.K + kSplitT - 1) / kSplitT;
  const int r0 = (t / ktiles) * kSplitT, k0 = (t % ktiles) * kSplitT;
  load_job_tile(jb, r0, k0, tile);
  __syncthreads();
  // 4 threads per row, 16 k each
  const int r = threadIdx.x >> 2, part = threadIdx.x & 3;
  int m = 0;
  for (int k = part * 16; k < part * 16 + 16; ++k) m = max(m, int((tile[r][k] >> 52) & 0x7FF));
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
  if (part == 0 && r0 + r < jb.rows && m > 0) atomicMax(&pn.exps[r0 + r], m);
}

// Row maxima of a column-major [rows x K] block (rows contiguous): 64 rows and
// up to kExpRowsK k of them.  A thread owns two rows (one 16-byte load per k)
// and every KG-th k, eight loads in flight; the row maxima meet in shared
// memory, and a row's k range in one global atomic (pieces of 512 rows x 32 k
// sent one per row and 32 k: the o=10/v=48 step's
// pass 19 us instead of 15).
constexpr int kExpRows = 64, kExpRowsK = 256;
__device__ __forceinline__ void exp_rows(const OzSplitJob& jb, const OzPanel& pn, int t, int* best) {
  const int ktiles = (jb.K + kExpRowsK - 1) / kExpRowsK;
  const int r0 = (t / ktiles) * kExpRows, k0 = (t % ktiles) * kExpRowsK;
  const int rows = min(kExpRows, jb.rows - r0), kn = min(kExpRowsK, jb.K - k0);
  const int rp = rows > 32 ? 32 : rows > 16 ? 16 : 8, kg = 256 / rp;
  const int lane = threadIdx.x % rp, kq = threadIdx.x / rp;
  if (threadIdx.x < kExpRows) best[threadIdx.x] = 0;
  __syncthreads();
  const int r = 2 * lane;
  unsigned long long m0 = 0, m1 = 0;
  constexpr unsigned long long kExp = 0x7FF0000000000000ull;
  if (r < rows) {
    const double* base = jb.src + size_t(k0) * jb.rows + r0 + r;
    if (r + 1 < rows && (jb.rows & 1) == 0) {
#pragma unroll 8
      for (int k = kq; k < kn; k += kg) {
        const double2 v = __ldg(reinterpret_cast<const double2*>(base + size_t(k) * jb.rows));
        m0 = max(m0, __double_as_longlong(v.x) & kExp);
        m1 = max(m1, __double_as_longlong(v.y) & kExp);
      }
    } else {
      const bool two = r + 1 < rows;
#pragma unroll 4
      for (int k = kq; k < kn; k += kg) {
        m0 = max(m0, __double_as_longlong(__ldg(base + size_t(k) * jb.rows)) & kExp);
        if (two) m1 = max(m1, __double_as_longlong(__ldg(base + size_t(k) * jb.rows + 1)) & kExp);
      }
    }
    if (m0) atomicMax(&best[r], int(m0 >> 52));
    if (m1) atomicMax(&best[r + 1], int(m1 >> 52));
  }
  __syncthreads();
  if (threadIdx.x < rows && best[threadIdx.x]) atomicMax(&pn.exps[r0 + threadIdx.x], best[threadIdx.x]);
}

// Row maxima of a [K x rows] block (k contiguous): one warp per row.
__device__ __forceinline__ void exp_kmaj(const OzSplitJob& jb, const OzPanel& pn, int t) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool vec = (jb.K & 1) == 0;
  for (int rr = 0; rr < 4; ++rr) {
    const int r = t * 32 + warp * 4 + rr;
    if (r >= jb.rows) return;
    const double* row = jb.src + size_t(r) * jb.K;
    unsigned long long m = 0;
    if (vec) {
      const double2* row2 = reinterpret_cast<const double2*>(row);
#pragma unroll 4
      for (int k = lane; k < jb.K / 2; k += 32) {
        const double2 v = __ldg(row2 + k);
        m = max(m, max(__double_as_longlong(v.x) & 0x7FF0000000000000ull,
                       __double_as_longlong(v.y) & 0x7FF0000000000000ull));
      }
    } else {
#pragma unroll 4
      for (int k = lane; k < jb.K; k += 32)
        m = max(m, __double_as_longlong(__ldg(row + k)) & 0x7FF0000000000000ull);
    }
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0 && m) atomicMax(&pn.exps[r], int(m >> 52));
  }
}

__global__ void __launch_bounds__(256) oz_exp_kernel(const __grid_constant__ OzJobSetRefs sets) {
  extern __shared__ __align__(16) unsigned long long exp_smem[];
  auto* tile = reinterpret_cast<unsigned long long(*)[kSplitT + 1]>(exp_smem);
  const JobPiece p = job_piece(sets);
  if (p.layout == kOzRowsMajor) exp_rows(p.jb, p.pn, p.tile, reinterpret_cast<int*>(tile));
  else if (p.layout == kOzKMajor) exp_kmaj(p.jb, p.pn, p.tile);
  else exp_generic(p.jb, p.pn, p.tile, tile);
}

// Balanced base-256 digits of n, most significant first: d[0] in [-128, 128],
// the others in [-128, 127]; sum_i d[i] * 256^(S-1-i) == n.  The low 24 bits
// give up to three digits with 32-bit arithmetic; the rest (|n| < 2^47 for up
// to 6 slices) also stays in 32 bits, only 7 slices need 64-bit steps.  S is
// a compile-time constant so every digit lives in a register.
template <int S>
__device__ __forceinline__ void balanced_digits(long long n, int (&d)[S]) {
  constexpr int K = S - 1 < 3 ? S - 1 : 3;  // digits taken from the low 24 bits
  int x = int(n & 0xFFFFFF);
  const long long hi = n >> 24;  // arithmetic shift: n == hi * 2^24 + x
#pragma unroll
  for (int t = 0; t < K; ++t) {
    const int r = ((x + 128) & 255) - 128;
    d[S - 1 - t] = r;
    x = (x - r) >> 8;
  }
  if constexpr (S <= 6) {
    int rem = int(hi << (24 - 8 * K)) + x;
#pragma unroll
    for (int t = K; t < S - 1; ++t) {
      const int r = ((rem + 128) & 255) - 128;
      d[S - 1 - t] = r;
      rem = (rem - r) >> 8;
    }
    d[0] = rem;
  } else {
    long long rem = (hi << (24 - 8 * K)) + x;
#pragma unroll
    for (int t = K; t < S - 1; ++t) {
      const long long r = ((rem + 128) & 255) - 128;
      d[S - 1 - t] = int(r);
      rem = (rem - r) >> 8;
    }
    d[0] = int(rem);
  }
}

// Exact BF16 bits of two digits in [-128, 128]: float(d) is formed exactly as
// (2^23 + 256 + d) - (2^23 + 256); one cvt.rn.bf16x2.f32 packs the pair (exact,
// at most 8 significant bits).
__device__ __forceinline__ uint32_t digits_bf16x2(int d0, int d1) {
  const float f0 = __fsub_rn(__uint_as_float(0x4B000000u + uint32_t(d0 + 256)), 8388864.0f);
  const float f1 = __fsub_rn(__uint_as_float(0x4B000000u + uint32_t(d1 + 256)), 8388864.0f);
  __nv_bfloat162 h = __floats2bfloat162_rn(f0, f1);
  return *reinterpret_cast<uint32_t*>(&h);
}

// Slices of any source layout: 64 x 64 tiles gathered through the tables.
template <int S>
__device__ __forceinline__ void split_generic(const OzSplitJob& jb, const OzPanel& pn, int tl,
                                              unsigned long long (*tile)[kSplitT + 1]) {
  const int ktiles = (jb.K + kSplitT - 1) / kSplitT;
  const int r0 = (tl / ktiles) * kSplitT, k0 = (tl % ktiles) * kSplitT;
  load_job_tile(jb, r0, k0, tile);
  __syncthreads();
  // each thread: one row, two consecutive k -> one bf16x2 store per slice
  const int kp = threadIdx.x & 31;
  for (int p = 0; p < 8; ++p) {
    const int r = (threadIdx.x >> 5) + 8 * p;
    if (r0 + r >= jb.rows) continue;
    const int k = 2 * kp;
    if (k0 + k >= jb.K) continue;
    const int mx = pn.exps[r0 + r];
    const unsigned long long b0 = tile[r][k], b1 = (k0 + k + 1 < jb.K) ? tile[r][k + 1] : 0ull;
    int d0[S], d1[S];
    balanced_digits<S>(quantize(b0, mx, S), d0);
    balanced_digits<S>(quantize(b1, mx, S), d1);
    uint32_t* dst = reinterpret_cast<uint32_t*>(pn.base + (size_t(r0 + r) * pn.kpad + jb.koff + k0 + k));
    const size_t slice_stride = size_t(pn.rows_pad) * pn.kpad / 2;
#pragma unroll
    for (int i = 0; i < S; ++i) dst[i * slice_stride] = digits_bf16x2(d0[i], d1[i]);
  }
}

// Slices of a [K x rows] block: one warp per row, each lane four consecutive k
// (two 16-byte loads, one 8-byte store per slice).
template <int S>
__device__ __forceinline__ void split_kmaj(const OzSplitJob& jb, const OzPanel& pn, int tl) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = tl * 8 + warp;
  if (r >= jb.rows) return;
  const int mx = pn.exps[r];
  const double* row = jb.src + size_t(r) * jb.K;
  uint2* dst = reinterpret_cast<uint2*>(pn.base + (size_t(r) * pn.kpad + jb.koff));
  const size_t slice_stride = size_t(pn.rows_pad) * pn.kpad / 4;  // in uint2 (4 bf16)
  const bool vec = (jb.K & 3) == 0;
  for (int k = 4 * lane; k < jb.K; k += 128) {
    unsigned long long b[4];
    if (vec) {
      const double2 v0 = __ldg(reinterpret_cast<const double2*>(row + k));
      const double2 v1 = __ldg(reinterpret_cast<const double2*>(row + k + 2));
      b[0] = __double_as_longlong(v0.x), b[1] = __double_as_longlong(v0.y);
      b[2] = __double_as_longlong(v1.x), b[3] = __double_as_longlong(v1.y);
    } else {
#pragma unroll
      for (int t = 0; t < 4; ++t) b[t] = k + t < jb.K ? __double_as_longlong(__ldg(row + k + t)) : 0ull;
    }
    int d[4][S];
#pragma unroll
    for (int t = 0; t < 4; ++t) balanced_digits<S>(quantize(b[t], mx, S), d[t]);
#pragma unroll
    for (int i = 0; i < S; ++i) {
      uint2 o;
      o.x = digits_bf16x2(d[0][i], d[1][i]);
      o.y = digits_bf16x2(d[2][i], d[3][i]);
      dst[i * slice_stride + (k >> 2)] = o;
    }
  }
}

// Column of k inside a row of the transpose tile: within each 16-column group
// the low two bits are rotated by the group index, so that the store phase's
// half-warp (one row, columns 4 kq + u for kq = 0..15) hits 16 distinct bank
// pairs instead of 4 (k = 16 b + 4 a + u is kept at 16 b + 4 a + (u + b) mod 4).
__device__ __forceinline__ int rows_tile_col(int k) { return (k & ~3) | (((k & 3) + (k >> 4)) & 3); }

// Slices of a column-major [rows x K] block: 64x64 tiles transposed through
// shared memory (16-byte loads along rows, 8-byte stores along k).
template <int S>
__device__ __forceinline__ void split_rows(const OzSplitJob& jb, const OzPanel& pn, int tl,
                                           unsigned long long (*tile)[kSplitT + 1]) {
  const int ktiles = (jb.K + 63) / 64;
  const int r0 = (tl / ktiles) * 64, k0 = (tl % ktiles) * 64;
  const int t = threadIdx.x;
  // load: thread -> (row pair, k): 32 row pairs x 8 k per pass, 8 passes
  const bool vec = (jb.rows & 1) == 0;
#pragma unroll
  for (int p = 0; p < 8; ++p) {
    const int rp = t & 31, k = (t >> 5) + 8 * p;
    const int r = r0 + 2 * rp;
    unsigned long long x0 = 0, x1 = 0;
    if (k0 + k < jb.K && r < jb.rows) {
      const double* src = jb.src + size_t(k0 + k) * jb.rows + r;
      if (vec) {
        const double2 v = __ldg(reinterpret_cast<const double2*>(src));
        x0 = __double_as_longlong(v.x), x1 = __double_as_longlong(v.y);
      } else {
        x0 = __double_as_longlong(__ldg(src));
        if (r + 1 < jb.rows) x1 = __double_as_longlong(__ldg(src + 1));
      }
    }
    tile[2 * rp][rows_tile_col(k)] = x0;
    tile[2 * rp + 1][rows_tile_col(k)] = x1;
  }
  __syncthreads();
  // store: thread -> (row, 4 consecutive k): 16 k-quads x 16 rows per pass, 4 passes
  const size_t slice_stride = size_t(pn.rows_pad) * pn.kpad / 4;
#pragma unroll 1
  for (int p = 0; p < 4; ++p) {
    const int kq = t & 15, r = (t >> 4) + 16 * p;
    if (r0 + r >= jb.rows || k0 + 4 * kq >= jb.K) continue;
    const int mx = pn.exps[r0 + r];
    int d[4][S];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned long long b = (k0 + 4 * kq + u < jb.K) ? tile[r][rows_tile_col(4 * kq + u)] : 0ull;
      balanced_digits<S>(quantize(b, mx, S), d[u]);
    }
    uint2* dst = reinterpret_cast<uint2*>(pn.base + (size_t(r0 + r) * pn.kpad + jb.koff + k0 + 4 * kq));
#pragma unroll
    for (int i = 0; i < S; ++i) {
      uint2 o;
      o.x = digits_bf16x2(d[0][i], d[1][i]);
      o.y = digits_bf16x2(d[2][i], d[3][i]);
      dst[i * slice_stride] = o;
    }
  }
}

template <int S>
__global__ void __launch_bounds__(256) oz_split_kernel(const __grid_constant__ OzJobSetRefs sets) {
  __shared__ unsigned long long tile[kSplitT][kSplitT + 1];
  const JobPiece p = job_piece(sets);
  if (p.layout == kOzRowsMajor) split_rows<S>(p.jb, p.pn, p.tile, tile);
  else if (p.layout == kOzKMajor) split_kmaj<S>(p.jb, p.pn, p.tile);
  else split_generic<S>(p.jb, p.pn, p.tile, tile);
}

// ------------------------------------------------------------------ recombine
// One block of 256 threads per 32-column strip of a tile, walked as 32x32
// pieces (four elements per thread): every level's split partials of a piece
// are loaded before any is used (20 loads in flight per thread at 5 slices),
// summed exactly (int64), the levels combined exactly (64-bit when the top
// level allows it, else 128-bit) and rounded once to FP64 with the row/column
// scales.  Reads run along rows (the workspace order); strips whose D is
// unit-stride along n transpose through shared memory so the stores run
// along n.
template <int S>
__global__ void __launch_bounds__(256) oz_recombine_kernel(const OzTile* __restrict__ tiles,
                                                           const OzDBlock* __restrict__ dblocks,
                                                           const OzPanel* __restrict__ pa,
                                                           const OzPanel* __restrict__ pb,
                                                           const int* __restrict__ ws, int log_rows, int log_cols,
                                                           int nsplit, int mode) {
  constexpr int kSub = 32, kPer = kSub * kSub / 256;
  __shared__ double sm[kSub][kSub + 1];
  const int strips_log = log_cols - 5;
  const int tile = blockIdx.x >> strips_log;
  const int sc = (blockIdx.x & ((1 << strips_log) - 1)) * kSub;
  const OzTile tl = tiles[tile];
  const OzDBlock db = dblocks[tl.dblock];
  const int* ea = pa[tl.panel_a].exps;
  const int* eb = pb[tl.panel_b].exps;
  const size_t plane = size_t(1) << (log_rows + log_cols);     // one split's [cols][rows]
  const int* wtile = ws + size_t(tile) * S * nsplit * plane;
  const int rows_here = min(1 << log_rows, db.M - tl.m0);
  for (int sr = 0; sr < rows_here; sr += kSub) {
    long long lev[kPer][S];
#pragma unroll
    for (int p = 0; p < kPer; ++p)
#pragma unroll
      for (int lv = 0; lv < S; ++lv) lev[p][lv] = 0;
    for (int sp = 0; sp < nsplit; ++sp) {
      int raw[kPer][S];
#pragma unroll
      for (int p = 0; p < kPer; ++p) {
        const int e = p * 256 + threadIdx.x;
        const int row = sr + (e & (kSub - 1)), col = sc + (e >> 5);
        const int* q = wtile + (size_t(sp) << (log_rows + log_cols)) + (size_t(col) << log_rows) + row;
#pragma unroll
        for (int lv = 0; lv < S; ++lv) raw[p][lv] = __ldg(q + size_t(lv) * nsplit * plane);
      }
#pragma unroll
      for (int p = 0; p < kPer; ++p)
#pragma unroll
        for (int lv = 0; lv < S; ++lv) lev[p][lv] += raw[p][lv];
    }
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
      const int e = p * 256 + threadIdx.x;
      const int row = sr + (e & (kSub - 1)), col = sc + (e >> 5);
      const int m = tl.m0 + row, n = tl.n0 + col;
      double v = 0.0;
      const bool live = m < db.M && n < db.N;
      if (live) {
        // value = sum_t lev[t] 2^(8(S-1-t)) * 2^(E + F + 2 - 8(S+1))
        const int E = (ea[m] ? ea[m] : 1) - 1022, F = (eb[n] ? eb[n] : 1) - 1022;
        const int e2 = E + F + 2 - kDigitBits * (S + 1);
        const long long top = lev[p][0] < 0 ? -lev[p][0] : lev[p][0];
        if (top < (1ll << (62 - kDigitBits * (S - 1)))) {  // the 64-bit sum cannot overflow
          long long acc = 0;
#pragma unroll
          for (int lv = 0; lv < S; ++lv) acc += lev[p][lv] * (1ll << (kDigitBits * (S - 1 - lv)));
          v = i64_scaled_to_double(acc, e2, false);
        } else {
          unsigned __int128 acc = 0;  // two's complement, wrapping (exact: |sum| < 2^101)
#pragma unroll
          for (int lv = 0; lv < S; ++lv)
            acc += (unsigned __int128)(__int128)lev[p][lv] << (kDigitBits * (S - 1 - lv));
          v = i128_scaled_to_double((__int128)acc, e2);
        }
        if (mode & 2) v = -v;  // negated term
        if (ea[m] == kNonFiniteExp || eb[n] == kNonFiniteExp) v = __longlong_as_double(0x7FF8000000000000ll);
      }
      if (db.col_fast) {
        sm[e & (kSub - 1)][e >> 5] = v;
      } else if (live) {
        double* dst = db.colptr[n] + db.rowoff[m];
        *dst = (mode & 1) ? *dst + v : v;
      }
    }
    if (!db.col_fast) continue;
    __syncthreads();
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
      const int e = p * 256 + threadIdx.x;
      const int col = sc + (e & (kSub - 1)), row = sr + (e >> 5);
      const int m = tl.m0 + row, n = tl.n0 + col;
      if (m < db.M && n < db.N) {
        const double v = sm[e >> 5][e & (kSub - 1)];
        double* dst = db.colptr[n] + db.rowoff[m];
        *dst = (mode & 1) ? *dst + v : v;
      }
    }
    __syncthreads();
  }
}

// Single-split form of the recombine (every level sum already complete, e.g.
// the short-k triples): a persistent CTA per SM walks pieces of 4096 elements
// (16 KB per level: one whole column run of the tile's int32 plane per
// level, 16 or 32 columns; 1024 threads, four elements each), each level's
// piece fetched by one bulk async copy
// into a double-buffered shared-memory stage, so the next piece streams in
// while this one is combined and stored.  Waits are bounded (error flag, then
// a bounded drain of the copy still in flight).
constexpr int kRecPiece = 4096;  // int32 elements per level per piece (16 KB)
// Pieces in flight: one ahead of the one being combined.  (Four stages of
// 2048-element pieces were measured slower: 14 instead of 11 ms on the
// triples' term 1, the per-piece overhead doubling.)
constexpr int kRecStages = 2;

template <int S>
struct __align__(128) RecSmem {
  int lev[kRecStages][S][kRecPiece];
  double val[kRecPiece + 64];  // [col][rows + 1] transpose buffer
  uint64_t full[kRecStages];
};

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ bool wait_bounded(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = now_ns();
#pragma unroll 1
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255) == 0 && now_ns() - t0 > kWaitLimitNs) return false;
  }
}

template <int S>
__global__ void __launch_bounds__(1024, 1) oz_recombine_bulk_kernel(const OzTile* __restrict__ tiles,
                                                                  const OzDBlock* __restrict__ dblocks,
                                                                         const OzPanel* __restrict__ pa,
                                                                  const OzPanel* __restrict__ pb,
                                                                  const int* __restrict__ ws, int log_rows,
                                                                  int log_cols, int n_tiles, int mode, int* err) {
  extern __shared__ __align__(128) unsigned char rec_smem_raw[];
  RecSmem<S>& sm = *reinterpret_cast<RecSmem<S>*>(rec_smem_raw);
  const int rows = 1 << log_rows;
  const int cols_pp = kRecPiece >> log_rows;                    // columns per piece
  const int pieces_per_tile = 1 << (log_rows + log_cols - 12);  // 4096 = 2^12
  const int npieces = n_tiles * pieces_per_tile;
  const size_t plane = size_t(1) << (log_rows + log_cols);
  if (threadIdx.x == 0) {
    for (int st = 0; st < kRecStages; ++st) mbar_init(&sm.full[st], 1);
    fence_mbar_init();
  }
  __syncthreads();
  auto issue = [&](int q, int st) {
    const int tile = q / pieces_per_tile, pc = q % pieces_per_tile;
    mbar_expect_tx(&sm.full[st], uint32_t(S) * kRecPiece * 4);
#pragma unroll
    for (int lv = 0; lv < S; ++lv)
      bulk_g2s(sm.lev[st][lv], ws + (size_t(tile) * S + lv) * plane + size_t(pc) * kRecPiece, kRecPiece * 4,
               &sm.full[st]);
  };
  int q = blockIdx.x;
  const int G = gridDim.x;
  if (threadIdx.x == 0)
    for (int i = 0; i < kRecStages - 1; ++i)
      if (q + i * G < npieces) issue(q + i * G, i);
  for (int it = 0; q < npieces; q += G, ++it) {
    const int st = it % kRecStages;
    // the stage of piece it + kRecStages - 1 was combined in iteration it - 1
    // (the barrier at the end of that iteration freed it)
    const int ahead = q + (kRecStages - 1) * G;
    if (threadIdx.x == 0 && ahead < npieces) issue(ahead, (it + kRecStages - 1) % kRecStages);
    if (!wait_bounded(&sm.full[st], uint32_t(it / kRecStages) & 1u)) {
      atomicExch(err, 5);
      // drain the later pieces' copies (those issued) before this CTA's memory is released
      if (threadIdx.x == 0)
        for (int i = 1; i < kRecStages && q + i * G < npieces; ++i)
          wait_bounded(&sm.full[(it + i) % kRecStages], uint32_t((it + i) / kRecStages) & 1u);
      return;
    }
    const int tile = q / pieces_per_tile, pc = q % pieces_per_tile;
    const OzTile tl = tiles[tile];
    const OzDBlock db = dblocks[tl.dblock];
    const int* ea = pa[tl.panel_a].exps;
    const int* eb = pb[tl.panel_b].exps;
    const int sc = pc * cols_pp;
    constexpr int kPerT = kRecPiece / 1024;
    double vals[kPerT];
    double* dsts[kPerT];
#pragma unroll
    for (int p = 0; p < kPerT; ++p) {
      const int e = p * 1024 + threadIdx.x;
      const int row = e & (rows - 1), cl = e >> log_rows;
      const int m = tl.m0 + row, n = tl.n0 + sc + cl;
      double v = 0.0;
      const bool live = m < db.M && n < db.N;
      if (live) {
        const int E = (ea[m] ? ea[m] : 1) - 1022, F = (eb[n] ? eb[n] : 1) - 1022;
        const int e2 = E + F + 2 - kDigitBits * (S + 1);
        long long acc = 0;  // a unit's level-t sum is below (t+1) 2^31 / S: the 64-bit sum is exact
#pragma unroll
        for (int lv = 0; lv < S; ++lv) acc += (long long)sm.lev[st][lv][e] * (1ll << (kDigitBits * (S - 1 - lv)));
        v = i64_scaled_to_double(acc, e2, mode & 2);  // negated term: the sign folded into the rounding
        if (ea[m] == kNonFiniteExp || eb[n] == kNonFiniteExp) v = __longlong_as_double(0x7FF8000000000000ll);
      }
      vals[p] = v;
      dsts[p] = nullptr;
      if (db.col_fast) sm.val[cl * (rows + 1) + row] = v;
      else if (live) dsts[p] = db.colptr[n] + db.rowoff[m];
    }
    if (!db.col_fast) {
      double old[kPerT];  // accumulate mode: the old values' loads in flight together
#pragma unroll
      for (int p = 0; p < kPerT; ++p) old[p] = (dsts[p] && (mode & 1)) ? *dsts[p] : 0.0;
#pragma unroll
      for (int p = 0; p < kPerT; ++p)
        if (dsts[p]) *dsts[p] = (mode & 1) ? old[p] + vals[p] : vals[p];
    }
    if (db.col_fast) {
      __syncthreads();
      constexpr int kPer = kRecPiece / 1024;
      double* dst[kPer];
      double old[kPer];
#pragma unroll
      for (int p = 0; p < kPer; ++p) {  // addresses and (beta) the old values first: loads in flight together
        const int e = p * 1024 + threadIdx.x;
        const int cl = e % cols_pp, row = e / cols_pp;
        const int m = tl.m0 + row, n = tl.n0 + sc + cl;
        dst[p] = (m < db.M && n < db.N) ? db.colptr[n] + db.rowoff[m] : nullptr;
        old[p] = (dst[p] && (mode & 1)) ? *dst[p] : 0.0;
      }
#pragma unroll
      for (int p = 0; p < kPer; ++p) {
        const int e = p * 1024 + threadIdx.x;
        const int cl = e % cols_pp, row = e / cols_pp;
        if (dst[p]) *dst[p] = (mode & 1) ? old[p] + sm.val[cl * (rows + 1) + row] : sm.val[cl * (rows + 1) + row];
      }
    }
    __syncthreads();  // stage st and the transpose buffer are free again
  }
}

// Self-test of the bounded-wait path every pipeline wait uses: one thread
// waits on an mbarrier that nothing arrives at, gives up after limit_ns, and
// reports through the device error flag exactly as a stalled pipeline would.
__global__ void wait_timeout_selftest_kernel(unsigned long long limit_ns, int* err, int* waited_ms) {
  __shared__ uint64_t bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar, 1);
  fence_mbar_init();
  const unsigned long long t0 = now_ns();
  bool done = mbar_try_wait(&bar, 0);
#pragma unroll 1
  for (uint32_t it = 1; !done; ++it) {
    done = mbar_try_wait(&bar, 0);
    if (!done && (it & 255) == 0 && now_ns() - t0 > limit_ns) break;
  }
  *waited_ms = int((now_ns() - t0) / 1000000ull);
  if (!done) atomicExch(err, 6);
}

// Self-tests of the one-rounding helpers exactly as the kernels run them: the
// integer-to-FP64 rounding of every split-precision epilogue and the exact
// division of the denominator and energy passes, one element per thread.
__global__ void round_selftest_kernel(int n, const long long* __restrict__ v, const int* __restrict__ e2,
                                      const int* __restrict__ neg, double* __restrict__ out) {
  const int i = int(blockIdx.x) * int(blockDim.x) + int(threadIdx.x);
  if (i < n) out[i] = i64_scaled_to_double(v[i], e2[i], neg[i] != 0);
}
__global__ void div_selftest_kernel(int n, const double* __restrict__ a, const double* __restrict__ b,
                                    double* __restrict__ out) {
  const int i = int(blockIdx.x) * int(blockDim.x) + int(threadIdx.x);
  if (i < n) out[i] = div_rn(a[i], b[i]);
}

// esum += efact * (sum of the n partial energies), the partials added in a
// fixed order (one CTA: strided per-thread sums, then a fixed tree), so a GPU
// gives the same bits every run.
__global__ void __launch_bounds__(1024) oz_energy_reduce_kernel(const double* __restrict__ part, int n,
                                                                double efact, double* esum) {
  __shared__ double red[1024];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += 1024) acc += part[i];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = 512; w > 0; w >>= 1) {
    if (int(threadIdx.x) < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *esum += efact * red[0];
}

using EncodeTiled = PFN_cuTensorMapEncodeTiled_v12000;
EncodeTiled get_encoder() {
  static EncodeTiled fn = nullptr;
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(p);
  }
  return fn;
}

}  // namespace

int oz_chunk_kb(int level) {
  // largest multiple of 64 k such that (level+1) * 128^2 * k < 2^24: every
  // FP32 partial sum of the chunk is an integer below 2^24, hence exact
  const long long per = (long long)(level + 1) * 128 * 128;
  const long long k = ((1LL << 24) - 1) / per;
  return int(k / kOzBK);
}

// A panel's planes as a 3-D map.  Its rows end at the last live one: a box that
// reaches into the padding gets zeros without reading them (the o=10/v=48
// step's 144 rows a block, padded to 256: its GEMM 43 -> 31 us, panel reads
// 208 -> 117 MB).
int oz_make_tensor_map(void* map128, const void* base, int64_t kpad, int64_t rows, int64_t rows_pad, int planes,
                       int box_rows) {
  EncodeTiled enc = get_encoder();
  if (!enc) return fail(A4G_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  if (kpad % kOzBK != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0)
    return fail(A4G_ERR_ARG, "panel not aligned for TMA");
  cuuint64_t dims[3] = {cuuint64_t(kpad), cuuint64_t(rows), cuuint64_t(planes)};
  cuuint64_t strides[2] = {cuuint64_t(kpad) * 2, cuuint64_t(rows_pad) * cuuint64_t(kpad) * 2};
  cuuint32_t box[3] = {cuuint32_t(kOzBK), cuuint32_t(box_rows), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(reinterpret_cast<CUtensorMap*>(map128), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3,
                   const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(A4G_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string(int(r)));
  return A4G_OK;
}

int oz_make_levels_map(void* map128, const void* base, int64_t kpad, int64_t rows, int64_t rows_pad, int slices,
                       int box_rows) {
  EncodeTiled enc = get_encoder();
  if (!enc) return fail(A4G_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  if (kpad % kOzBK != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0)
    return fail(A4G_ERR_ARG, "panel not aligned for TMA");
  cuuint64_t dims[3] = {cuuint64_t(kpad), cuuint64_t(rows), cuuint64_t(slices)};
  cuuint64_t strides[2] = {cuuint64_t(kpad) * 2, cuuint64_t(rows_pad) * cuuint64_t(kpad) * 2};
  cuuint32_t box[3] = {cuuint32_t(kLvBK), cuuint32_t(box_rows), cuuint32_t(slices)};
  cuuint32_t estr[3] = {1, 1, 1};
  // rows of 64 B (32 k) with the 64-byte swizzle
  CUresult r = enc(reinterpret_cast<CUtensorMap*>(map128), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3,
                   const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(A4G_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string(int(r)));
  return A4G_OK;
}

int64_t oz_exp_tiles(int layout, int rows, int K) {
  if (layout == kOzRowsMajor) return int64_t((rows + kExpRows - 1) / kExpRows) * ((K + kExpRowsK - 1) / kExpRowsK);
  if (layout == kOzKMajor) return (rows + 31) / 32;
  return int64_t((rows + 63) / 64) * ((K + 63) / 64);
}

int64_t oz_split_tiles(int layout, int rows, int K) {
  if (layout == kOzKMajor) return (rows + 7) / 8;
  return int64_t((rows + 63) / 64) * ((K + 63) / 64);
}

int oz_launch_exp(const OzJobSetRefs& sets, cudaStream_t s) {
  if (!sets.total) return A4G_OK;
  if (!sets.fits()) return fail(A4G_ERR_RANGE, "too many split tiles");
  // what the layouts at hand need (the row maxima, or a gathered tile): it bounds the CTAs per SM
  size_t smem = 512 * sizeof(int);
  for (int q = 0; q < sets.n; ++q)
    if (sets.s[q].layout == kOzGeneric) smem = kSplitT * (kSplitT + 1) * sizeof(unsigned long long);
  oz_exp_kernel<<<unsigned(sets.total), 256, smem, s>>>(sets);
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

int oz_launch_split(const OzJobSetRefs& sets, int slices, cudaStream_t s) {
  if (!sets.total) return A4G_OK;
  if (!sets.fits()) return fail(A4G_ERR_RANGE, "too many split tiles");
  switch (slices) {
    case 1: oz_split_kernel<1><<<unsigned(sets.total), 256, 0, s>>>(sets); break;
    case 2: oz_split_kernel<2><<<unsigned(sets.total), 256, 0, s>>>(sets); break;
    case 3: oz_split_kernel<3><<<unsigned(sets.total), 256, 0, s>>>(sets); break;
    case 4: oz_split_kernel<4><<<unsigned(sets.total), 256, 0, s>>>(sets); break;
    case 5: oz_split_kernel<5><<<unsigned(sets.total), 256, 0, s>>>(sets); break;
    case 6: oz_split_kernel<6><<<unsigned(sets.total), 256, 0, s>>>(sets); break;
    case 7: oz_split_kernel<7><<<unsigned(sets.total), 256, 0, s>>>(sets); break;
    default: return fail(A4G_ERR_ARG, "slices must be 1..7");
  }
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

template <bool PAIR, int BN, bool DIRECT = false, bool ENERGY = false, bool RES = false>
int set_smem_attr() {
  A4G_CUDA(cudaFuncSetAttribute(oz_gemm_kernel<PAIR, BN, DIRECT, ENERGY, RES>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(OzSmemT<PAIR, BN>)) + 1024));
  return A4G_OK;
}

template <bool ENERGY, int S = kLvMaxS>
int set_levels_attr() {
  A4G_CUDA(cudaFuncSetAttribute(oz_levels_kernel<ENERGY, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                int(sizeof(LvSmem)) + 1024));
  if constexpr (S > 1) return set_levels_attr<ENERGY, S - 1>();
  else return A4G_OK;
}

template <bool ENERGY>
void launch_levels(const OzGemmArgs& args, int grid, cudaStream_t s) {
  const size_t smem = sizeof(LvSmem) + 1024;
  switch (args.slices) {
    case 1: oz_levels_kernel<ENERGY, 1><<<grid, kThreadsOzDirect, smem, s>>>(args); break;
    case 2: oz_levels_kernel<ENERGY, 2><<<grid, kThreadsOzDirect, smem, s>>>(args); break;
    case 3: oz_levels_kernel<ENERGY, 3><<<grid, kThreadsOzDirect, smem, s>>>(args); break;
    case 4: oz_levels_kernel<ENERGY, 4><<<grid, kThreadsOzDirect, smem, s>>>(args); break;
    default: oz_levels_kernel<ENERGY, 5><<<grid, kThreadsOzDirect, smem, s>>>(args); break;
  }
}

// Function attributes are set once per device (they belong to the device's
// instance of the kernel).
bool first_on_device(std::atomic<unsigned long long>& mask) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return true;
  const unsigned long long bit = 1ull << dev;
  return (mask.fetch_or(bit) & bit) == 0;
}

int oz_prepare() {
  static std::atomic<unsigned long long> done{0};
  if (first_on_device(done)) {
    int rc;
    if ((rc = set_smem_attr<false, 128>()) || (rc = set_smem_attr<true, 128>()) ||
        (rc = set_smem_attr<false, 256>()) || (rc = set_smem_attr<true, 256>()) ||
        (rc = set_smem_attr<false, 128, true>()) || (rc = set_smem_attr<true, 128, true>()) ||
        (rc = set_smem_attr<false, 128, false, false, true>()) || (rc = set_smem_attr<true, 128, false, false, true>()) ||
        (rc = set_smem_attr<false, 256, false, false, true>()) || (rc = set_smem_attr<true, 256, false, false, true>()) ||
        (rc = set_smem_attr<false, 128, true, true>()) || (rc = set_levels_attr<false>()) ||
        (rc = set_levels_attr<true>()) || (rc = oz_residue_prepare())) {
      done.store(0);
      return rc;
    }
  }
  return A4G_OK;
}

int oz_max_pairs(int* pairs) {
  int rc = oz_prepare();
  if (rc) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * 76, 1, 1);
  cfg.blockDim = dim3(kThreadsOz, 1, 1);
  cfg.dynamicSmemBytes = sizeof(OzSmemT<true, 128>) + 1024;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0, n2 = 0;
  A4G_CUDA(cudaOccupancyMaxActiveClusters(&n, oz_gemm_kernel<true, 128>, &cfg));
  cfg.dynamicSmemBytes = sizeof(OzSmemT<true, 256>) + 1024;
  A4G_CUDA(cudaOccupancyMaxActiveClusters(&n2, oz_gemm_kernel<true, 256>, &cfg));
  *pairs = std::min(n, n2);
  return A4G_OK;
}

template <bool PAIR, int BN, bool DIRECT = false, bool ENERGY = false, bool RES = false>
int launch_form(const OzGemmArgs& args, int grid, cudaStream_t s) {
  const size_t smem = sizeof(OzSmemT<PAIR, BN>) + 1024;
  if constexpr (!PAIR) {
    oz_gemm_kernel<false, BN, DIRECT, ENERGY, RES><<<grid, DIRECT ? kThreadsOzDirect : kThreadsOz, smem, s>>>(args);
  } else {
    if (grid % 2) return fail(A4G_ERR_ARG, "CTA-pair grid must be even");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(DIRECT ? kThreadsOzDirect : kThreadsOz, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    A4G_CUDA(cudaLaunchKernelEx(&cfg, oz_gemm_kernel<true, BN, DIRECT, false, RES>, args));
  }
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

int oz_launch_gemm(const OzGemmArgs& args, int grid, bool pair, int tile_cols, cudaStream_t s) {
  if (!args.residue && args.slices > kOzMaxUsableSlices) return fail(A4G_ERR_ARG, "at most 7 slices");
  int rc = oz_prepare();
  if (rc) return rc;
  if (args.n_units <= 0) return A4G_OK;
  if (args.residue) {
    if (args.direct || args.slices > kOzMaxResidues) return fail(A4G_ERR_ARG, "residue form: workspace, at most 15 moduli");
    if (tile_cols == 256)
      return pair ? launch_form<true, 256, false, false, true>(args, grid, s)
                  : launch_form<false, 256, false, false, true>(args, grid, s);
    return pair ? launch_form<true, 128, false, false, true>(args, grid, s)
                : launch_form<false, 128, false, false, true>(args, grid, s);
  }
  if (args.direct) {
    if (tile_cols != 128 || args.nsplit != 1 || args.n_units % args.slices)
      return fail(A4G_ERR_ARG, "direct form: 128-column tiles, one split, whole tiles");
    if (args.energy) {
      if (pair || !args.eblocks || !args.epart) return fail(A4G_ERR_ARG, "energy form: one SM per tile, tables");
      return launch_form<false, 128, true, true>(args, grid, s);
    }
    return pair ? launch_form<true, 128, true>(args, grid, s) : launch_form<false, 128, true>(args, grid, s);
  }
  if (tile_cols == 256) return pair ? launch_form<true, 256>(args, grid, s) : launch_form<false, 256>(args, grid, s);
  return pair ? launch_form<true, 128>(args, grid, s) : launch_form<false, 128>(args, grid, s);
}

bool oz_levels_fit(int slices, int kb_total) { return slices >= 1 && slices <= kLvMaxS && kb_total <= 5; }

int oz_launch_levels(const OzGemmArgs& args, int grid, cudaStream_t s) {
  if (!oz_levels_fit(args.slices, 0) || !args.direct) return fail(A4G_ERR_ARG, "all-levels form: 1..5 slices, direct");
  int rc = oz_prepare();
  if (rc) return rc;
  if (args.n_tiles <= 0) return A4G_OK;
  if (args.energy) {
    if (!args.eblocks || !args.epart) return fail(A4G_ERR_ARG, "energy form: tables");
    launch_levels<true>(args, grid, s);
  } else {
    launch_levels<false>(args, grid, s);
  }
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

int oz_launch_recombine(const OzTile* tiles, int ntiles, int tile_rows, int tile_cols, const OzDBlock* dblocks,
                        const OzPanel* pa, const OzPanel* pb, const int* ws, int slices,
                        int nsplit, int mode, cudaStream_t s) {
  if (ntiles <= 0) return A4G_OK;
  if ((tile_rows != 128 && tile_rows != 256) || (tile_cols != 128 && tile_cols != 256))
    return fail(A4G_ERR_ARG, "recombine: unsupported tile shape");
  const int lr = tile_rows == 256 ? 8 : 7, lc = tile_cols == 256 ? 8 : 7;
  if (nsplit == 1 && slices <= 5) {
    // single split: the bulk-copy pipelined form (one CTA per SM)
    const int npieces = ntiles * (tile_rows * tile_cols / kRecPiece);
    const int grid = std::min(npieces, ctx()->num_sms > 0 ? ctx()->num_sms : 152);
    int* err = ctx()->d_error_flag;
    switch (slices) {
#define A4G_RECOMBINE_BULK(SL)                                                                                   \
  case SL: {                                                                                                     \
    static std::atomic<unsigned long long> attr{0};                                                             \
    if (first_on_device(attr))                                                                                   \
      A4G_CUDA(cudaFuncSetAttribute(oz_recombine_bulk_kernel<SL>, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                                    int(sizeof(RecSmem<SL>))));                                                 \
    oz_recombine_bulk_kernel<SL><<<grid, 1024, sizeof(RecSmem<SL>), s>>>(tiles, dblocks, pa, pb, ws, lr, lc, \
                                                                       ntiles, mode, err);                       \
    break;                                                                                                       \
  }
      A4G_RECOMBINE_BULK(1) A4G_RECOMBINE_BULK(2) A4G_RECOMBINE_BULK(3) A4G_RECOMBINE_BULK(4) A4G_RECOMBINE_BULK(5)
#undef A4G_RECOMBINE_BULK
    }
    A4G_CUDA(cudaGetLastError());
    return A4G_OK;
  }
  const int per = tile_cols / 32;  // 32-column strips per tile
  if (int64_t(ntiles) * per > 0x7fffffffLL) return fail(A4G_ERR_RANGE, "too many tiles");
  const unsigned g = unsigned(ntiles * per);
  switch (slices) {
#define A4G_RECOMBINE(SL) \
  case SL: oz_recombine_kernel<SL><<<g, 256, 0, s>>>(tiles, dblocks, pa, pb, ws, lr, lc, nsplit, mode); break;
    A4G_RECOMBINE(1) A4G_RECOMBINE(2) A4G_RECOMBINE(3) A4G_RECOMBINE(4) A4G_RECOMBINE(5) A4G_RECOMBINE(6)
    A4G_RECOMBINE(7)
#undef A4G_RECOMBINE
    default: return fail(A4G_ERR_ARG, "recombine: slices must be 1..7");
  }
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

int oz_launch_energy_reduce(const double* part, int n, double efact, double* esum, cudaStream_t s) {
  oz_energy_reduce_kernel<<<1, 1024, 0, s>>>(part, n, efact, esum);
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

int oz_wait_timeout_selftest(int limit_ms, int* waited_ms, cudaStream_t s) {
  int* d_ms = nullptr;
  if (const int rc_ = async_alloc(reinterpret_cast<void**>(&d_ms), sizeof(int), s)) return rc_;
  wait_timeout_selftest_kernel<<<1, 32, 0, s>>>((unsigned long long)limit_ms * 1000000ull, ctx()->d_error_flag, d_ms);
  A4G_CUDA(cudaGetLastError());
  A4G_CUDA(cudaMemcpyAsync(waited_ms, d_ms, sizeof(int), cudaMemcpyDeviceToHost, s));
  A4G_CUDA(cudaFreeAsync(d_ms, s));
  return A4G_OK;
}

int oz_round_selftest(int n, const long long* v, const int* e2, const int* neg, double* out, cudaStream_t s) {
  if (n <= 0) return A4G_OK;
  round_selftest_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(n, v, e2, neg, out);
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

int oz_div_selftest(int n, const double* a, const double* b, double* out, cudaStream_t s) {
  if (n <= 0) return A4G_OK;
  div_selftest_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(n, a, b, out);
  A4G_CUDA(cudaGetLastError());
  return A4G_OK;
}

}  // namespace a4g
