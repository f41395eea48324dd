// Prefill clustering: segmented inner-product Lloyd k-means, per-cluster value sums and the
// cluster-contiguous KV layout.
//
//   centre   mean key per group (fp32 sums in a fixed order), centred = round(key - mean)
//   assign   argmax_c <x, c> for every token of every problem: tcgen05 MMA (M = 128 tokens,
//            N = 128 centroids, K = 128 channels as 8 x K16) with operands staged by TMA
//            (128-byte swizzle) and fp32 accumulators in TMEM; a warp-specialised CTA
//            (TMA producer / MMA issuer / epilogue warps) overlaps the running arg-max of one
//            accumulator buffer with the MMAs into the other: blocks of 256 tokens (tiles of 128
//            where a problem's centroids stay in shared memory, N = 256 there), persistent CTAs
//            over the blocks of all problems, eight epilogue warps.
//   bucket   stable counting sort of the tokens of a problem by cluster: counts, offsets and
//            the member list in ascending token order (deterministic, no global atomics).
//   update   a warp per run of clusters sums their member rows in list order (fp32), forms the means,
//            optionally L2-normalises, and stores the centroid in the key dtype if the cluster
//            is non-empty.  On the last iteration the same pass also produces the value sums
//            and writes the cluster-contiguous copy of K and V.
//
// A "problem" is one (group, segment) pair during the segmented iterations and one group
// during the last, global iteration (reference: cache_hub/kmeans.py:240-250).
#include <cuda.h>
#include <stdio.h>
#include <stdlib.h>

#include <cooperative_groups.h>

#include "ri_common.cuh"
#include "ri_tc.cuh"

namespace {

using namespace ri_tc;
namespace cg = cooperative_groups;

constexpr int kTileM = 128;       // tokens per CTA tile
constexpr int kTileN = 128;       // centroids per MMA tile
constexpr int kHalfBytes = kTileM * 128;   // one K-block (64 channels) of a 128-row tile: 16 KB

// ---- assign ---------------------------------------------------------------------------------
struct AssignArgs {
  int32_t* assign;       // [total tokens] local centroid index of each token within its problem
  int* error_flag;       // set to 1 if a bounded wait ran out
  int n_tok;             // tokens per problem
  int n_cen;             // centroids per problem
  int seg_per_group;     // problems per group
  int64_t group_stride;  // token rows per group (N)
  uint32_t idesc;
};

// ---- assign kernel --------------------------------------------------------------------------------
// A persistent CTA works through consecutive 256-token blocks of the flat sequence over all problems.  Per block
// two 128-row token tiles (A, double-buffered per block) meet every centroid tile (B, streamed
// through three stages) in two MMAs, so a centroid tile fetched into shared memory serves 256 tokens
// and the CTA's set-up is paid once for all its blocks; the accumulators fill all 512 TMEM columns
// (2 buffers x 2 token tiles x 128 centroids).  Ten warps: TMA producer, MMA issuer, and eight
// epilogue warps (four per token tile, one per TMEM lane quarter) that keep the running arg-max
// of their 32 tokens: per 32 columns a max tree, the values of the winning block kept; once per token, behind the last tile,
// the first kept value equal to the max gives the column (ties -> lowest index, the rule of torch.argmax).
// Every mbarrier wait has a time and an iteration limit; on expiry the CTA records where it gave up, releases its
// TMEM and returns.
constexpr int kEpilogueWarps = 8;
constexpr int kWideThreads = 64 + 32 * kEpilogueWarps;
constexpr int kWideBStages = 3;
constexpr uint32_t kWideTmemCols = 512;
// The dynamic block is all the shared memory there is, so that it starts on the 1024-byte boundary that tiles with the
// 128-byte swizzle need: the small arrays stand behind the tiles.
constexpr int kSmallBytes = 256 + 16;      // barriers, then TMEM base, abort and skip words
constexpr int kWideTiles = 2 * 4 * kHalfBytes /*A: 2 blocks x 2 tiles*/ + kWideBStages * 2 * kHalfBytes /*B*/;
constexpr int kWideSmem = kWideTiles + kSmallBytes;

struct WideArgs {
  AssignArgs a;
  int n_units;           // units of work over all problems: blocks of 256 tokens (wide) or tiles of 128 (resident)
  int per_problem;       // units of one problem
};
// A persistent CTA's share: units [lo, hi) of the flat sequence over problems, so that the CTAs differ by one unit at most.
__device__ __forceinline__ void unit_share(const WideArgs& w, int& lo, int& hi) {
  lo = (int)((int64_t)w.n_units * blockIdx.x / gridDim.x);
  hi = (int)((int64_t)w.n_units * (blockIdx.x + 1) / gridDim.x);
}
// first token row (of all groups' rows) of a problem
__device__ __forceinline__ int64_t problem_row(const AssignArgs& a, int problem) {
  return (int64_t)(problem / a.seg_per_group) * a.group_stride + (int64_t)(problem % a.seg_per_group) * a.n_tok;
}

// Running arg-max of a token over blocks of 32 accumulator columns.  Which column of a block is the maximum is not looked
// for in every block that raises it (with 32 tokens in a warp nearly every block does for one of them, and a search costs
// several times the maximum itself): the 32 values of the winning block are kept, by 16 packed moves, and searched once,
// in `index`.  The first column equal to the maximum wins, as with torch.argmax.
struct RunningMax {
  float best;
  int base;              // first column of the winning block
  uint64_t kept[16];     // its values

  __device__ __forceinline__ void reset() {
    best = -INFINITY;
    base = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) kept[i] = 0ull;
  }
  // FULL: all 32 columns exist
  template <bool FULL>
  __device__ __forceinline__ void take(const uint32_t (&r)[32], int col_base, int valid) {
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = FULL || i < valid ? __uint_as_float(r[i]) : -INFINITY;
    float m11[11];
#pragma unroll
    for (int i = 0; i < 10; ++i) m11[i] = max3(v[3 * i], v[3 * i + 1], v[3 * i + 2]);
    m11[10] = fmaxf(v[30], v[31]);
    const float a0 = max3(m11[0], m11[1], m11[2]), a1 = max3(m11[3], m11[4], m11[5]), a2 = max3(m11[6], m11[7], m11[8]);
    const float m = max3(max3(a0, a1, a2), m11[9], m11[10]);
    const bool raise = m > best;             // strict: an equal value in a later block never replaces an earlier one
    if (__any_sync(0xffffffffu, raise)) {
      // two values per instruction on the FMA pipe: v + (-0) is v
      const uint64_t neg_zero = 0x8000000080000000ull;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\t@p add.rn.f32x2 %0, %1, %2;\n\t}"
            : "+l"(kept[i]) : "l"(pack_f2(v[2 * i], v[2 * i + 1])), "l"(neg_zero), "r"((int)raise));
      best = raise ? m : best;
      base = raise ? col_base : base;
    }
  }
  __device__ __forceinline__ int index() const {
    // once per token: plain comparisons, right for infinite and for very small scores too
    int first = 0;
#pragma unroll
    for (int i = 15; i >= 0; --i) {
      float lo, hi;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(kept[i]));
      if (hi == best) first = 2 * i + 1;
      if (lo == best) first = 2 * i;
    }
    return best > -INFINITY ? base + first : 0;
  }
  // one finished accumulator tile (128 columns) of this warp's TMEM lanes; 32 columns are on their way while others are reduced
  template <bool FULL>
  __device__ __forceinline__ void take_tile(uint32_t taddr, int col0, int valid) {
    uint32_t r0[32], r1[32], r2[32];
    tc_ld32(taddr, r0);
    tc_ld32(taddr + 32, r1);
    tc_wait_ld();
    tc_ld_landed(r0);
    tc_ld_landed(r1);
    tc_ld32(taddr + 64, r2);
    take<FULL>(r0, col0, valid);
    take<FULL>(r1, col0 + 32, valid - 32);
    tc_wait_ld();
    tc_ld_landed(r2);
    tc_ld32(taddr + 96, r0);
    take<FULL>(r2, col0 + 64, valid - 64);
    tc_wait_ld();
    tc_ld_landed(r0);
    take<FULL>(r0, col0 + 96, valid - 96);
  }
};

__global__ void __launch_bounds__(kWideThreads, 1)
kmeans_assign_wide_kernel(const __grid_constant__ CUtensorMap map_keys, const __grid_constant__ CUtensorMap map_cent,
                          WideArgs w) {
  const AssignArgs& a = w.a;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t sA = base;                                         // [block parity][tile][K half]
  const uint32_t sB = base + 2 * 4 * kHalfBytes;                    // [stage][K half]
  const uint32_t bars = sB + kWideBStages * 2 * kHalfBytes;
  auto bar_a_full = [&](int s) { return bars + 8u * s; };
  auto bar_a_empty = [&](int s) { return bars + 8u * (2 + s); };
  auto bar_b_full = [&](int s) { return bars + 8u * (4 + s); };
  auto bar_b_empty = [&](int s) { return bars + 8u * (4 + kWideBStages + s); };
  auto bar_acc_full = [&](int b) { return bars + 8u * (4 + 2 * kWideBStages + b); };
  auto bar_acc_empty = [&](int b) { return bars + 8u * (6 + 2 * kWideBStages + b); };
  uint32_t& s_tmem_base = *reinterpret_cast<uint32_t*>(smem_raw + kWideTiles + 256);
  int& s_abort = *reinterpret_cast<int*>(smem_raw + kWideTiles + 260);
  int& s_skip = *reinterpret_cast<int*>(smem_raw + kWideTiles + 264);

  // once any CTA of this launch has given up, the rest leave at once (uniformly per CTA)
  if (threadIdx.x == 0) {
    s_skip = *reinterpret_cast<volatile int*>(a.error_flag);
    if (base & 1023u) *a.error_flag = s_skip = 19;      // the tiles would not lie as the descriptors say
  }
  __syncthreads();
  if (s_skip) {              // not before the kernel in front has ended: the one behind waits for this grid alone
    ri_pdl_wait();
    return;
  }

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int unit_lo, unit_hi;                             // this CTA's 256-token blocks
  unit_share(w, unit_lo, unit_hi);
  const int nb = unit_hi - unit_lo;                 // > 0 by the grid's construction
  const int n_tiles = (a.n_cen + kTileN - 1) / kTileN;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < 2; ++s) { mbar_init(bar_a_full(s), 1); mbar_init(bar_a_empty(s), 1); }
    for (int s = 0; s < kWideBStages; ++s) { mbar_init(bar_b_full(s), 1); mbar_init(bar_b_empty(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(bar_acc_full(b), 1); mbar_init(bar_acc_empty(b), kEpilogueWarps); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                 "r"(kWideTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = s_tmem_base;
  volatile int* abort_flag = &s_abort;
  ri_pdl_wait();           // launched programmatically: the set-up above runs under the kernel before

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int a_issued = 0, b_issued = 0;
      auto load_a = [&](int blk) {          // both token tiles of a block: 4 boxes of 128 rows x 64 channels
        const int sa = blk & 1;
        if (!mbar_wait(bar_a_empty(sa), ((blk >> 1) & 1) ^ 1, abort_flag, 11)) return false;
        mbar_arrive_expect_tx(bar_a_full(sa), 4 * kHalfBytes);
        const int unit = unit_lo + blk, problem = unit / w.per_problem;
        const int row = (int)(problem_row(a, problem) + (int64_t)(unit - problem * w.per_problem) * 2 * kTileM);
#pragma unroll
        for (int tile = 0; tile < 2; ++tile) {
          tma_load_2d(sA + (sa * 4 + tile * 2) * kHalfBytes, &map_keys, bar_a_full(sa), 0, row + tile * kTileM);
          tma_load_2d(sA + (sa * 4 + tile * 2 + 1) * kHalfBytes, &map_keys, bar_a_full(sa), 64, row + tile * kTileM);
        }
        a_issued = blk + 1;
        return true;
      };
      bool ok = load_a(0);
      for (int blk = 0; ok && blk < nb; ++blk) {
        const int cen_row0 = (unit_lo + blk) / w.per_problem * a.n_cen;
        for (int t = 0; ok && t < n_tiles; ++t) {
          const int s = b_issued % kWideBStages;
          ok = mbar_wait(bar_b_empty(s), ((b_issued / kWideBStages) & 1) ^ 1, abort_flag, 12);
          if (!ok) break;
          mbar_arrive_expect_tx(bar_b_full(s), 2 * kHalfBytes);
          tma_load_2d(sB + s * 2 * kHalfBytes, &map_cent, bar_b_full(s), 0, cen_row0 + t * kTileN);
          tma_load_2d(sB + s * 2 * kHalfBytes + kHalfBytes, &map_cent, bar_b_full(s), 64, cen_row0 + t * kTileN);
          ++b_issued;
          if (t == 0 && blk + 1 < nb) ok = load_a(blk + 1);   // the next block's tokens, well ahead of their use
        }
      }
      if (*abort_flag) {
        // give our own copies still in flight a bounded chance to land before the CTA exits
        for (int blk = max(0, a_issued - 2); blk < a_issued; ++blk)
          mbar_wait(bar_a_full(blk & 1), (blk >> 1) & 1, abort_flag, 16);
        for (int j = max(0, b_issued - kWideBStages); j < b_issued; ++j)
          mbar_wait(bar_b_full(j % kWideBStages), (j / kWideBStages) & 1, abort_flag, 17);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int j = 0;                       // centroid tiles issued so far (accumulator buffer = j & 1, B stage = j % 3)
      bool ok = true;
      for (int blk = 0; ok && blk < nb; ++blk) {
        const int sa = blk & 1;
        ok = mbar_wait(bar_a_full(sa), (blk >> 1) & 1, abort_flag, 13);
        for (int t = 0; ok && t < n_tiles; ++t, ++j) {
          const int s = j % kWideBStages, buf = j & 1;
          ok = mbar_wait(bar_b_full(s), (j / kWideBStages) & 1, abort_flag, 14) &&
               mbar_wait(bar_acc_empty(buf), ((j >> 1) & 1) ^ 1, abort_flag, 15);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int tile = 0; tile < 2; ++tile) {
            const uint32_t d_tmem = tmem_base + buf * 2 * kTileN + tile * kTileN;
#pragma unroll
            for (int kb = 0; kb < 2; ++kb) {
              const uint64_t da = umma_desc_sw128(sA + (sa * 4 + tile * 2 + kb) * kHalfBytes);
              const uint64_t db = umma_desc_sw128(sB + s * 2 * kHalfBytes + kb * kHalfBytes);
#pragma unroll
              for (int k = 0; k < 4; ++k)   // K16 steps: 32 bytes along the swizzled row = +2 in the address field
                tc_mma_f16(d_tmem, da + 2 * k, db + 2 * k, a.idesc, (kb | k) != 0);
            }
          }
          tc_commit(bar_b_empty(s));     // the stage is free once these MMAs have read it
          tc_commit(bar_acc_full(buf));  // and both accumulators of the buffer are complete
        }
        if (ok) tc_commit(bar_a_empty(sa));   // the block's token tiles are free once all its MMAs have read them
      }
    }
  } else {
    // ---------------- epilogue: running arg-max over the centroid tiles ----------------
    const int tile = (warp - 2) >> 2;                // which token tile of the block
    const int lane_group = warp & 3;                 // TMEM lanes 32*lane_group .. +31 (a warp may touch only its quarter)
    const int row = tile * kTileM + lane_group * 32 + lane;
    int j = 0;
    bool ok = true;
    for (int blk = 0; ok && blk < nb; ++blk) {
      RunningMax run;
      run.reset();
      for (int t = 0; ok && t < n_tiles; ++t, ++j) {
        const int buf = j & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(bar_acc_full(buf), (j >> 1) & 1, abort_flag, 18));   // warp-uniform
        if (!ok) break;
        tc_fence_after();
        const int col0 = t * kTileN, valid = a.n_cen - col0;
        const uint32_t taddr = tmem_base + ((uint32_t)(lane_group * 32) << 16) + buf * 2 * kTileN + tile * kTileN;
        if (valid >= kTileN) run.take_tile<true>(taddr, col0, kTileN);
        else run.take_tile<false>(taddr, col0, valid);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_acc_empty(buf));
      }
      const int unit = unit_lo + blk, problem = unit / w.per_problem;
      const int local_tok = (unit - problem * w.per_problem) * 2 * kTileM + row;
      if (ok && local_tok < a.n_tok) a.assign[problem_row(a, problem) + local_tok] = run.index();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && s_abort) *a.error_flag = s_abort;   // which wait gave up (see mbar_wait call sites)
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kWideTmemCols));
  }
}

// ---- assign kernel, centroids resident ----------------------------------------------------------------
// Problems of at most 512 centroids (the segmented iterations of the reference's schedule, the re-index build): the
// problem's centroid tiles (up to four, 128 KB) are fetched once per CTA and problem and stay in shared memory, and only the
// tokens stream, as single 128-row tiles through a three-slot ring (the wide kernel above re-fetches the centroid
// tiles for every 256 tokens).  Per token tile two rounds of two centroid tiles each (accumulators: 2 buffers x
// 2 centroid tiles x 128 columns); the eight epilogue warps are four lane quarters x the two centroid tiles of a
// round, so a token's running arg-max lives in two warps, which meet through shared memory once per token tile
// (equal maxima: the lower index wins, as within a warp).  Every warp runs a fixed number of token tiles and rounds
// whatever its waits return, so the named barrier of that merge is always reached.
// CTAs are persistent, one per SM, each with an even run of token tiles over all problems.  The two centroid tiles of a round
// are one product of N 256: as two of N 128 they read the token tile twice, and shared memory, which the operands of an N 128
// product fill to the last byte a clock, held the tensor pipe up (8 heads x 128K rows: 164 -> 134 us a segmented launch).
// Measured and left out, with the two products: sixteen epilogue warps instead of eight (176 against 162 us), token tiles asked
// for in L2 ten tiles ahead (no change), the first tokens loaded under the kernel before (slower).
constexpr int kResSlots = 3;
constexpr int kResTiles = 4 * 2 * kHalfBytes /*B: 4 tiles*/ + kResSlots * 2 * kHalfBytes /*A ring*/;
constexpr int kResSmem = kResTiles + kSmallBytes + 2 * kTileM * 6 /*merge of a token's two warps*/;

__global__ void __launch_bounds__(kWideThreads, 1)
kmeans_assign_resident_kernel(const __grid_constant__ CUtensorMap map_keys, const __grid_constant__ CUtensorMap map_cent,
                              WideArgs w) {
  const AssignArgs& a = w.a;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t sB = base;                                         // [round][K half][centroid tile]
  const uint32_t sA = base + 4 * 2 * kHalfBytes;                    // [slot][K half]
  const uint32_t bars = sA + kResSlots * 2 * kHalfBytes;
  auto bar_a_full = [&](int s) { return bars + 8u * s; };
  auto bar_a_empty = [&](int s) { return bars + 8u * (kResSlots + s); };
  const uint32_t bar_b_full = bars + 8u * (2 * kResSlots);
  const uint32_t bar_b_empty = bars + 8u * (2 * kResSlots + 1);
  auto bar_acc_full = [&](int b) { return bars + 8u * (2 * kResSlots + 2 + b); };
  auto bar_acc_empty = [&](int b) { return bars + 8u * (2 * kResSlots + 4 + b); };
  uint32_t& s_tmem_base = *reinterpret_cast<uint32_t*>(smem_raw + kResTiles + 256);
  int& s_abort = *reinterpret_cast<int*>(smem_raw + kResTiles + 260);
  int& s_skip = *reinterpret_cast<int*>(smem_raw + kResTiles + 264);
  float (*s_best)[kTileM] = reinterpret_cast<float (*)[kTileM]>(smem_raw + kResTiles + kSmallBytes);   // [2][kTileM]
  uint16_t (*s_idx)[kTileM] = reinterpret_cast<uint16_t (*)[kTileM]>(s_best + 2);     // <= 512 centroids: 16 bits

  if (threadIdx.x == 0) {
    s_skip = *reinterpret_cast<volatile int*>(a.error_flag);
    if (base & 1023u) *a.error_flag = s_skip = 19;      // the tiles would not lie as the descriptors say
  }
  __syncthreads();
  if (s_skip) {              // not before the kernel in front has ended: the one behind waits for this grid alone
    ri_pdl_wait();
    return;
  }

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int unit_lo, unit_hi;                             // this CTA's 128-token tiles, over one problem or more
  unit_share(w, unit_lo, unit_hi);
  const int n_tiles = (a.n_cen + kTileN - 1) / kTileN;              // 1 .. 4
  const int rounds = (n_tiles + 1) / 2;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < kResSlots; ++s) { mbar_init(bar_a_full(s), 1); mbar_init(bar_a_empty(s), 1); }
    mbar_init(bar_b_full, 1);
    mbar_init(bar_b_empty, 1);
    for (int b = 0; b < 2; ++b) { mbar_init(bar_acc_full(b), 1); mbar_init(bar_acc_empty(b), kEpilogueWarps); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                 "r"(kWideTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = s_tmem_base;
  volatile int* abort_flag = &s_abort;
  ri_pdl_wait();           // launched programmatically: the set-up above runs under the kernel before

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int issued = 0, loaded = 0;                   // token tiles, problems
      bool ok = true;
      for (int unit = unit_lo; ok && unit < unit_hi;) {
        const int problem = unit / w.per_problem, end = min(unit_hi, (problem + 1) * w.per_problem);
        const int64_t row0 = problem_row(a, problem);
        ok = mbar_wait(bar_b_empty, (loaded & 1) ^ 1, abort_flag, 20);      // the last problem's centroids are done with
        if (!ok) break;
        mbar_arrive_expect_tx(bar_b_full, n_tiles * 2 * kHalfBytes);
        for (int t = 0; t < n_tiles; ++t) {
          // the two tiles of a round behind one another in either half: 256 rows for one product
          const uint32_t dst = sB + ((t >> 1) * 4 + (t & 1)) * kHalfBytes;
          tma_load_2d(dst, &map_cent, bar_b_full, 0, problem * a.n_cen + t * kTileN);
          tma_load_2d(dst + 2 * kHalfBytes, &map_cent, bar_b_full, 64, problem * a.n_cen + t * kTileN);
        }
        ++loaded;
        for (; ok && unit < end; ++unit) {
          const int s = issued % kResSlots;
          ok = mbar_wait(bar_a_empty(s), ((issued / kResSlots) & 1) ^ 1, abort_flag, 21);
          if (!ok) break;
          mbar_arrive_expect_tx(bar_a_full(s), 2 * kHalfBytes);
          const int row = (int)(row0 + (int64_t)(unit - problem * w.per_problem) * kTileM);
          tma_load_2d(sA + s * 2 * kHalfBytes, &map_keys, bar_a_full(s), 0, row);
          tma_load_2d(sA + s * 2 * kHalfBytes + kHalfBytes, &map_keys, bar_a_full(s), 64, row);
          ++issued;
        }
      }
      if (*abort_flag) {
        // give our own copies still in flight a bounded chance to land before the CTA exits
        if (loaded > 0) mbar_wait(bar_b_full, (loaded - 1) & 1, abort_flag, 26);
        for (int u = max(0, issued - kResSlots); u < issued; ++u)
          mbar_wait(bar_a_full(u % kResSlots), (u / kResSlots) & 1, abort_flag, 27);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      bool ok = true;
      int j = 0, u = 0, problem = -1, used = 0;     // rounds issued (accumulator buffer = j & 1), token tiles, problems
      for (int unit = unit_lo; ok && unit < unit_hi; ++unit, ++u) {
        const int s = u % kResSlots;
        if (unit / w.per_problem != problem) {
          problem = unit / w.per_problem;
          ok = mbar_wait(bar_b_full, used & 1, abort_flag, 22);
          ++used;
        }
        ok = ok && mbar_wait(bar_a_full(s), (u / kResSlots) & 1, abort_flag, 23);
        for (int r = 0; ok && r < rounds; ++r, ++j) {
          const int buf = j & 1;
          ok = mbar_wait(bar_acc_empty(buf), ((j >> 1) & 1) ^ 1, abort_flag, 24);
          if (!ok) break;
          tc_fence_after();
          // both centroid tiles of the round as one product of N 256 (the token tile is read once for the two)
          const uint32_t idesc = 2 * r + 1 < n_tiles ? a.idesc + ((uint32_t)(kTileN >> 3) << 17) : a.idesc;
#pragma unroll
          for (int kb = 0; kb < 2; ++kb) {
            const uint64_t da = umma_desc_sw128(sA + (s * 2 + kb) * kHalfBytes);
            const uint64_t db = umma_desc_sw128(sB + (r * 2 + kb) * 2 * kHalfBytes);
#pragma unroll
            for (int k = 0; k < 4; ++k) tc_mma_f16(tmem_base + buf * 2 * kTileN, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
          }
          tc_commit(bar_acc_full(buf));
        }
        if (ok) {
          tc_commit(bar_a_empty(s));         // the token tile is free once all its MMAs have read it
          if (unit + 1 < unit_hi && (unit + 1) / w.per_problem != problem) tc_commit(bar_b_empty);
        }
      }
    }
  } else {
    // ---------------- epilogue: running arg-max, two warps per token ----------------
    const int part = (warp - 2) >> 2;                // which centroid tile of a round
    const int lane_group = warp & 3;                 // TMEM lanes 32*lane_group .. +31 (a warp may touch only its quarter)
    const int row = lane_group * 32 + lane;          // this lane's token within the tile
    int j = 0;
    bool ok = true;
    for (int unit = unit_lo; unit < unit_hi; ++unit) {   // fixed trip counts: the barrier below must be reached by all
      RunningMax run;
      run.reset();
      for (int r = 0; r < rounds; ++r, ++j) {
        const int buf = j & 1;
        ok = ok && __all_sync(0xffffffffu, mbar_wait(bar_acc_full(buf), (j >> 1) & 1, abort_flag, 25));   // warp-uniform
        const int col0 = (2 * r + part) * kTileN, valid = a.n_cen - col0;
        if (ok && valid > 0) {
          tc_fence_after();
          const uint32_t taddr = tmem_base + ((uint32_t)(lane_group * 32) << 16) + buf * 2 * kTileN + part * kTileN;
          if (valid >= kTileN) run.take_tile<true>(taddr, col0, kTileN);
          else run.take_tile<false>(taddr, col0, valid);
          tc_fence_before();
        }
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(bar_acc_empty(buf));
      }
      // the two warps of a token meet (buffers alternate per token tile, so one barrier per tile is enough)
      const int par = unit & 1;
      int best_idx = run.index();
      if (part == 1) { s_best[par][row] = run.best; s_idx[par][row] = (uint16_t)best_idx; }
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpilogueWarps) : "memory");
      if (part == 0) {
        const float ob = s_best[par][row];
        const int oi = (int)s_idx[par][row];
        if (ob > run.best || (ob == run.best && oi < best_idx)) best_idx = oi;
        const int problem = unit / w.per_problem, local_tok = (unit - problem * w.per_problem) * kTileM + row;
        if (ok && local_tok < a.n_tok) a.assign[problem_row(a, problem) + local_tok] = best_idx;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && s_abort) *a.error_flag = s_abort;   // which wait gave up (see mbar_wait call sites)
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kWideTmemCols));
  }
}

// Rows of 128 channels that are not necessarily one behind the other: row r of group z starts at
// (z * group + r * row) 256-byte units.
struct RowPlace { int64_t group, row; };

// ---- centre ---------------------------------------------------------------------------------
constexpr int kMeanRows = 2048;   // rows per partial-sum CTA

template <int DT>
__global__ void __launch_bounds__(256) colsum_partial_kernel(const uint4* __restrict__ keys, RowPlace src,
                                                             float* __restrict__ partial, int n_tok, int chunks) {
  const int z = blockIdx.y, chunk = blockIdx.x;
  const int piece = threadIdx.x & 15, rl = threadIdx.x >> 4;   // 16 pieces of 8 channels x 16 row lanes
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const int r0 = chunk * kMeanRows, r1 = min(n_tok, r0 + kMeanRows);
  constexpr int kAhead = 8;          // rows in flight per thread; they are added in row order
  auto add = [&](const uint4& v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[2 * i] += Elem<DT>::from_bits((uint16_t)(w[i] & 0xffffu));
      acc[2 * i + 1] += Elem<DT>::from_bits((uint16_t)(w[i] >> 16));
    }
  };
  const uint4* from = keys + z * src.group * 16 + piece;
  int r = r0 + rl;
  for (; r + 16 * (kAhead - 1) < r1; r += 16 * kAhead) {
    uint4 v[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[u].x), "=r"(v[u].y), "=r"(v[u].z), "=r"(v[u].w)
                   : "l"(from + (r + 16 * u) * src.row * 16));
#pragma unroll
    for (int u = 0; u < kAhead; ++u) add(v[u]);
  }
  for (; r < r1; r += 16) add(ri_ldg16(from + r * src.row * 16));
  __shared__ float red[16][128];
#pragma unroll
  for (int i = 0; i < 8; ++i) red[rl][piece * 8 + i] = acc[i];
  __syncthreads();
  if (threadIdx.x < 128) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) s += red[k][threadIdx.x];
    partial[((int64_t)z * chunks + chunk) * 128 + threadIdx.x] = s;
  }
}

template <int DT>
__global__ void colmean_final_kernel(const float* __restrict__ partial, uint16_t* __restrict__ mean, int n_tok, int chunks) {
  const int z = blockIdx.x, c = threadIdx.x;
  float s = 0.f;
  for (int k = 0; k < chunks; ++k) s += partial[((int64_t)z * chunks + k) * 128 + c];
  mean[z * 128 + c] = Elem<DT>::bits(s / (float)n_tok);
}

template <int DT>
__global__ void __launch_bounds__(256) centre_apply_kernel(const uint4* __restrict__ keys, RowPlace src,
                                                           const uint16_t* __restrict__ mean, uint4* __restrict__ out,
                                                           int64_t pieces_per_group) {
  const int z = blockIdx.y;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pieces_per_group) return;
  const int piece = (int)(i & 15);
  const uint4 v = ri_ldg16(keys + (z * src.group + (i >> 4) * src.row) * 16 + piece);
  const uint4 m = *reinterpret_cast<const uint4*>(mean + z * 128 + piece * 8);
  const uint32_t vw[4] = {v.x, v.y, v.z, v.w}, mw[4] = {m.x, m.y, m.z, m.w};
  uint32_t ow[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float lo = Elem<DT>::from_bits((uint16_t)(vw[k] & 0xffffu)) - Elem<DT>::from_bits((uint16_t)(mw[k] & 0xffffu));
    const float hi = Elem<DT>::from_bits((uint16_t)(vw[k] >> 16)) - Elem<DT>::from_bits((uint16_t)(mw[k] >> 16));
    ow[k] = Elem<DT>::pack2(lo, hi);
  }
  out[(int64_t)z * pieces_per_group + i] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
}

// ---- initial centroids (cache_hub/kmeans.py:234-237: index arithmetic in float32) -------------
__global__ void init_centroids_kernel(const uint4* __restrict__ centred, uint4* __restrict__ cent, int n_tok, int n_cen,
                                      float step, float half) {
  const int z = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;   // one 16-byte piece
  if (i >= n_cen * 16) return;
  const int c = i >> 4, piece = i & 15;
  const long long idx = (long long)__fadd_rn(__fmul_rn((float)c, step), half);
  const long long row = idx < 0 ? 0 : (idx >= n_tok ? n_tok - 1 : idx);
  cent[((int64_t)z * n_cen + c) * 16 + piece] = ri_ldg16(centred + ((int64_t)z * n_tok + row) * 16 + piece);
}

// ---- bucket ---------------------------------------------------------------------------------
struct BucketArgs {
  const int32_t* assign;   // [total tokens] local centroid ids
  int32_t* order;          // [total tokens] local token ids, cluster-major, ascending inside a cluster
  int32_t* count;          // [problems, n_cen]
  int32_t* offset;         // [problems, n_cen + 1]
  int n_tok, n_cen, seg_per_group;
  int64_t group_stride;
  int range;               // tokens per warp
};

// The form for what the kernel below does not take (more than about 20000 clusters or 480000 tokens per problem): one CTA
// per problem, 32-bit counts.  The tokens are cut into `workers` contiguous ranges; a table [workers][n_cen] first holds
// how many tokens of each range fall into each cluster, then (after the scan of the totals) where each range
// starts writing inside each cluster, so that `workers` warps can scatter their ranges side by side and the
// order inside a cluster is still ascending in the token id.
__global__ void __launch_bounds__(1024) kmeans_bucket_one_cta_kernel(BucketArgs a, int workers) {
  extern __shared__ int32_t bucket_smem[];
  int32_t* cursor = bucket_smem;                 // [n_cen]: counts, then first positions
  int32_t* table = workers == 1 ? bucket_smem : bucket_smem + a.n_cen;   // [workers][n_cen]; one range: the same array
  __shared__ uint32_t warp_sums[32];
  __shared__ uint32_t s_carry;
  const int problem = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t tok0 = (int64_t)(problem / a.seg_per_group) * a.group_stride + (int64_t)(problem % a.seg_per_group) * a.n_tok;
  const int32_t* asg = a.assign + tok0;
  const int chunk = ((a.n_tok + workers - 1) / workers + 31) & ~31;     // tokens per range, whole warp steps
  for (int i = tid; i < a.n_cen * (workers == 1 ? 1 : workers + 1); i += 1024) bucket_smem[i] = 0;
  if (tid == 0) s_carry = 0;
  __syncthreads();
  auto clamp_id = [&](int32_t c) { return min(max(c, 0), a.n_cen - 1); };   // never index outside the table
  for (int t = tid; t < a.n_tok; t += 1024) {
    const int c = clamp_id(asg[t]);
    atomicAdd(&table[(t / chunk) * a.n_cen + c], 1);
  }
  __syncthreads();
  for (int c = tid; c < a.n_cen; c += 1024) {
    int total = 0;
    for (int w = 0; w < workers; ++w) total += table[w * a.n_cen + c];
    cursor[c] = total;
  }
  __syncthreads();
  // exclusive scan of the counts, 1024 at a time
  for (int c0 = 0; c0 < a.n_cen; c0 += 1024) {
    const int c = c0 + tid;
    const uint32_t v = c < a.n_cen ? (uint32_t)cursor[c] : 0u;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t n = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += n;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    uint32_t ws = warp_sums[lane], winc = ws;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t n = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= o) winc += n;
    }
    const uint32_t carry = s_carry;
    const uint32_t excl = carry + __shfl_sync(0xffffffffu, winc - ws, warp) + inc - v;
    if (c < a.n_cen) {
      a.count[(int64_t)problem * a.n_cen + c] = (int32_t)v;
      a.offset[(int64_t)problem * (a.n_cen + 1) + c] = (int32_t)excl;
      // where each range starts inside this cluster
      uint32_t running = excl;
      for (int w = 0; w < workers; ++w) {
        const int32_t n_w = table[w * a.n_cen + c];
        table[w * a.n_cen + c] = (int32_t)running;
        running += (uint32_t)n_w;
      }
    }
    const uint32_t chunk_total = __shfl_sync(0xffffffffu, winc, 31);   // every lane takes part in the shuffle
    __syncthreads();
    if (tid == 1023) s_carry = carry + chunk_total;
    __syncthreads();
  }
  if (tid == 0) a.offset[(int64_t)problem * (a.n_cen + 1) + a.n_cen] = (int32_t)s_carry;
  __syncthreads();
  // stable scatter: warp w takes range w, 32 tokens at a time in token order
  if (warp >= workers) return;
  int32_t* ord = a.order + tok0;
  int32_t* my_cursor = table + warp * a.n_cen;
  const int t_begin = warp * chunk, t_end = min(a.n_tok, t_begin + chunk);
  constexpr int kAhead = 8;
  for (int t0 = t_begin; t0 < t_end; t0 += 32 * kAhead) {
    int32_t cl[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int t = t0 + u * 32 + lane;
      cl[u] = t < t_end ? clamp_id(asg[t]) : -1;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int t = t0 + u * 32 + lane;
      const unsigned active = __ballot_sync(0xffffffffu, cl[u] >= 0);
      if (cl[u] >= 0) {
        const unsigned peers = __match_any_sync(active, cl[u]);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        const int pos = my_cursor[cl[u]] + rank;
        ord[pos] = t;
        __syncwarp(active);
        if (lane == 31 - __clz(peers)) my_cursor[cl[u]] = pos + 1;
      }
      __syncwarp();
    }
  }
}

// A cluster of CTAs per problem.  The tokens are cut into contiguous ranges, one per warp of the cluster; a table
// [warps of the CTA][n_cen] of 16-bit counts first holds how many tokens of each range fall into each cluster, then how
// many lie in the ranges before it (in this CTA); the CTAs' totals meet through distributed shared memory.  So every warp
// scatters its own range, and the order inside a cluster is still ascending in the token id.
// 8 problems of 131004 tokens and 8192 clusters: 350 us with one CTA per problem, 51 now; 128 problems of 8187 tokens and 512
// clusters: 17 -> 12 us.
template <int CL>
__global__ void __launch_bounds__(512) kmeans_bucket_kernel(BucketArgs a) {
  ri_pdl_trigger();
  extern __shared__ __align__(16) uint8_t sort_smem[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int workers = (int)blockDim.x / 32;
  uint32_t* total = reinterpret_cast<uint32_t*>(sort_smem);              // [n_cen] this CTA's tokens per cluster
  int32_t* base = reinterpret_cast<int32_t*>(total + a.n_cen);             // [n_cen] where this CTA's tokens start
  uint32_t* table32 = reinterpret_cast<uint32_t*>(base + a.n_cen);         // [workers][n_cen] 16-bit counts
  __shared__ uint32_t warp_sums[16];
  const int problem = (int)blockIdx.x / CL, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x;
  const int64_t tok0 = (int64_t)(problem / a.seg_per_group) * a.group_stride + (int64_t)(problem % a.seg_per_group) * a.n_tok;
  const int32_t* asg = a.assign + tok0;
  const int t_begin = min(a.n_tok, (rank * workers + warp) * a.range), t_end = min(a.n_tok, t_begin + a.range);
  for (int i = tid; i < a.n_cen * workers / 2; i += T) table32[i] = 0;     // n_cen is a multiple of 32
  ri_pdl_wait();
  __syncthreads();
  auto clamp_id = [&](int32_t c) { return min(max(c, 0), a.n_cen - 1); };  // never index outside the table
  constexpr int kAhead = 8;
  for (int t0 = t_begin; t0 < t_end; t0 += 32 * kAhead) {
    int32_t cl[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int t = t0 + u * 32 + lane;
      cl[u] = t < t_end ? clamp_id(asg[t]) : -1;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (cl[u] >= 0) atomicAdd(&table32[(warp * a.n_cen + cl[u]) >> 1], (cl[u] & 1) ? 0x10000u : 1u);
  }
  __syncthreads();
  // counts of the ranges before, per cluster pair (packed 16-bit sums: a CTA has fewer than 65536 tokens)
  for (int i = tid; i < a.n_cen / 2; i += T) {
    uint32_t run = 0;
    for (int w = 0; w < workers; ++w) {
      const uint32_t n = table32[(w * a.n_cen >> 1) + i];
      table32[(w * a.n_cen >> 1) + i] = run;
      run += n;
    }
    total[2 * i] = run & 0xffffu;
    total[2 * i + 1] = run >> 16;
  }
  cluster.sync();
  // exclusive scan of the problem's counts over the clusters: a warp takes a contiguous run of them, 32 at a time
  const int per = ((a.n_cen / 32 + workers - 1) / workers) * 32, c_lo = min(a.n_cen, warp * per), c_hi = min(a.n_cen, c_lo + per);
  uint32_t running = 0;
  for (int c0 = c_lo; c0 < c_hi; c0 += 32) {
    const int c = c0 + lane;
    uint32_t all = 0, lower = 0;
#pragma unroll
    for (int r = 0; r < CL; ++r) {
      const uint32_t n = CL == 1 ? total[c] : cluster.map_shared_rank(total, r)[c];
      lower += r < rank ? n : 0u;
      all += n;
    }
    if (rank == 0) a.count[(int64_t)problem * a.n_cen + c] = (int32_t)all;
    uint32_t inc = all;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t n = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += n;
    }
    base[c] = (int32_t)(running + inc - all + lower);      // relative to the warp's first cluster, for now
    running += __shfl_sync(0xffffffffu, inc, 31);
  }
  if (lane == 0) warp_sums[warp] = running;
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < warp; ++w) before += warp_sums[w];
  for (int c = c_lo + lane; c < c_hi; c += 32) {
    base[c] += (int32_t)before;
    if (rank == 0) a.offset[(int64_t)problem * (a.n_cen + 1) + c] = base[c];     // no CTA of lower rank: the cluster's first
  }
  if (rank == 0 && warp == workers - 1 && lane == 0) a.offset[(int64_t)problem * (a.n_cen + 1) + a.n_cen] = (int32_t)(before + running);
  if (CL > 1) cluster_arrive();                   // this CTA's remote reads are over (awaited before it exits)
  __syncthreads();
  // stable scatter: 32 tokens of the warp's range at a time, in token order
  int32_t* ord = a.order + tok0;
  for (int t0 = t_begin; t0 < t_end; t0 += 32 * kAhead) {
    int32_t cl[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int t = t0 + u * 32 + lane;
      cl[u] = t < t_end ? clamp_id(asg[t]) : -1;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int t = t0 + u * 32 + lane;
      // the lane's place behind the tokens of the steps before; lanes that share a cluster with an earlier lane find the
      // counter moved on and are put in token order one cluster after the other (few: __match_any_sync on 32 mostly
      // different clusters took most of this kernel's time)
      const int slot = warp * a.n_cen + max(cl[u], 0), shift = (slot & 1) * 16;
      const uint32_t cur = (table32[slot >> 1] >> shift) & 0xffffu;
      __syncwarp();
      uint32_t old = cur;
      if (cl[u] >= 0) old = (atomicAdd(&table32[slot >> 1], 1u << shift) >> shift) & 0xffffu;
      uint32_t rank_in = 0;
      for (unsigned todo = __ballot_sync(0xffffffffu, old != cur); todo;) {
        const int c = __shfl_sync(0xffffffffu, cl[u], __ffs(todo) - 1);
        const unsigned peers = __ballot_sync(0xffffffffu, cl[u] == c);
        if (cl[u] == c) rank_in = __popc(peers & ((1u << lane) - 1u));
        todo &= ~peers;
      }
      if (cl[u] >= 0) ord[base[cl[u]] + cur + rank_in] = t;
      __syncwarp();
    }
  }
  if (CL > 1) cluster_wait();
}

// Launch plan of the bucket pass: CTAs per problem, warps per CTA, tokens per warp.
struct BucketPlan { int cl, workers; size_t smem; };

BucketPlan bucket_plan(int problems, int n_tok, int n_cen, int sms) {
  BucketPlan p;
  // up to 8 CTAs per problem, as long as all problems together have at most two per SM (with up to about 2800 clusters their
  // tables let two be resident; with more, the larger launches take two rounds)
  p.cl = 8;
  while (p.cl > 1 && p.cl * problems > 2 * sms) p.cl >>= 1;
  // 16-bit counts and packed sums: a CTA's tokens stay below 65536
  while (p.cl < 8 && (n_tok + p.cl - 1) / p.cl > 60000) p.cl <<= 1;
  p.workers = 16;
  auto bytes = [&](int w) { return (size_t)n_cen * (8 + 2 * (size_t)w); };
  while (p.workers > 1 && bytes(p.workers) > 200 * 1024) p.workers >>= 1;
  p.smem = bytes(p.workers);
  return p;
}

template <int CL>
int launch_bucket(BucketArgs a, const BucketPlan& p, int problems, cudaStream_t s) {
  a.range = ((a.n_tok + p.cl * p.workers - 1) / (p.cl * p.workers) + 31) & ~31;
  if (p.smem > 48 * 1024)
    RI_CUDA_OK(cudaFuncSetAttribute(kmeans_bucket_kernel<CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem));
  RI_CUDA_OK(ri_launch_pdl_cluster(9, CL, kmeans_bucket_kernel<CL>, dim3(problems * CL), dim3(p.workers * 32), p.smem, s, a));
  return RI_OK;
}

// ---- update ---------------------------------------------------------------------------------
struct UpdateArgs {
  const uint2* rows;         // rows to average: centred keys, or the raw keys with `mean` to be subtracted (LAST)
  const uint2* values;       // LAST: V rows (value sums + copy)
  RowPlace src;              // place of a row of `rows` and `values`
  const int32_t* order;
  const int32_t* offset;
  uint2* centroids;          // [problems, n_cen, 128] in/out (centred)
  uint2* out_centroids;      // optional final: centroid + mean
  const uint16_t* mean;      // optional [Z, 128]
  uint2* value_sum;          // LAST: [Z, C, 128]
  uint16_t* size_dt;         // LAST: [Z, C]
  uint8_t* empty;            // LAST, optional: [Z, C] whether the cluster has no members
  uint2* keys_out;           // LAST, optional: cluster-contiguous copy, group stride `out_group` rows
  uint2* values_out;
  int64_t out_group;
  int n_tok, n_cen, seg_per_group, normalize;
  int64_t group_stride;
  int clusters_per_warp;
};

template <int DT>
__device__ __forceinline__ void add_row(float (&acc)[4], uint2 v) {
  acc[0] += Elem<DT>::from_bits((uint16_t)(v.x & 0xffffu));
  acc[1] += Elem<DT>::from_bits((uint16_t)(v.x >> 16));
  acc[2] += Elem<DT>::from_bits((uint16_t)(v.y & 0xffffu));
  acc[3] += Elem<DT>::from_bits((uint16_t)(v.y >> 16));
}
template <int DT>
__device__ __forceinline__ uint2 sub_row(uint2 v, uint2 m) {      // round(v - m), channel by channel
  uint2 o;
  o.x = Elem<DT>::pack2(Elem<DT>::from_bits((uint16_t)(v.x & 0xffffu)) - Elem<DT>::from_bits((uint16_t)(m.x & 0xffffu)),
                        Elem<DT>::from_bits((uint16_t)(v.x >> 16)) - Elem<DT>::from_bits((uint16_t)(m.x >> 16)));
  o.y = Elem<DT>::pack2(Elem<DT>::from_bits((uint16_t)(v.y & 0xffffu)) - Elem<DT>::from_bits((uint16_t)(m.y & 0xffffu)),
                        Elem<DT>::from_bits((uint16_t)(v.y >> 16)) - Elem<DT>::from_bits((uint16_t)(m.y >> 16)));
  return o;
}

// A warp takes `clusters_per_warp` consecutive clusters of one problem, lane l the channels 4l .. 4l+3.  Their members are
// one run of the order list, so the rows stream through a ring in shared memory (cp.async, windows of four rows: half a
// warp copies a row in 16-byte pieces) whatever the clusters' sizes, about 15 members as a rule: three windows are on
// their way while one is added.  A cluster's rows are added one after the other in list order, so the sums are those of a
// serial sum (the rows of a window that belong to another cluster add +0, which changes no sum that began at +0).
// A segmented launch of 8 heads x 128K rows: 155 -> 69 us, bound by issue slots (78 %, 45 instructions a row, a third of them
// the divisions and the root at a cluster's end) beside 273 MB from DRAM; fetching count, offset, list and rows of one
// cluster after the other spent its time waiting.
constexpr int kUpdateThreads = 128;
constexpr int kWindow = 4;          // rows per step
constexpr int kWindows = 4;         // steps in the ring

// LONG: clusters of kLongCluster members and more are left to the whole CTA, which sums them when its warps are done with the
// others.  Through the ring such a cluster is one warp's chain of 75 clocks a row, every four rows of which wait, shuffle and
// compare; the CTA streams its rows in batches of 32, two of them ahead of the one that is added (a warp's ring: 12 rows), and a
// thread adds one channel of a row after the other, in the same order.  The initial centroids are rows as they are, and those of
// the longest keys may win most of a segment: the first two updates are launched in this form, the later ones without it.  Whole
// builds against all updates without it (us, B200): 8 heads x 128K rows 3979 -> 3782, 4 x 20K 835 -> 566, 8 x 17K fp16 894 -> 662;
// where no cluster is long 2420 -> 2417 (8 x 91K) and 1915 -> 1913 (8 x 75K).  Three batches are 24 KB, nine CTAs an SM; with five
// (40 KB, five CTAs) the last two took 2441 and 1939, the others no less; with four of 16 rows 8 x 17K took 680.  For the second
// update alone: 4 x 32K fp16 847 instead of 761, 2 x 59K 652 instead of 622.
constexpr int kLongCluster = 512;
constexpr int kLongRows = 32;       // rows of a batch
constexpr int kLongBatches = 3;     // batches in shared memory

template <int DT, bool LAST, bool LONG>
__global__ void __launch_bounds__(kUpdateThreads) kmeans_update_kernel(UpdateArgs a) {
  ri_pdl_enter();
  constexpr int kWarps = kUpdateThreads / 32, kRowsBytes = kWindows * kWindow * 256;
  static_assert(!(LAST && LONG) && kLongBatches * kLongRows * 256 >= kWarps * kRowsBytes, "the batches lie over the warps' rings");
  __shared__ __align__(16) uint8_t ring[kWarps][LONG ? kLongBatches * kLongRows * 256 / kWarps : (LAST ? 2 : 1) * kRowsBytes];
  __shared__ int s_long[LONG ? kWarps : 1][3];                // per warp: a long cluster's place in its run, first member, end
  __shared__ float s_sum[LONG ? 128 : 1];
  const int lane = threadIdx.x & 31;
  const int job = (int)blockIdx.x * kWarps + (int)(threadIdx.x >> 5);
  // n_cen is a multiple of 32 and clusters_per_warp 1, 2, 4 or 8: the warps of a CTA all have clusters, and of one problem
  const int idx0 = job * a.clusters_per_warp;
  const int problem = idx0 / a.n_cen, z = problem / a.seg_per_group;
  int c = idx0 - problem * a.n_cen;
  const int tok_in_group = (problem - z * a.seg_per_group) * a.n_tok;
  const int32_t* off = a.offset + (int64_t)problem * (a.n_cen + 1) + c;
  // ends of this warp's clusters (at most 32), one per lane
  const int my_end = off[min(lane, a.clusters_per_warp - 1) + 1];
  const int first = off[0];
  const int last = __shfl_sync(0xffffffffu, my_end, a.clusters_per_warp - 1);
  const int32_t* ord = a.order + (int64_t)z * a.group_stride + tok_in_group;
  const int half = lane >> 4;                                 // copies the first or the second row of a step
  const int64_t src0 = ((int64_t)z * a.src.group + (int64_t)tok_in_group * a.src.row) * 16 + (lane & 15);   // 16-byte pieces
  const int64_t row_step = a.src.row * 16;
  uint2 mean = make_uint2(0u, 0u);
  if (a.mean) mean = *reinterpret_cast<const uint2*>(a.mean + z * 128 + lane * 4);

  float ks[4] = {0, 0, 0, 0}, vs[4] = {0, 0, 0, 0};
  int done = 0, end = __shfl_sync(0xffffffffu, my_end, 0), start = first;
  auto finish = [&]() {       // cluster c + done is complete
    const int cnt = end - start;
    const int64_t cl = (int64_t)problem * a.n_cen + c + done, crow = cl * 32 + lane;
    if (LAST) {
      if (a.size_dt) a.size_dt[cl] = Elem<DT>::bits((float)cnt);
      if (a.empty) a.empty[cl] = cnt == 0;
      if (a.value_sum) a.value_sum[crow] = make_uint2(Elem<DT>::pack2(vs[0], vs[1]), Elem<DT>::pack2(vs[2], vs[3]));
    }
    uint2 cd;
    if (cnt > 0) {
      const float fc = (float)cnt;
      float x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = ks[i] / fc;
      if (a.normalize) {
        float ss = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float nrm = sqrtf(ss);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = x[i] / nrm;
      }
      cd = make_uint2(Elem<DT>::pack2(x[0], x[1]), Elem<DT>::pack2(x[2], x[3]));
      a.centroids[crow] = cd;
    } else if (LAST && a.out_centroids) {
      cd = a.centroids[crow];
    }
    if (LAST && a.out_centroids) {
      // stored centroid = round(centroid_dt + mean_dt), both already in the key dtype
      // (cache_hub/retroinfer_cache.py:429)
      uint2 o;
      o.x = Elem<DT>::pack2(Elem<DT>::from_bits((uint16_t)(cd.x & 0xffffu)) + Elem<DT>::from_bits((uint16_t)(mean.x & 0xffffu)),
                            Elem<DT>::from_bits((uint16_t)(cd.x >> 16)) + Elem<DT>::from_bits((uint16_t)(mean.x >> 16)));
      o.y = Elem<DT>::pack2(Elem<DT>::from_bits((uint16_t)(cd.y & 0xffffu)) + Elem<DT>::from_bits((uint16_t)(mean.y & 0xffffu)),
                            Elem<DT>::from_bits((uint16_t)(cd.y >> 16)) + Elem<DT>::from_bits((uint16_t)(mean.y >> 16)));
      a.out_centroids[crow] = o;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) { ks[i] = 0.f; vs[i] = 0.f; }
    start = end;
    ++done;
    end = __shfl_sync(0xffffffffu, my_end, min(done, 31));
  };

  // clusters `done` .. to - 1 through the ring, whatever their sizes
  uint8_t* my_ring = ring[threadIdx.x >> 5];
  auto stream = [&](const int to, const int first, const int n) {      // first: their first member, n: how many they have
  const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(my_ring);
  int ids = lane < n ? ord[first + lane] : 0;                 // 32 list entries; the next 32 below
  int ids_next = 32 + lane < n ? ord[first + 32 + lane] : 0;
  int filled = 0;                                             // members asked for so far
  auto fetch = [&]() {
    if (filled < n) {
      const uint32_t dst = ring_s + (filled & (kWindows * kWindow - 1)) * 256 + lane * 16;
#pragma unroll
      for (int u = 0; u < kWindow; u += 2) {
        const int row = __shfl_sync(0xffffffffu, ids, (filled + u + half) & 31);
        if (filled + u + half < n) {
          const int64_t at = src0 + row * row_step;
          cp_async16(dst + u * 256, reinterpret_cast<const uint4*>(a.rows) + at);
          if (LAST) cp_async16(dst + u * 256 + kRowsBytes, reinterpret_cast<const uint4*>(a.values) + at);
        }
      }
      filled += kWindow;
      if ((filled & 31) == 0) {
        ids = ids_next;
        ids_next = filled + 32 + lane < n ? ord[first + filled + 32 + lane] : 0;
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int i = 0; i < kWindows - 1; ++i) fetch();
#pragma unroll 1
  for (int r = 0; r < n; r += kWindow) {
    cp_async_wait<kWindows - 2>();
    __syncwarp();                                             // the other half's rows; and everyone is done with the slots below
    fetch();
    const uint8_t* src = my_ring + (r & (kWindows * kWindow - 1)) * 256 + lane * 8;
    uint2 kv[kWindow], vv[kWindow];
#pragma unroll
    for (int u = 0; u < kWindow; ++u) {
      kv[u] = *reinterpret_cast<const uint2*>(src + u * 256);
      if (LAST) {
        vv[u] = *reinterpret_cast<const uint2*>(src + u * 256 + kRowsBytes);
        if (a.keys_out && r + u < n) {
          const int64_t o = ((int64_t)z * a.out_group + first + r + u) * 32 + lane;
          a.keys_out[o] = kv[u];
          a.values_out[o] = vv[u];
        }
        if (a.mean) kv[u] = sub_row<DT>(kv[u], mean);         // the centred key, rounded as the copy the assignment reads
      }
    }
    int lo = 0;                                               // rows of the window behind the last finished cluster
    for (;;) {
      const int hi = end - first - r;                         // the current cluster's end, from the window's first row
      if (lo == 0 && hi >= kWindow) {
#pragma unroll
        for (int u = 0; u < kWindow; ++u) {
          add_row<DT>(ks, kv[u]);
          if (LAST) add_row<DT>(vs, vv[u]);
        }
      } else {
#pragma unroll
        for (int u = 0; u < kWindow; ++u) {
          const bool in = u >= lo && u < hi;
          add_row<DT>(ks, in ? kv[u] : make_uint2(0u, 0u));
          if (LAST) add_row<DT>(vs, in ? vv[u] : make_uint2(0u, 0u));
        }
      }
      if (hi > kWindow || done == to) break;
      finish();
      lo = hi;
      if (done == to) break;
    }
  }
  while (done < to) finish();
  };
  if (!LONG) {
    stream(a.clusters_per_warp, first, last - first);
    return;
  }
  const int end_before = __shfl_up_sync(0xffffffffu, my_end, 1), my_start = lane > 0 ? end_before : first;
  unsigned todo = __ballot_sync(0xffffffffu, lane < a.clusters_per_warp && my_end - my_start >= kLongCluster);
  for (unsigned rest = todo;; rest &= rest - 1) {
    const int at = rest ? __ffs(rest) - 1 : a.clusters_per_warp;      // the next long one, or the end
    if (done < at) {
      stream(at, start, __shfl_sync(0xffffffffu, my_end, at - 1) - start);
      cp_async_wait<0>();
      __syncwarp();                                           // all lanes are done with the ring: the next stream fills it anew
    }
    if (!rest) break;
    start = end;                                              // not now
    ++done;
    end = __shfl_sync(0xffffffffu, my_end, min(done, 31));
  }
  // the long clusters, one of every warp after the other
  const int warp = threadIdx.x >> 5, tid = threadIdx.x;
  for (;;) {
    const int at = todo ? __ffs(todo) - 1 : -1;
    const int from = __shfl_sync(0xffffffffu, my_start, max(at, 0)), to = __shfl_sync(0xffffffffu, my_end, max(at, 0));
    if (lane == 0) { s_long[warp][0] = at; s_long[warp][1] = from; s_long[warp][2] = to; }
    if (!__syncthreads_or(at >= 0)) break;
    for (int w = 0; w < kWarps; ++w) {
      if (s_long[w][0] < 0) continue;                         // the same for every warp of the CTA
      const int l_from = s_long[w][1], l_n = s_long[w][2] - l_from;
      const int32_t* l_ord = ord + l_from;
      const uint4* l_rows = reinterpret_cast<const uint4*>(a.rows) + src0;
      const uint32_t batch = (uint32_t)__cvta_generic_to_shared(&ring[0][0]);
      constexpr int kCopies = kLongRows * 16 / kUpdateThreads;      // 16-byte pieces of a batch per thread
      int id[kCopies];
      auto list = [&](int r) {                                // of the batch's rows, those whose pieces this thread copies
#pragma unroll
        for (int u = 0; u < kCopies; ++u) id[u] = l_ord[min(r + u * (kUpdateThreads / 16) + (tid >> 4), l_n - 1)];
      };
      auto copy = [&](int r) {
#pragma unroll
        for (int u = 0; u < kCopies; ++u)
          cp_async16(batch + ((r / kLongRows) % kLongBatches) * kLongRows * 256 + (u * kUpdateThreads + tid) * 16, l_rows + id[u] * row_step);
      };
      constexpr int kAhead = (kLongBatches - 1) * kLongRows;
#pragma unroll
      for (int r = 0; r < kAhead; r += kLongRows) {
        list(r);
        copy(r);
        cp_async_commit();
      }
      list(kAhead);
      float sum = 0.f;
      for (int r = 0; r < l_n; r += kLongRows) {
        if (r + kAhead < l_n) copy(r + kAhead);
        cp_async_commit();
        list(r + kAhead + kLongRows);
        cp_async_wait<kLongBatches - 1>();
        __syncthreads();                                      // every thread's pieces of the batch
        const uint16_t* v = reinterpret_cast<const uint16_t*>(&ring[0][0] + ((r / kLongRows) % kLongBatches) * kLongRows * 256) + tid;
        if (r + kLongRows <= l_n) {
#pragma unroll
          for (int u = 0; u < kLongRows; ++u) sum += Elem<DT>::from_bits(v[u * 128]);
        } else {
          for (int u = 0; u < l_n - r; ++u) sum += Elem<DT>::from_bits(v[u * 128]);
        }
        __syncthreads();                                      // the batch may be overwritten
      }
      cp_async_wait<0>();
      s_sum[tid] = sum;
      __syncthreads();
      if (warp == w) {
#pragma unroll
        for (int i = 0; i < 4; ++i) ks[i] = s_sum[lane * 4 + i];
        done = at;
        start = from;
        end = to;
        finish();
        todo &= todo - 1;
      }
      __syncthreads();
    }
    __syncthreads();                                          // the list has been read by all
  }
}

// ---- host side --------------------------------------------------------------------------------
// rows x 128 channels, 16-bit elements, box = 128 rows x 64 channels, 128-byte swizzle
int make_row_map(CUtensorMap* map, const void* base, int64_t rows, int dtype) {
  return make_map_2d(map, base, 128, rows, 256, dtype);
}

struct FitLayout {
  int64_t cent_work, assign, order, count, offset, centred, mean, partial, error, total;
  int chunks;
};

FitLayout fit_layout(const ri_kmeans* p, bool with_centring) {
  FitLayout L;
  int64_t off = 0;
  auto take = [&](int64_t bytes) { int64_t o = off; off = ri_align_up(off + bytes, 1024); return o; };
  const int64_t Z = p->groups, N = p->n_tokens, C = p->n_centroids;
  L.chunks = (int)((N + kMeanRows - 1) / kMeanRows);
  L.error = take(4);
  L.cent_work = take(Z * C * 256);
  L.assign = take(Z * N * 4);
  L.order = take(Z * N * 4);
  L.count = take(Z * C * 4);
  L.offset = take((Z * C + Z * (int64_t)p->n_segments) * 4 + 4);
  L.centred = with_centring ? take(Z * N * 256) : 0;
  L.mean = with_centring ? take(Z * 256) : 0;
  L.partial = with_centring ? take(Z * L.chunks * 512) : 0;
  L.total = off;
  return L;
}

int validate_fit(const ri_kmeans* p) {
  RI_REQUIRE(p != nullptr, "ri_kmeans is null");
  RI_REQUIRE(p->groups > 0 && p->n_tokens > 0 && p->n_centroids > 0, "groups/n_tokens/n_centroids must be positive");
  RI_REQUIRE(p->n_segments >= 1 && p->n_centroids % p->n_segments == 0, "n_centroids must be a multiple of n_segments");
  RI_REQUIRE((p->n_centroids / p->n_segments) % 32 == 0,
             "centroids per segment (%d) must be a multiple of 32", p->n_centroids / p->n_segments);
  RI_REQUIRE(p->n_centroids <= 49152, "n_centroids=%d too large (limit 49152)", p->n_centroids);
  RI_REQUIRE(p->n_iters >= 1, "n_iters must be at least 1");
  RI_REQUIRE(p->dtype == RI_BF16 || p->dtype == RI_F16, "dtype=%d unsupported", p->dtype);
  RI_REQUIRE((int64_t)p->groups * p->n_tokens < (1ll << 31), "groups*n_tokens must stay below 2^31 rows");
  RI_REQUIRE(p->n_tokens / p->n_segments >= 1, "fewer tokens than segments");
  return RI_OK;
}

// Where the caller's rows lie: places of a K or V row, of a row of the cluster-contiguous copy, optional mask of empty clusters.
struct Place { RowPlace src; int64_t out_group; uint8_t* empty; };

template <int DT>
int run_fit(const ri_kmeans* p, const FitLayout& L, const Place& pl, const void* centred, cudaStream_t s) {
  uint8_t* sc = static_cast<uint8_t*>(p->d_scratch);
  const int Z = p->groups, N = p->n_tokens, C = p->n_centroids, S = p->n_segments;
  int* err = p->d_error ? p->d_error : reinterpret_cast<int*>(sc + L.error);
  void* cent = sc + L.cent_work;
  int32_t* assign = p->d_assign ? p->d_assign : reinterpret_cast<int32_t*>(sc + L.assign);
  int32_t* order = p->d_order ? p->d_order : reinterpret_cast<int32_t*>(sc + L.order);
  int32_t* count_work = reinterpret_cast<int32_t*>(sc + L.count);
  int32_t* offset_work = reinterpret_cast<int32_t*>(sc + L.offset);

  RI_CUDA_OK(cudaMemsetAsync(err, 0, 4, s));
  {
    const float step = (float)((double)N / (double)C);
    const float half = (float)((double)N / (double)C / 2.0);
    dim3 grid((C * 16 + 255) / 256, Z);
    init_centroids_kernel<<<grid, 256, 0, s>>>(static_cast<const uint4*>(centred), static_cast<uint4*>(cent), N, C, step, half);
    RI_LAUNCH_OK("init_centroids_kernel");
  }
  CUtensorMap map_keys, map_cent;
  int rc = make_row_map(&map_keys, centred, (int64_t)Z * N, DT);
  if (rc != RI_OK) return rc;
  rc = make_row_map(&map_cent, cent, (int64_t)Z * C, DT);
  if (rc != RI_OK) return rc;
  RI_CUDA_OK(cudaFuncSetAttribute(kmeans_assign_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmem));
  RI_CUDA_OK(cudaFuncSetAttribute(kmeans_assign_resident_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem));

  int sms = 0;
  if ((rc = ri_sm_count(&sms)) != RI_OK) return rc;
  for (int it = 0; it < p->n_iters; ++it) {
    const bool last = it == p->n_iters - 1;
    const int seg = last ? 1 : S;
    const int n_tok = last ? N : N / S;
    const int n_cen = C / seg;
    const int problems = Z * seg;
    AssignArgs aa;
    aa.assign = assign; aa.error_flag = err; aa.n_tok = n_tok; aa.n_cen = n_cen; aa.seg_per_group = seg;
    aa.group_stride = N;
    aa.idesc = idesc_f16(DT, kTileM, kTileN);
    {
      // persistent CTAs, one per SM, an even share of the units each
      WideArgs wa;
      wa.a = aa;
      const bool resident = n_cen <= 4 * kTileN;        // the problem's centroids fit shared memory: they stay there
      wa.per_problem = resident ? (n_tok + kTileM - 1) / kTileM : (n_tok + 2 * kTileM - 1) / (2 * kTileM);
      RI_REQUIRE((int64_t)wa.per_problem * problems < (1ll << 30), "too many token tiles in one launch");
      wa.n_units = wa.per_problem * problems;
      const dim3 wgrid((unsigned)(wa.n_units < sms ? wa.n_units : sms));
      if (resident) {
        RI_CUDA_OK(ri_launch_pdl_id(10, kmeans_assign_resident_kernel, wgrid, dim3(kWideThreads), kResSmem, s, map_keys, map_cent, wa));
      } else {
        RI_CUDA_OK(ri_launch_pdl_id(10, kmeans_assign_wide_kernel, wgrid, dim3(kWideThreads), kWideSmem, s, map_keys, map_cent, wa));
      }
    }

    BucketArgs ba;
    ba.assign = assign; ba.order = order;
    ba.count = last && p->d_cluster_count ? p->d_cluster_count : count_work;
    ba.offset = last && p->d_cluster_offset ? p->d_cluster_offset : offset_work;
    ba.n_tok = n_tok; ba.n_cen = n_cen; ba.seg_per_group = seg; ba.group_stride = N;
    const BucketPlan bp = bucket_plan(problems, n_tok, n_cen, sms);
    if ((n_tok + bp.cl - 1) / bp.cl <= 60000 && bp.smem <= 200 * 1024) {
      rc = bp.cl == 8 ? launch_bucket<8>(ba, bp, problems, s) : bp.cl == 4 ? launch_bucket<4>(ba, bp, problems, s)
         : bp.cl == 2 ? launch_bucket<2>(ba, bp, problems, s) : launch_bucket<1>(ba, bp, problems, s);
      if (rc != RI_OK) return rc;
    } else {
      // as many token ranges (scattering warps) as fit the shared memory: a table of [ranges + 1][n_cen] words
      int workers = 32;
      while (workers > 1 && (size_t)(workers + 1) * n_cen * 4 > 200 * 1024) workers >>= 1;
      const size_t bsmem = (size_t)(workers == 1 ? 1 : workers + 1) * n_cen * 4;
      RI_REQUIRE(bsmem <= 227 * 1024, "n_centroids per problem = %d too large for the bucket pass", n_cen);
      if (bsmem > 48 * 1024)
        RI_CUDA_OK(cudaFuncSetAttribute(kmeans_bucket_one_cta_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsmem));
      kmeans_bucket_one_cta_kernel<<<problems, 1024, bsmem, s>>>(ba, workers);
      RI_LAUNCH_OK("kmeans_bucket_one_cta_kernel");
    }

    UpdateArgs ua = {};
    ua.rows = static_cast<const uint2*>(centred);
    ua.src = {N, 1};
    ua.order = order; ua.offset = ba.offset;
    ua.centroids = static_cast<uint2*>(cent);
    ua.n_tok = n_tok; ua.n_cen = n_cen; ua.seg_per_group = seg; ua.normalize = last ? 0 : 1; ua.group_stride = N;
    if (last) {
      ua.values = static_cast<const uint2*>(p->d_values);
      ua.value_sum = static_cast<uint2*>(p->d_value_sum);
      ua.size_dt = static_cast<uint16_t*>(p->d_cluster_size);
      ua.empty = pl.empty;
      ua.src = pl.src;
      ua.rows = static_cast<const uint2*>(p->d_keys);         // raw keys: centred on the fly, copied as they are
      ua.keys_out = static_cast<uint2*>(p->d_keys_out);
      ua.values_out = static_cast<uint2*>(p->d_values_out);
      ua.out_group = pl.out_group;
      if (p->center) {
        ua.mean = reinterpret_cast<const uint16_t*>(sc + L.mean);
        ua.out_centroids = static_cast<uint2*>(p->d_centroids);
      }
    }
    RI_REQUIRE((int64_t)n_cen * problems < (1ll << 30), "too many clusters in one launch (%d x %d)", n_cen, problems);
    const int n_clusters = n_cen * problems;
    // clusters per warp: a longer run of rows hides more latency, but enough warps for a few rounds of the chip
    int cpw = 8;
    while (cpw > 1 && n_clusters / cpw < sms * 96) cpw >>= 1;
    ua.clusters_per_warp = cpw;
    constexpr int per_cta = kUpdateThreads / 32;
    const dim3 ugrid(n_clusters / cpw / per_cta);               // without remainder: n_cen is a multiple of 32
    RI_CUDA_OK(last     ? ri_launch_pdl_id(9, kmeans_update_kernel<DT, true, false>, ugrid, dim3(kUpdateThreads), 0, s, ua)
               : it < 2 ? ri_launch_pdl_id(9, kmeans_update_kernel<DT, false, true>, ugrid, dim3(kUpdateThreads), 0, s, ua)
                        : ri_launch_pdl_id(9, kmeans_update_kernel<DT, false, false>, ugrid, dim3(kUpdateThreads), 0, s, ua));
  }
  if (!p->center)
    RI_CUDA_OK(cudaMemcpyAsync(p->d_centroids, cent, (size_t)Z * C * 256, cudaMemcpyDeviceToDevice, s));
  return RI_OK;
}

template <int DT>
int run_build(const ri_kmeans* p, const Place& pl, cudaStream_t s) {
  const FitLayout L = fit_layout(p, p->center != 0);
  uint8_t* sc = static_cast<uint8_t*>(p->d_scratch);
  const void* centred = p->d_keys;
  if (p->center) {
    const int Z = p->groups, N = p->n_tokens;
    float* partial = reinterpret_cast<float*>(sc + L.partial);
    uint16_t* mean = reinterpret_cast<uint16_t*>(sc + L.mean);
    colsum_partial_kernel<DT><<<dim3(L.chunks, Z), 256, 0, s>>>(static_cast<const uint4*>(p->d_keys), pl.src, partial, N, L.chunks);
    RI_LAUNCH_OK("colsum_partial_kernel");
    colmean_final_kernel<DT><<<Z, 128, 0, s>>>(partial, mean, N, L.chunks);
    RI_LAUNCH_OK("colmean_final_kernel");
    const int64_t pieces = (int64_t)N * 16;
    centre_apply_kernel<DT><<<dim3((unsigned)((pieces + 255) / 256), Z), 256, 0, s>>>(
        static_cast<const uint4*>(p->d_keys), pl.src, mean, reinterpret_cast<uint4*>(sc + L.centred), pieces);
    RI_LAUNCH_OK("centre_apply_kernel");
    centred = sc + L.centred;
    if (p->d_mean_key) RI_CUDA_OK(cudaMemcpyAsync(p->d_mean_key, mean, (size_t)Z * 256, cudaMemcpyDeviceToDevice, s));
  }
  return run_fit<DT>(p, L, pl, centred, s);
}

}  // namespace

extern "C" int64_t ri_kmeans_scratch_bytes(const ri_kmeans* p) {
  if (validate_fit(p) != RI_OK) return RI_ERR_INVALID;
  return fit_layout(p, p->center != 0).total;
}

namespace {

int validate_build(const ri_kmeans* p) {
  const int rc = validate_fit(p);
  if (rc != RI_OK) return rc;
  RI_REQUIRE(p->d_keys && p->d_values && p->d_centroids && p->d_value_sum && p->d_cluster_size && p->d_scratch,
             "ri_kmeans: a required pointer is null");
  RI_REQUIRE((p->d_keys_out == nullptr) == (p->d_values_out == nullptr), "keys_out and values_out go together");
  RI_REQUIRE(((uintptr_t)p->d_keys | (uintptr_t)p->d_values | (uintptr_t)p->d_centroids | (uintptr_t)p->d_value_sum |
              (uintptr_t)p->d_scratch | (uintptr_t)p->d_keys_out | (uintptr_t)p->d_values_out) % 16 == 0,
             "tensor pointers must be 16-byte aligned");
  return RI_OK;
}

int build(const ri_kmeans* p, const Place& pl, cudaStream_t s) {
  return p->dtype == RI_BF16 ? run_build<RI_BF16>(p, pl, s) : run_build<RI_F16>(p, pl, s);
}

// Sink and recent rows of every head into the steady zone: rows [0, n_sink) and [n_tokens_total - n_recent, n_tokens_total)
// of the prompt, one 16-byte piece of K and of V per thread.
__global__ void __launch_bounds__(256) steady_fill_kernel(const uint4* __restrict__ k, const uint4* __restrict__ v, RowPlace src,
                                                          uint4* __restrict__ sk, uint4* __restrict__ sv, int n_sink,
                                                          int n_recent, int64_t recent_row, int64_t stride) {
  const int i = blockIdx.x * 256 + threadIdx.x, row = i >> 4, piece = i & 15, z = blockIdx.y;
  if (row >= n_sink + n_recent) return;
  const int64_t r = row < n_sink ? row : recent_row + row - n_sink;
  const int64_t from = (z * src.group + r * src.row) * 16 + piece, to = (z * stride + row) * 16 + piece;
  sk[to] = ri_ldg16(k + from);
  sv[to] = ri_ldg16(v + from);
}

}  // namespace

extern "C" int ri_kmeans_build(const ri_kmeans* p, void* stream) {
  const int rc = validate_build(p);
  if (rc != RI_OK) return rc;
  const Place pl = {{p->n_tokens, 1}, p->n_tokens, nullptr};
  return build(p, pl, static_cast<cudaStream_t>(stream));
}

extern "C" int ri_kmeans_build_prompt(const ri_kmeans* p, const ri_kmeans_prompt* q, void* stream) {
  int rc = validate_build(p);
  if (rc != RI_OK) return rc;
  RI_REQUIRE(q != nullptr, "ri_kmeans_prompt is null");
  RI_REQUIRE(p->center == 1, "ri_kmeans_build_prompt: center must be 1");
  RI_REQUIRE(q->n_sink >= 0 && q->n_recent >= 0 && q->out_group_rows >= p->n_tokens, "ri_kmeans_prompt: bad sizes");
  RI_REQUIRE((q->n_sink + q->n_recent == 0) || (q->d_steady_keys && q->d_steady_values && q->steady_group_rows >= q->n_sink + q->n_recent),
             "ri_kmeans_prompt: bad steady zone");
  RI_REQUIRE(((uintptr_t)q->d_steady_keys | (uintptr_t)q->d_steady_values) % 16 == 0, "tensor pointers must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // token-major prompt [tokens, Z, 128]: the clustered rows lie behind the sink rows
  const RowPlace src = {1, p->groups};
  if (q->n_sink + q->n_recent > 0) {
    steady_fill_kernel<<<dim3(((q->n_sink + q->n_recent) * 16 + 255) / 256, p->groups), 256, 0, s>>>(
        static_cast<const uint4*>(p->d_keys), static_cast<const uint4*>(p->d_values), src, static_cast<uint4*>(q->d_steady_keys),
        static_cast<uint4*>(q->d_steady_values), q->n_sink, q->n_recent, (int64_t)q->n_sink + p->n_tokens, q->steady_group_rows);
    RI_LAUNCH_OK("steady_fill_kernel");
  }
  ri_kmeans c = *p;
  const int64_t skip = (int64_t)q->n_sink * p->groups * 256;
  c.d_keys = static_cast<const uint8_t*>(p->d_keys) + skip;
  c.d_values = static_cast<const uint8_t*>(p->d_values) + skip;
  const Place pl = {src, q->out_group_rows, q->d_empty};
  return build(&c, pl, s);
}
