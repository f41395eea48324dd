// Dense (causal) prefill attention, head_dim 128, grouped-query heads, 16-bit inputs, fp32 accumulation.
// Replaces the flash-attn call of attn_hub/retroinfer_attn.py:4-13 (`retroinfer_prefill_attn`:
// flash_attn_with_kvcache(q, k_cache, v_cache, causal) over the whole prompt).
//
// One persistent CTA per SM works through items of (two neighbouring tiles of 128 query rows, query head, request); an
// item walks the key/value tiles of 128 tokens the rows may see, and both query tiles use every tile that is brought in.
//   S_g = Q_g.K^T   tcgen05.mma, M 128 x N 128 x K 128 (8 x K16), operands staged by TMA with the 128-byte swizzle
//                   straight from the token-major tensors, fp32 accumulator in TMEM;
//   softmax         one group of 128 threads per query tile, one thread per query row (= TMEM lane): a row of S comes
//                   down with tcgen05.ld into registers; online softmax in the log2 domain with a LAZY reference maximum
//                   (the running maximum is only adopted when it has grown by more than a step, so an accumulator
//                   is rescaled rarely); P goes back to TMEM as packed 16-bit pairs over the columns of S it came from;
//   O_g += P_g.V    tcgen05.mma with A = P_g from TMEM and B = the V tile as TMA brought it (channels contiguous:
//                   an MN-major operand), accumulator in TMEM for the whole walk.
// TMEM: S_0 | S_1 | O_0 | O_1, 128 columns each.  Warps: TMA producer, MMA issuer, two idle, eight softmax/epilogue warps,
// which take the registers the first four give up (a row of S is 128 of them).
//
// Why this split: an MMA of M 128 x N 128 with both operands in shared memory reads 128 bytes a clock, all that shared
// memory has.  With one query tile per CTA and P in shared memory a key/value tile cost 224 KB of it (Q, K, P, V read,
// K, V, P written) = 1792 clocks against 1024 of tensor work, and the kernel ran at 0.51 of the measured peak.  Two query
// tiles that share K and V, and P in TMEM, make it 128 KB per tile and query tile; V needs no transposed copy.  While one
// group's softmax runs, the tensor pipe does the other group's two products.
// 32 query and 8 key/value heads, causal, bf16, 32768 tokens: 9.9 -> 7.3 ms from rest (889 -> 1200 TFLOP/s), 10.7 -> 8.3 ms
// in a repeated run, which the power limit holds at 1055 TFLOP/s; 8192 tokens 0.48 ms repeated, a call for 777 tokens 53 ->
// 20.5 us.  What bounds it now (ncu, 8192 tokens): each group's chain of scores, softmax and product, about 1700 clocks per
// tile and group; tensor pipe 56 % and exponentials 56 % of the active cycles, issue slots 35 %.  Doing a quarter of the
// exponentials as polynomials on the FMA pipe was slower (1170 TFLOP/s): they are not what the chain waits for.
// SPLIT: for few query tiles a CTA takes one of them, and its groups take the even and the odd key/value tiles.
// Every mbarrier wait is bounded; on expiry a CTA records where, releases its TMEM and returns.  The word it is recorded in
// is only written: what an earlier call left there makes no later one give up (all CTAs of a launch are resident at once, so
// one that gives up saves the others nothing).
#include <cuda.h>

#include "ri_common.cuh"
#include "ri_tc.cuh"

namespace {

using namespace ri_tc;

constexpr int kTile = 128;                 // query rows per tile, keys per step
constexpr int kHalf = kTile * 128;         // bytes of a 128-row x 64-element operand half-tile
constexpr int kSlots = 5;                  // ring of K and V tiles: K0, V0, K1, V1, ...
constexpr int kThreads = 384;            // three warpgroups: TMA producer and MMA issuer (two warps idle), softmax of Q_0, of Q_1
constexpr uint32_t kTmemCols = 512;        // S_0 | S_1 | O_0 | O_1, 128 columns each
constexpr int smem_bytes(bool split) {
  return 1024 /*align*/ + (split ? 1 : 2) * 2 * kHalf /*Q_0, Q_1*/ + kSlots * 2 * kHalf /*K, V*/ + 256 /*barriers*/;
}
// The reference maximum follows the running one in steps of more than 2^lazy.  A key whose score is the reference has a
// probability of exactly 1, any other one is rounded to 16 bits, so a reference that lags behind costs accuracy: for keys
// with a few near ones among many (a trained model's) the paired form's one walk per row was 3 % further from 64-bit
// attention at 2^8 than two walks, which start from two references, are at the same step.  Relative error of the paired
// form, bf16, 32768 tokens: 2.12e-3 at 2^8, 1.97e-3 at 2^4 with rows catching up together (two walks 2.06e-3, rounding the
// result alone 1.65e-3), for 1 % of the time (8.28 -> 8.36 ms a repeated run, 32 query heads).
__host__ __device__ constexpr float lazy_step(bool split) { return split ? 8.0f : 4.0f; }

struct AttnArgs {
  void* out;             // [B, S, Hq, 128]
  int* error_flag;
  int B, S, Hq, Hk, causal;
  int units;             // items of a head: pairs of query tiles, or single ones
  float scale2;          // log2(e) / sqrt(128)
  uint32_t idesc_qk, idesc_pv;
};

// One CTA's share of the work: (pair of query tiles, head, request) items, longest walks first.  The grid has one CTA per
// SM and takes the items round by round, every second round backwards, so that the sums of the walks come out alike.
struct Item {
  int q_tile, h, b;      // group g's query tile is q_tile + g, or q_tile for both (SPLIT)
  int n[2];              // key/value tiles each group walks (0: nothing to do for the second one)
  int n_kv, tiles;       // steps of the longer walk; tiles brought in
};
__device__ __forceinline__ int item_index(int round) {
  const int c = (int)blockIdx.x, g = (int)gridDim.x;
  return round * g + ((round & 1) ? g - 1 - c : c);
}
template <bool SPLIT>
__device__ __forceinline__ Item get_item(const AttnArgs& a, int index) {
  const int heads = a.Hq * a.B, u = index / heads, hb = index - u * heads;
  Item it;
  it.q_tile = (a.units - 1 - u) * (SPLIT ? 1 : 2);
  it.b = hb / a.Hq;
  it.h = hb - it.b * a.Hq;
  const int kv_total = (a.S + kTile - 1) / kTile;
  const int n0 = a.causal ? min(it.q_tile + 1, kv_total) : kv_total;
  if (SPLIT) {
    it.n[0] = (n0 + 1) / 2;
    it.n[1] = n0 / 2;
    it.tiles = n0;
  } else {
    it.n[0] = n0;
    it.n[1] = (it.q_tile + 1) * kTile >= a.S ? 0 : (a.causal ? min(it.q_tile + 2, kv_total) : kv_total);
    it.tiles = max(it.n[0], it.n[1]);
  }
  it.n_kv = max(it.n[0], it.n[1]);
  return it;
}

// ---- softmax arithmetic ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float ex2(float x) {       // 2^x; results below 2^-126 become 0
  float d;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(d) : "f"(x));
  return d;
}

template <int DT, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
prefill_attn_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, AttnArgs a) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sQ = base, sKV = sQ + (SPLIT ? 1 : 2) * 2 * kHalf;
  const uint32_t bars = sKV + kSlots * 2 * kHalf;
  auto bar_q = [&](int g) { return bars + 8u * g; };
  auto bar_full = [&](int s) { return bars + 8u * (2 + s); };
  auto bar_empty = [&](int s) { return bars + 8u * (2 + kSlots + s); };
  auto bar_s_full = [&](int g) { return bars + 8u * (2 + 2 * kSlots + g); };
  auto bar_p_full = [&](int g) { return bars + 8u * (4 + 2 * kSlots + g); };
  auto bar_o_full = [&](int g) { return bars + 8u * (6 + 2 * kSlots + g); };
  auto bar_q_empty = [&](int g) { return bars + 8u * (10 + 2 * kSlots + g); };
  auto bar_p_part = [&](int g) { return bars + 8u * (8 + 2 * kSlots + g); };
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  __shared__ float2 s_stat[2][SPLIT ? kTile : 1];          // SPLIT: a row's (maximum, sum) in either group

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_items = a.units * a.Hq * a.B;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int g = 0; g < 2; ++g) {
      mbar_init(bar_q(g), 1); mbar_init(bar_q_empty(g), 1); mbar_init(bar_s_full(g), 1);
      mbar_init(bar_p_part(g), 4); mbar_init(bar_p_full(g), 4); mbar_init(bar_o_full(g), 1);
    }
    for (int s = 0; s < kSlots; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem_base;
  volatile int* abort_flag = &s_abort;

  // registers at launch: 384 x 168; after the split 128 x 96 + 256 x 200, which is less
  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
  if (warp == 0) {
    // ---------------- TMA producer: Q_0, K0, Q_1, V0, K1, V1, ... of one item after the other ----------------
    if (lane == 0) {
      int issued = 0, q_issued[2] = {0, 0};
      bool ok = true;
      for (int round = 0; ok; ++round) {
        const int index = item_index(round);
        if (index >= n_items) break;
        const Item it = get_item<SPLIT>(a, index);
        const int hk = it.h / (a.Hq / a.Hk);
        auto load_q = [&](int g) {
          if (!mbar_wait(bar_q_empty(g), (q_issued[g] & 1) ^ 1, abort_flag, 20)) return false;
          mbar_arrive_expect_tx(bar_q(g), 2 * kHalf);
          tma_load_3d(sQ + g * 2 * kHalf, &map_q, bar_q(g), it.h * 128, (it.q_tile + g) * kTile, it.b);
          tma_load_3d(sQ + g * 2 * kHalf + kHalf, &map_q, bar_q(g), it.h * 128 + 64, (it.q_tile + g) * kTile, it.b);
          ++q_issued[g];
          return true;
        };
        ok = load_q(0);
        for (int t = 0; ok && t < 2 * it.tiles; ++t) {
          const int s = issued % kSlots;
          ok = mbar_wait(bar_empty(s), ((issued / kSlots) & 1) ^ 1, abort_flag, 21);
          if (!ok) break;
          const CUtensorMap* map = (t & 1) ? &map_v : &map_k;
          mbar_arrive_expect_tx(bar_full(s), 2 * kHalf);
          tma_load_3d(sKV + s * 2 * kHalf, map, bar_full(s), hk * 128, (t >> 1) * kTile, it.b);
          tma_load_3d(sKV + s * 2 * kHalf + kHalf, map, bar_full(s), hk * 128 + 64, (t >> 1) * kTile, it.b);
          ++issued;
          if (!SPLIT && t == 0 && it.n[1] > 0) ok = load_q(1);
        }
      }
      if (*abort_flag) {     // give the copies still in flight a bounded chance to land before the CTA exits
        for (int g = 0; g < 2; ++g)
          if (q_issued[g] > 0) mbar_wait(bar_q(g), (q_issued[g] - 1) & 1, abort_flag, 26);
        for (int t = max(0, issued - kSlots); t < issued; ++t) mbar_wait(bar_full(t % kSlots), (t / kSlots) & 1, abort_flag, 28);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // Per key/value tile j: P_0.V, then S_0 of tile j+1, then the same for query tile 1; behind the last tile of an item
    // come the first scores of the next one, so that the softmax of neither group waits for the other's epilogue.
    // S_g of the next tile overwrites the columns P_g was read from: both are MMAs of this thread, which the tensor pipe
    // takes in order.
    if (lane == 0) {
      int tile0 = 0;                       // ring index of the item's first K tile
      int q_used[2] = {0, 0}, p_used[2] = {0, 0};
      auto wait_tile = [&](int t) { return mbar_wait(bar_full(t % kSlots), (t / kSlots) & 1, abort_flag, 23); };
      // ring index of the K tile of group g's step j, relative to the item's first; its V tile is the next one
      auto ring_k = [&](int g, int j) { return tile0 + 2 * (SPLIT ? 2 * j + g : j); };
      auto issue_qk = [&](int g, int t, bool last) {
        const uint32_t sk = sKV + (t % kSlots) * 2 * kHalf;
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
          const uint64_t da = umma_desc_sw128(sQ + ((SPLIT ? 0 : g) * 2 + kb) * kHalf), db = umma_desc_sw128(sk + kb * kHalf);
#pragma unroll
          for (int k = 0; k < 4; ++k) tc_mma_f16(tmem + g * kTile, da + 2 * k, db + 2 * k, a.idesc_qk, (kb | k) != 0);
        }
        tc_commit(bar_s_full(g));          // also says that P_g.V of the tile before has completed
        if (last) tc_commit(bar_q_empty(SPLIT ? 0 : g));
        if (SPLIT) tc_commit(bar_empty(t % kSlots));
      };
      // V tile: two halves of 64 channels x 128 tokens, a token's 64 channels in 128 swizzled bytes; 16 tokens = 2048 bytes
      auto issue_pv = [&](int g, int t, int k0, int k1, bool first) {
        const uint64_t db = umma_desc_mn_sw128(sKV + (t % kSlots) * 2 * kHalf, kHalf);
#pragma unroll
        for (int k = k0; k < k1; ++k)
          tc_mma_f16_ts(tmem + (2 + g) * kTile, tmem + g * kTile + 8 * k, db + 128 * k, a.idesc_pv, !first || k != 0);
      };
      // whether group g's step j is the last user of its Q tile (SPLIT: the walks' last steps, group 1 behind group 0)
      auto last_of_q = [&](const Item& it, int g, int j) {
        return SPLIT ? (it.tiles == 2 * j + g + 1) : j + 1 == it.n[g];
      };
      auto start_item = [&](const Item& it) {       // first scores of both groups
        for (int g = 0; g < 2; ++g) {
          if (it.n[g] == 0) continue;
          if (!wait_tile(ring_k(g, 0))) return false;
          if (!SPLIT || g == 0) {
            if (!mbar_wait(bar_q(g), q_used[g] & 1, abort_flag, 22)) return false;
            ++q_used[g];
          }
          tc_fence_after();
          issue_qk(g, ring_k(g, 0), last_of_q(it, g, 0));
        }
        if (!SPLIT) tc_commit(bar_empty(tile0 % kSlots));
        return true;
      };
      bool ok = true;
      Item it = get_item<SPLIT>(a, item_index(0));         // the grid is no larger than the number of items
      ok = start_item(it);
      for (int round = 1; ok; ++round) {
        for (int j = 0; ok && j < it.n_kv; ++j) {
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            if (ok && j < it.n[g]) {
              const int tv = ring_k(g, j) + 1;
              ok = wait_tile(tv) && mbar_wait(bar_p_part(g), p_used[g] & 1, abort_flag, 24);
              if (!ok) break;
              tc_fence_after();
              issue_pv(g, tv, 0, 4, j == 0);
              ok = mbar_wait(bar_p_full(g), p_used[g] & 1, abort_flag, 25);
              if (!ok) break;
              tc_fence_after();
              issue_pv(g, tv, 4, 8, false);
              if (SPLIT) tc_commit(bar_empty(tv % kSlots));
              ++p_used[g];
              if (j + 1 < it.n[g]) {
                ok = wait_tile(ring_k(g, j + 1));
                if (!ok) break;
                tc_fence_after();
                issue_qk(g, ring_k(g, j + 1), last_of_q(it, g, j + 1));
              } else {
                tc_commit(bar_o_full(g));
              }
            }
          }
          if (!SPLIT && ok) {
            tc_commit(bar_empty((tile0 + 2 * j + 1) % kSlots));
            if (j + 1 < it.n_kv) tc_commit(bar_empty((tile0 + 2 * j + 2) % kSlots));
          }
        }
        const int index = item_index(round);
        if (!ok || index >= n_items) break;
        tile0 += 2 * it.tiles;
        it = get_item<SPLIT>(a, index);
        ok = start_item(it);
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
    // ---------------- softmax and epilogue: thread = query row = TMEM lane; group g owns query tile g ----------------
    const int grp = (warp - 4) >> 2;                       // 0 or 1
    const int lane_group = warp & 3;                       // a warp may touch only its quarter of the TMEM lanes
    const int row = lane_group * 32 + lane;                // row of the tile
    const uint32_t t_lane = (uint32_t)(lane_group * 32) << 16;
    const uint32_t tmem_s = tmem + grp * kTile + t_lane, tmem_o = tmem + (2 + grp) * kTile + t_lane;
    const uint64_t scale_2 = pack_f2(a.scale2, a.scale2);
    bool ok = true;
    int done = 0, outs[2] = {0, 0};                        // tiles of this group, outputs of both groups so far
    for (int round = 0;; ++round) {                        // as many rounds whatever the waits return (named barriers)
    const int index = item_index(round);
    if (index >= n_items) break;
    const Item it = get_item<SPLIT>(a, index);
    const int n = it.n[grp];
    if (!SPLIT && n == 0) continue;
    const int q_row = (it.q_tile + (SPLIT ? 0 : grp)) * kTile + row;   // position of the query in its request
    float m_ref = -INFINITY, l_run = 0.f;
    for (int j = 0; ok && j < n; ++j, ++done) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar_s_full(grp), done & 1, abort_flag, 31));
      if (!ok) break;
      tc_fence_after();
      uint32_t sr[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tc_ld32(tmem_s + c * 32, sr[c]);
      tc_wait_ld();
#pragma unroll
      for (int c = 0; c < 4; ++c) tc_ld_landed(sr[c]);

      // masked scores (edge tiles only) and the row maximum, on the raw products (the scale is positive)
      const int col0 = (SPLIT ? 2 * j + grp : j) * kTile;
      if (col0 + kTile > a.S || (a.causal && col0 + kTile - 1 > q_row)) {
        const int limit = a.causal ? min(a.S - 1, q_row) : a.S - 1;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (col0 + c * 32 + i > limit) sr[c][i] = 0xff800000u;     // -inf
      }
      float mx[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        mx[c] = fmaxf(__uint_as_float(sr[c][0]), __uint_as_float(sr[c][1]));
#pragma unroll
        for (int i = 2; i < 32; i += 2) mx[c] = max3(mx[c], __uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1]));
      }
      const float m_tile = max3(fmaxf(mx[0], mx[1]), mx[2], mx[3]) * a.scale2;
      // lazy reference maximum: adopt the running maximum only when it has grown by more than the step
      const bool move = m_tile > m_ref + lazy_step(SPLIT);      // also true for the first tile (m_ref = -inf)
      if (__any_sync(0xffffffffu, move)) {
        // pairs: the warp's accumulator rows are multiplied anyway, so every row of it catches up with its maximum
        const float m_new = SPLIT ? (move ? m_tile : m_ref) : fmaxf(m_ref, m_tile);
        const float factor = m_ref == -INFINITY ? 0.f : exp2f(m_ref - m_new);      // 1 when the maximum stays
        l_run *= factor;
        m_ref = m_new;
        if (j > 0) {                                       // rare: bring this warp's rows of O to the new reference
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t orow[32];
            tc_ld32(tmem_o + c * 32, orow);
            tc_wait_ld();
            tc_ld_landed(orow);
#pragma unroll
            for (int i = 0; i < 32; ++i) orow[i] = __float_as_uint(__uint_as_float(orow[i]) * factor);
            tc_st32(tmem_o + c * 32, orow);
          }
        }
      }
      // probabilities p = 2^(s * scale - m), packed as the 16-bit operand of the second product: word w of the row =
      // keys 2w, 2w+1, over the first 64 columns of S
      const uint64_t neg_m = pack_f2(-m_ref, -m_ref);
      uint64_t sum2[2] = {0ull, 0ull};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pw[16];
#pragma unroll
        for (int w = 0; w < 16; ++w) {
          const uint64_t x = fma_f2(pack_f2(__uint_as_float(sr[c][2 * w]), __uint_as_float(sr[c][2 * w + 1])), scale_2, neg_m);
          float x0, x1;
          unpack_f2(x, x0, x1);
          const float p0 = ex2(x0), p1 = ex2(x1);
          sum2[w & 1] = add_f2(sum2[w & 1], pack_f2(p0, p1));
          pw[w] = Elem<DT>::pack2(p0, p1);
        }
        tc_st16(tmem_s + c * 16, pw);
        if (c == 1) {          // the product over the first 64 keys may start
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_p_part(grp));
        }
      }
      float s0, s1;
      unpack_f2(add_f2(sum2[0], sum2[1]), s0, s1);
      l_run += s0 + s1;
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_p_full(grp));
    }
    // ---- epilogue, one row per thread.  A query tile of its own: the accumulator divided by the sum.  SPLIT: the groups
    //      exchange (maximum, sum) through shared memory, then each merges half of the channels of both accumulators by
    //      log-sum-exp; the second barrier keeps an accumulator until the other group has read it ----
    float w0, w1 = 0.f;                                    // weights of the accumulators read below
    if (SPLIT) {
      s_stat[grp][row] = make_float2(m_ref, l_run);
      asm volatile("bar.sync 1, 256;" ::: "memory");
      const float2 other = s_stat[grp ^ 1][row];
      const float m = fmaxf(m_ref, other.x);               // group 0 always has a tile: finite
      const float f_own = m_ref == -INFINITY ? 0.f : ex2(m_ref - m), f_other = other.x == -INFINITY ? 0.f : ex2(other.x - m);
      const float l = l_run * f_own + other.y * f_other, inv = l > 0.f ? 1.0f / l : 0.f;
      w0 = (grp ? f_other : f_own) * inv;
      w1 = (grp ? f_own : f_other) * inv;
    } else {
      w0 = l_run > 0.f ? 1.0f / l_run : 0.f;
    }
#pragma unroll
    for (int g = 0; g < 2; ++g)
      if ((SPLIT || g == grp) && it.n[g] > 0) {
        ok = ok && __all_sync(0xffffffffu, mbar_wait(bar_o_full(g), outs[g] & 1, abort_flag, 33));
        ++outs[g];
      }
    if (ok) {
      tc_fence_after();
      uint4* dst = reinterpret_cast<uint4*>(static_cast<uint16_t*>(a.out) + (((int64_t)it.b * a.S + q_row) * a.Hq + it.h) * 128);
      const bool two = SPLIT && it.n[1] > 0;
      const int c0 = SPLIT ? grp * 2 : 0, c1 = SPLIT ? c0 + 2 : 4;
#pragma unroll 1
      for (int c = c0; c < c1; ++c) {
        uint32_t o0[32], o1[32];
        tc_ld32(tmem + (2 + (SPLIT ? 0 : grp)) * kTile + t_lane + c * 32, o0);
        if (two) tc_ld32(tmem + 3 * kTile + t_lane + c * 32, o1);
        tc_wait_ld();
        tc_ld_landed(o0);
        if (two) tc_ld_landed(o1);
        if (q_row < a.S) {
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i)
            v[i] = __uint_as_float(o0[i]) * w0 + (two ? __uint_as_float(o1[i]) * w1 : 0.f);
#pragma unroll
          for (int i = 0; i < 32; i += 8)
            dst[c * 4 + i / 8] = make_uint4(Elem<DT>::pack2(v[i], v[i + 1]), Elem<DT>::pack2(v[i + 2], v[i + 3]),
                                            Elem<DT>::pack2(v[i + 4], v[i + 5]), Elem<DT>::pack2(v[i + 6], v[i + 7]));
        }
      }
    }
    if (SPLIT) asm volatile("bar.sync 1, 256;" ::: "memory");
    }   // next item
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && s_abort) *a.error_flag = s_abort;
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
  }
}

template <int DT>
int launch(const void* q, const void* k, const void* v, void* out, int32_t* error, int B, int S, int Hq, int Hk, int causal,
           cudaStream_t s) {
  CUtensorMap map_q, map_k, map_v;
  int rc;
  if ((rc = make_map_3d(&map_q, q, (int64_t)Hq * 128, S, B, DT)) != RI_OK) return rc;
  if ((rc = make_map_3d(&map_k, k, (int64_t)Hk * 128, S, B, DT)) != RI_OK) return rc;
  if ((rc = make_map_3d(&map_v, v, (int64_t)Hk * 128, S, B, DT)) != RI_OK) return rc;
  AttnArgs a;
  a.out = out; a.error_flag = error; a.B = B; a.S = S; a.Hq = Hq; a.Hk = Hk; a.causal = causal;
  a.scale2 = RI_LOG2E * 0.08838834764831845f;
  a.idesc_qk = idesc_f16(DT, kTile, kTile);
  a.idesc_pv = a.idesc_qk | (1u << 16);      // B = V is MN-major (channels contiguous)
  int sms = 0;
  if ((rc = ri_sm_count(&sms)) != RI_OK) return rc;
  const int tiles = (S + kTile - 1) / kTile;
  // Pairs of query tiles share K and V and are 15 % faster where there are enough of them to fill the chip; below one
  // pair per SM a single query tile per CTA, its key/value tiles shared out to both groups, uses more SMs and halves the
  // longest walk (4096 tokens, 8 heads: 42 against 66 us; 777 tokens, 28 heads: 18.6 against 20.5; at 160 pairs equal).
  const bool split = (int64_t)((tiles + 1) / 2) * Hq * B < sms;
  a.units = split ? tiles : (tiles + 1) / 2;
  const int64_t items = (int64_t)a.units * Hq * B;
  RI_REQUIRE(items < (1ll << 30), "ri_prefill_attn: too large");
  const dim3 grid((unsigned)(items < sms ? items : sms));
  if (split) {
    RI_CUDA_OK(cudaFuncSetAttribute(prefill_attn_kernel<DT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(true)));
    prefill_attn_kernel<DT, true><<<grid, kThreads, smem_bytes(true), s>>>(map_q, map_k, map_v, a);
  } else {
    RI_CUDA_OK(cudaFuncSetAttribute(prefill_attn_kernel<DT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(false)));
    prefill_attn_kernel<DT, false><<<grid, kThreads, smem_bytes(false), s>>>(map_q, map_k, map_v, a);
  }
  RI_LAUNCH_OK("prefill_attn_kernel");
  return RI_OK;
}

}  // namespace

// The kernel needs no scratch (V is read as it lies, d_scratch may be null); the size callers allocate stays what it was.
extern "C" int64_t ri_prefill_attn_scratch_bytes(int32_t batch, int32_t seq_len, int32_t kv_heads) {
  if (batch < 1 || seq_len < 1 || kv_heads < 1) return RI_ERR_INVALID;
  const int64_t s_pad = ((int64_t)seq_len + kTile - 1) / kTile * kTile;
  return (int64_t)batch * kv_heads * 128 * s_pad * 2;
}

extern "C" int ri_prefill_attn(const void* d_q, const void* d_k, const void* d_v, void* d_out, void* d_scratch,
                               int32_t* d_error, int32_t batch, int32_t seq_len, int32_t q_heads, int32_t kv_heads,
                               int32_t causal, int32_t dtype, void* stream) {
  (void)d_scratch;
  RI_REQUIRE(d_q && d_k && d_v && d_out && d_error, "ri_prefill_attn: null pointer");
  RI_REQUIRE(batch >= 1 && seq_len >= 1 && kv_heads >= 1 && q_heads >= kv_heads && q_heads % kv_heads == 0,
             "ri_prefill_attn: bad sizes (batch %d, seq_len %d, %d q heads, %d kv heads)", batch, seq_len, q_heads, kv_heads);
  RI_REQUIRE((int64_t)batch * seq_len < (1ll << 31) && (int64_t)batch * kv_heads * 128 < (1ll << 31), "ri_prefill_attn: too large");
  RI_REQUIRE(dtype == RI_BF16 || dtype == RI_F16, "dtype=%d unsupported", dtype);
  RI_REQUIRE(((uintptr_t)d_q | (uintptr_t)d_k | (uintptr_t)d_v | (uintptr_t)d_out) % 16 == 0,
             "ri_prefill_attn: tensors must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return dtype == RI_BF16 ? launch<RI_BF16>(d_q, d_k, d_v, d_out, d_error, batch, seq_len, q_heads, kv_heads, causal, s)
                          : launch<RI_F16>(d_q, d_k, d_v, d_out, d_error, batch, seq_len, q_heads, kv_heads, causal, s);
}
