// The whole decode step of one layer in ONE kernel: a thread-block cluster per group (1 .. 16 CTAs of 256 threads, one CTA
// per SM; see cluster_size) runs
//   phase 1  scan    s = alpha * q.C^T over the group's centroids (each CTA one slice, streamed through a lane-private
//                    cp.async ring), scores kept in shared memory;
//   phase 2  select  the selection of ri_wave_select.cuh reorganised for scores that never leave shared memory;
//   phase 3  attend  the shared attention steps (ri_wave_attend.cuh) over the group's estimation and exact rows.
// Groups are independent, so nothing crosses a cluster: the two kernel boundaries of the staged path (drain, launch, ramp-up,
// and the scores' trip through the per-tile partials) disappear.
//
// What the CTAs of a cluster tell each other (softmax statistics, two histograms, candidates, partial outputs) is PUSHED: the
// producer stores it into every consumer's shared memory with st.async, which counts its bytes on an mbarrier there, and the
// consumer waits for the bytes it expects.  An exchange is one trip over the cluster's network; as a cluster barrier followed
// by loads from the other CTAs it was three (arrive, release, load).  Each of the five mbarriers is used once, so there is
// nothing to reset, and no CTA has to wait for the others to have read.  Every wait is bounded; one that runs out is recorded
// in the process's status word, and the CTA leaves without an output.
//
// What bounds it: at 128K tokens the scan runs at the copy rate (67 MB in 10.5 us), the scattered rows of the attend phase at
// 3.7 TB/s (45 MB in 12 us, up to 15 for the groups with most rows), and between them lies a chain of dependent block-wide
// steps, 8.5 us (of 11), in which no memory is read; at 8K the chain is all there is.  us a layer, before (barriers and loads
// instead of pushes, candidates pulled, one CTA's first warp held up by the append, nothing asked for ahead of the wait for the
// kernel in front) and now: 8K x 8 groups 14.8 / 11.3; 45K x 12 19.5 / 15.5; 128K x 32 44.6 / 36.4; 128K x 16 of 8 heads
// 32.6 / 28.5; 30K x 128 (clusters of 4 taking turns, now one CTA a group) 82 / 35; 100K x 2 25.7 / 16.4 (16 CTAs instead of 8);
// 256K x 32 (three stage kernels, now 16 keys a thread) 117 / 64.  Measured and left out: asking for the estimation entries'
// and the candidates' rows in L2 as soon as they are known (36.0 -> 37.6, they hold up what the chain needs).
// Reference path: cache_hub/retroinfer_cache.py:549-697 (compute).
#include <atomic>
#include <mutex>

#include "ri_tc.cuh"
#include "ri_wave_attend.cuh"
#include "ri_wave_select.cuh"

namespace ri_wave {
namespace {

using ri_tc::smem_u32;

constexpr int kFusedThreads = 256;
constexpr int kFusedWarps = kFusedThreads / 32;
constexpr int kFusedMaxCentroids = 16384;             // per group: four CTAs of 256 threads of 16 keys
// CTAs per group.  More than eight are not portable, and a kernel that may be launched so is slower at every size (128K x 32
// groups in clusters of 4: 36 -> 40 us): the kernel exists for up to 8 and for up to 16 (MAXCL).
constexpr int kMaxCluster = 16;
constexpr int kScanStages = 2;
// In a gather's error word, from a decode kernel that gave up to the wait kernel behind it: a slice is missing.
constexpr int kSliceMissing = 2;

// What follows from the centroids a thread looks after in the selection (KEYS; a CTA's slice has at most 256 * KEYS).
template <int KEYS>
struct Geom {
  static_assert(KEYS == 4 || KEYS == 8 || KEYS == 16, "a thread's keys are loaded in 16-byte pieces");
  static constexpr int kMaxSlice = KEYS * kFusedThreads;
  // floats per head in shared memory: four words of padding after every 32 (see score_at), eight more between heads
  static constexpr int kScoreStride = kMaxSlice + kMaxSlice / 8 + 8;
  // A large slice leaves room for a smaller ring: 16 centroids instead of 32 per warp step, two attend stages instead of three.
  static constexpr int kScanRows = KEYS == 16 ? 16 : 32;
  static constexpr int kScanRing = kFusedWarps * kScanStages * kScanRows * 256;
  static constexpr int kAttendStages = KEYS == 16 ? 2 : 3;
  static constexpr int kAttendRing = kFusedWarps * kAttendStages * kStageBytes;
};

// Place of centroid e of the slice in a head's row of scores: a thread of the selection owns a run of consecutive
// centroids, so without the padding its lanes would sit 4, 8 or 16 words apart and collide on a few banks.
__device__ __forceinline__ int score_at(int e) { return e + ((e >> 5) << 2); }

struct FusedArgs {
  SelectArgs sel;
  AttendArgs att;
  const uint4* cent;
  float* scores;     // global copy of the scores (a view for tests), written only when `views`
  int32_t* status;   // the process's status word
  int32_t* gather_error;   // several GPUs: the gather's error word
  float alpha;
  int views;         // also fill the global lists and views (tests, callers that asked for the id outputs)
  uint4* steady_k_w;       // att.new_k / new_v go to row static_len - 1 of these
  uint4* steady_v_w;
  int page_shift;    // log2 of the page size, or -1
  int out_aligned;   // d_out is 8-byte aligned
  int cl;            // CTAs of a cluster
  // Dynamic shared memory: [scan ring, later the lists that outlive the selection] ... [scores] [mail]; `temp_off` (arrays of
  // the selection) and `ring_off` (the attend ring, over the scores) lie behind the lists.
  int scores_off, temp_off, ring_off, mail_off;
  int cap;           // estimation entries a CTA can keep in shared memory (multiple of 16)
};

// Mail: what other CTAs push while this one may still be scanning or attending.
__host__ __device__ constexpr int chunks_per_cta(int gs, int cl) { return (gs * 32 + cl - 1) / cl; }   // outputs, 4 at a time
__host__ __device__ constexpr int mail_bytes(int gs, int cl) {
  return cl * kFusedWarps * kMaxHeads * 8 + cl * chunks_per_cta(gs, cl) * 24;
}
// Temporary arrays of the selection: histograms pushed by every CTA (256 and 512 16-bit counts), and of each candidate its entry
// (four words) and four words for ranking.
__host__ __device__ constexpr int temp_bytes(int p_pad, int cl) { return cl * 1536 + p_pad * 32; }
__host__ __device__ constexpr int range_bytes(int p_pad) { return (2 * p_pad + 4) * 4; }
__host__ __device__ constexpr int entry_bytes(int gs) { return 4 * gs + 4; }   // scores; index and size

// ---- pushes between the CTAs of a cluster ----------------------------------------------------------------------
__device__ __forceinline__ uint32_t peer(uint32_t addr, int rank) {      // the same place in another CTA's shared memory
  uint32_t d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(addr), "r"(rank));
  return d;
}
__device__ __forceinline__ void push4(uint32_t dst, uint32_t bar, uint32_t x) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(x), "r"(bar) : "memory");
}
__device__ __forceinline__ void push8(uint32_t dst, uint32_t bar, uint32_t x, uint32_t y) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];"
               ::"r"(dst), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void push16(uint32_t dst, uint32_t bar, uint4 v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar) : "memory");
}
// Waits until the expected bytes have arrived; false (and *abort set to `where`) when they do not within two seconds.
__device__ __forceinline__ bool await_mail(uint32_t bar, volatile int* abort, int where) {
  unsigned long long t0 = 0;
  for (uint32_t spin = 0; spin < (1u << 26); ++spin) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar) : "memory");
    if (ok) return true;
    if ((spin & 255u) == 255u) {
      if (t0 == 0) t0 = ri_tc::global_ns();
      else if (ri_tc::global_ns() - t0 > ri_tc::kWaitLimitNs) break;
      if (*abort) return false;
    }
  }
  *abort = where;
  return false;
}
enum Mail { kMailStats, kMailHigh, kMailLow, kMailCandidates, kMailOut, kMails };

// This thread's clusters, fetched before the scan so that their latency is not on the selection's critical path:
// exact sizes, first row of the first of them, sizes in the 16-bit type.
template <int KEYS>
struct ThreadClusters {
  int cnt[KEYS];
  int off0;
  uint32_t szw[KEYS / 2];

  __device__ __forceinline__ void fetch(const SelectArgs& sel, int g, int lo, int n_loc) {
    const int e0 = threadIdx.x * KEYS;
#pragma unroll
    for (int i = 0; i < KEYS; ++i) cnt[i] = 0;
#pragma unroll
    for (int i = 0; i < KEYS / 2; ++i) szw[i] = 0u;
    off0 = 0;
    const int64_t gc = (int64_t)g * sel.C + lo + e0;
    // volatile: issued here, ahead of the scan, whatever the compiler would prefer.  Slices are multiples of 8, so of a
    // thread's 16 clusters the second eight may lie behind its end.
    if (e0 < n_loc) {
#pragma unroll
      for (int q4 = 0; q4 < KEYS / 4; ++q4)
        if (q4 < 2 || e0 + 8 < n_loc)
          asm volatile("ld.global.nc.v4.s32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(cnt[4 * q4]), "=r"(cnt[4 * q4 + 1]), "=r"(cnt[4 * q4 + 2]), "=r"(cnt[4 * q4 + 3])
                       : "l"(sel.count + gc + 4 * q4));
      asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(off0) : "l"(sel.offset + (int64_t)g * (sel.C + 1) + lo + e0));
      if (KEYS >= 8 && (uintptr_t)sel.size_dt % 16 == 0) {      // 8-byte alignment is all that the sizes need
#pragma unroll
        for (int q8 = 0; q8 < KEYS / 8; ++q8)
          if (q8 == 0 || e0 + 8 < n_loc)
            asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(szw[4 * q8]), "=r"(szw[4 * q8 + 1]), "=r"(szw[4 * q8 + 2]), "=r"(szw[4 * q8 + 3])
                         : "l"(sel.size_dt + gc + 8 * q8));
      } else {
#pragma unroll
        for (int q4 = 0; q4 < KEYS / 4; ++q4)
          if (q4 < 2 || e0 + 8 < n_loc)
            asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(szw[2 * q4]), "=r"(szw[2 * q4 + 1]) : "l"(sel.size_dt + gc + 4 * q4));
      }
    }
  }
};

// Phase 1 for this CTA's slice [lo, hi) of group g: scores into shared memory (s_sc[h * kScoreStride + score_at(e)]), and this
// warp's (max, sum of exponentials) of the rounded scores of head lane / 4.  `meanwhile` runs behind the first copies.
template <int DT, int KEYS, typename F>
__device__ __forceinline__ void scan_slice(const FusedArgs& f, int g, int lo, int hi, uint8_t* ring, float* s_sc, float& m_run,
                                           float& s_run, F meanwhile) {
  constexpr int W = kFusedWarps, kScoreStride = Geom<KEYS>::kScoreStride, ROWS = Geom<KEYS>::kScanRows, NJ = ROWS / 8;
  constexpr int kSlotBytes = ROWS * 256, kSlotStride = W * kSlotBytes;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = lane >> 2, t = lane & 3;
  const int C = f.sel.C, gs = f.sel.gs;
  const uint32_t my_ring = smem_u32(ring) + warp * kSlotBytes + lane * 16;      // stage-major, as in the attend phase
  const uint8_t* my_ring_ptr = ring + warp * kSlotBytes + lane * 16;
  const int n_steps = (hi - lo + ROWS - 1) / ROWS;

  // piece j*4+kk of a stage: row j*8+r of the step, bytes 16*(t+4kk) — the fragment layout of the scan kernel
  auto issue = [&](int step, int stage) {
    const uint32_t dst = my_ring + stage * kSlotStride;
    const int base = lo + step * ROWS;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int row = min(base + j * 8 + r, hi - 1);   // rows past the slice are masked below
      const uint4* p = f.cent + ((int64_t)g * C + row) * 16 + t;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) cp_async16(dst + (j * 4 + kk) * 512, p + kk * 4);
    }
  };

  int s_issue = warp;                                  // a warp takes steps warp, warp+W, ...
#pragma unroll
  for (int st = 0; st < kScanStages; ++st) {
    if (s_issue < n_steps) { issue(s_issue, st); s_issue += W; }
    cp_async_commit();
  }
  uint4 qa[4];
#pragma unroll
  for (int kk = 0; kk < 4; ++kk)
    qa[kk] = r < gs ? ri_ldg16(f.att.q + ((int64_t)g * gs + r) * 16 + t + kk * 4) : make_uint4(0, 0, 0, 0);
  meanwhile();

  m_run = -INFINITY;   // softmax statistics of head r over this warp's centroids
  s_run = 0.f;
  int stage = 0;
#pragma unroll 1
  for (int step = warp; step < n_steps; step += W) {
    cp_async_wait<kScanStages - 1>();
    const uint8_t* src = my_ring_ptr + stage * kSlotStride;
    const int base = lo + step * ROWS;
    // the stage goes to registers and is refilled at once (the same lane wrote it and reads it), so that two stages
    // are in flight while this one is worked on
    uint4 kb[NJ * 4];
#pragma unroll
    for (int i = 0; i < NJ * 4; ++i) kb[i] = *reinterpret_cast<const uint4*>(src + i * 512);
    if (s_issue < n_steps) { issue(s_issue, stage); s_issue += W; }
    cp_async_commit();
    stage ^= 1;
    float rv[NJ][2];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        Elem<DT>::mma16816(acc, qa[kk].x, 0u, qa[kk].y, 0u, kb[j * 4 + kk].x, kb[j * 4 + kk].y);
        Elem<DT>::mma16816(acc, qa[kk].z, 0u, qa[kk].w, 0u, kb[j * 4 + kk].z, kb[j * 4 + kk].w);
      }
      const int c0 = base + j * 8 + 2 * t;
      const float v0 = f.alpha * acc[0], v1 = f.alpha * acc[1];
      const bool ok = r < gs && c0 < hi;               // slices are multiples of 8: a tile is entirely in or out
      if (ok) {
        *reinterpret_cast<float2*>(s_sc + r * kScoreStride + score_at(c0 - lo)) = make_float2(v0, v1);
        if (f.views) *reinterpret_cast<float2*>(f.scores + ((int64_t)g * gs + r) * C + c0) = make_float2(v0, v1);
      }
      rv[j][0] = ok ? Elem<DT>::round(v0) : -INFINITY;
      rv[j][1] = ok ? Elem<DT>::round(v1) : -INFINITY;
    }

    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < NJ; ++j) mx = fmaxf(mx, fmaxf(rv[j][0], rv[j][1]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float m_new = fmaxf(m_run, mx);
    if (m_new > -INFINITY) {
      float add = 0.f;
#pragma unroll
      for (int j = 0; j < NJ; ++j) add += exp2f((rv[j][0] - m_new) * RI_LOG2E) + exp2f((rv[j][1] - m_new) * RI_LOG2E);
      s_run = s_run * exp2f((m_run - m_new) * RI_LOG2E) + add;   // m_run = -inf: factor 0, s_run was 0
      m_run = m_new;
    }
  }
  cp_async_wait<0>();
  s_run += __shfl_xor_sync(0xffffffffu, s_run, 1);
  s_run += __shfl_xor_sync(0xffffffffu, s_run, 2);
}

// Exclusive scan of two 64-bit values per thread at once (one pair of block barriers for both).
// `warp_sums` is used once.
template <int THREADS>
__device__ __forceinline__ void block_scan2(uint64_t& a, uint64_t& b, uint64_t (*warp_sums)[2]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t ia = a, ib = b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t na = __shfl_up_sync(0xffffffffu, ia, o), nb = __shfl_up_sync(0xffffffffu, ib, o);
    if (lane >= o) { ia += na; ib += nb; }
  }
  if (lane == 31) { warp_sums[warp][0] = ia; warp_sums[warp][1] = ib; }
  __syncthreads();
  uint64_t ba = 0, bb = 0;
#pragma unroll
  for (int w = 0; w < THREADS / 32; ++w)
    if (w < warp) { ba += warp_sums[w][0]; bb += warp_sums[w][1]; }
  a = ba + ia - a;
  b = bb + ib - b;
}

// Where a cut falls in a histogram of 256 bins scanned from the top (bin 255 = largest keys): the bin, then the
// keys above that bin and the keys in it — cluster-wide, in the CTAs of lower rank, in this CTA.
struct CutBin { int bin, above_g, above_l, above_m, at_g, at_l, at_m; };

__device__ __forceinline__ void note_cut(CutBin* out, int bin, uint64_t pre, uint64_t v, int k) {
  const int ag = (int)(pre & 0xffffu), cg_ = (int)(v & 0xffffu);
  if (ag < k && ag + cg_ >= k) {
    out->bin = bin; out->above_g = ag; out->above_l = (int)((pre >> 16) & 0xffffu); out->above_m = (int)((pre >> 32) & 0xffffu);
    out->at_g = cg_; out->at_l = (int)((v >> 16) & 0xffffu); out->at_m = (int)((v >> 32) & 0xffffu);
  }
}
// Counts of one bin as a packed triple: cluster-wide | in the CTAs of lower rank | in this CTA.  `h`: the bin in the first CTA's
// histogram, the next CTA's `stride` further.
template <int MAXCL>
__device__ __forceinline__ uint64_t bin_triple(const uint16_t* h, int stride, int cl, int rank, uint32_t mine) {
  uint32_t sum = 0, lower = 0;
  auto add = [&](int rr) {
    const uint32_t w = h[rr * stride];
    sum += w;
    lower += rr < rank ? w : 0u;
  };
#pragma unroll
  for (int rr = 0; rr < 8; ++rr)
    if (rr < cl) add(rr);
  if (MAXCL > 8) {
#pragma unroll
    for (int rr = 8; rr < MAXCL; ++rr)
      if (rr < cl) add(rr);
  }
  return (uint64_t)sum | ((uint64_t)lower << 16) | ((uint64_t)mine << 32);
}
// Eight 32-bit counts as 16-bit ones.
__device__ __forceinline__ uint4 pack_counts(const uint32_t* h) {
  const uint4 a = *reinterpret_cast<const uint4*>(h), b = *reinterpret_cast<const uint4*>(h + 4);
  return make_uint4(a.x | (a.y << 16), a.z | (a.w << 16), b.x | (b.y << 16), b.z | (b.w << 16));
}

// The n lowest of the bits that are set (n may be negative, or more than there are).
__device__ __forceinline__ uint32_t lowest_bits(uint32_t x, int n) {
  if (n <= 0) return 0u;
  while (__popc(x) > n) x &= ~(0x80000000u >> __clz(x));
  return x;
}

// Two values rounded to the 16-bit type.
template <int DT>
__device__ __forceinline__ uint64_t round2(float a, float b) {
  const uint32_t p = Elem<DT>::pack2(a, b);
  return ri_tc::pack_f2(Elem<DT>::from_bits((uint16_t)(p & 0xffffu)), Elem<DT>::from_bits((uint16_t)(p >> 16)));
}

// Phase 2.  The arithmetic and the tie rules are those of the selection body in ri_wave_select.cuh;
// the organisation differs: a thread keeps its keys in registers, the scores come from shared
// memory, and every histogram is scanned as packed triples (cluster-wide count | count in the CTAs of
// lower rank | count in this CTA), so that one scan per radix level yields the cut AND what this CTA
// needs to place its own entries: how many selected keys, and how many ties on each cut, the CTAs of
// lower rank hold (they hold the lower ids, and ties are taken in id order: "ties taken before me" =
// min(ties before me, ties to take)).  The positions in the compacted lists then follow from ONE more
// packed block scan plus closed forms.  A retrieval candidate is pushed to its place in every CTA's list, and every CTA
// applies the page budget on its own copy (ranking it first where the order matters).
// Three exchanges (two histogram levels, candidates).
// What the attend phase needs stays in shared memory (`ll`): this CTA's own estimation entries, the kept
// clusters' row ranges and this CTA's share of the exact steps (balanced against the estimation work
// every CTA has).  Returns 1 when that form is usable; 0 (some CTA holds more estimation entries
// than its list takes) after writing the global lists that the attend steps read instead; -1 when a wait ran out.
template <int DT, int KEYS, int MAXCL, typename F>
__device__ __forceinline__ int select_in_cluster(const FusedArgs& f, int g, int rank, int lo, int n_loc, uint8_t* dyn,
                                                 const float* s_sc, const float* s_max, const float* s_inv, int static_len,
                                                 const ThreadClusters<KEYS>& tc, uint32_t bars, volatile int* abort, LocalLists& ll,
                                                 F meanwhile) {
  constexpr int T = kFusedThreads, kScoreStride = Geom<KEYS>::kScoreStride;
  static_assert(T == 256, "one histogram bin per thread");
  const SelectArgs& a = f.sel;
  const int CL = f.cl;
  uint16_t* rx_high = reinterpret_cast<uint16_t*>(dyn + f.temp_off);      // [CL][256] pushed by every CTA
  uint16_t* rx_low = rx_high + CL * 256;                                   // [CL][2][256]
  uint4* cand = reinterpret_cast<uint4*>(rx_low + CL * 512);              // [p_pad] all P candidates of the group, in id order:
                                                                          //   key<<16 | (0xffff - id), cluster size, first row
  uint32_t* cand_key = reinterpret_cast<uint32_t*>(cand + a.p_pad);       // ranking: the keys, then the three in rank order,
  uint32_t* ranked = cand_key + a.p_pad;                                  // plus the place in the row list
  uint32_t* rcnt = ranked + a.p_pad;
  uint32_t* roff = rcnt + a.p_pad;
  uint4* own = reinterpret_cast<uint4*>(cand_key);                        // [p_pad] before that: this CTA's own candidates

  // lists that outlive this phase
  uint32_t* dstart = reinterpret_cast<uint32_t*>(dyn);                   // [p_pad + 4]
  uint32_t* doff = dstart + a.p_pad + 4;                                 // [p_pad]
  uint32_t* est = doff + a.p_pad;                                        // [cap] index in the slice, size (16-bit type) above it
  float* est_sc = reinterpret_cast<float*>(est + f.cap);                 // [gs][cap]

  __shared__ __align__(16) uint32_t hist1[256], hist2[512];   // bin 255 = largest keys; low bytes at the K cut, at the P cut
  __shared__ CutBin fk, fp, lk, lp;   // high byte of the K and P cuts, then their low bytes
  __shared__ uint32_t rx_nest[MAXCL];   // every CTA's estimation entries
  __shared__ uint32_t warp_sums[T / 32];
  __shared__ uint64_t warp_sums64[3][T / 32];
  __shared__ uint64_t warp_sums2[T / 32][2];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int C = a.C, gs = a.gs;
  hist1[tid] = 0; hist2[tid] = 0; hist2[256 + tid] = 0;
  if (tid == 0) {
    const CutBin z = {0, 0, 0, 0, 0, 0, 0};
    fk = z; fp = z; lk = z; lp = z;
  }
  __syncthreads();

  // ---- keys of this thread's centroids (ids lo + KEYS*tid ..), first-level histogram ----
  const int e0 = tid * KEYS;
  const int n_mine = min(max(n_loc - e0, 0), KEYS);   // slices are multiples of 8: 0, 4, 8 or all 16
  const int64_t gc = (int64_t)g * C + lo + e0;
  uint16_t key[KEYS];
  {
    uint64_t dist2[KEYS / 2];        // two centroids each
#pragma unroll
    for (int i = 0; i < KEYS; ++i) { dist2[i / 2] = 0ull; key[i] = 0; }
    const uint64_t log2e = ri_tc::pack_f2(RI_LOG2E, RI_LOG2E);
    // round(exp(round(s) - max) / sum) of two centroids, two to an instruction where there is one
    auto share = [&](float s0, float s1, int h) {
      const uint64_t x = ri_tc::mul_f2(ri_tc::add_f2(round2<DT>(s0, s1), ri_tc::pack_f2(-s_max[h], -s_max[h])), log2e);
      float x0, x1;
      ri_tc::unpack_f2(x, x0, x1);
      ri_tc::unpack_f2(ri_tc::mul_f2(ri_tc::pack_f2(exp2f(x0), exp2f(x1)), ri_tc::pack_f2(s_inv[h], s_inv[h])), x0, x1);
      return round2<DT>(x0, x1);
    };
    if (n_mine > 0) {
#pragma unroll
      for (int h = 0; h < kMaxHeads; ++h)
        if (h < gs) {
#pragma unroll
          for (int q4 = 0; q4 < KEYS / 4; ++q4) {      // behind the slice's end: scores that are never used
            const float4 s4 = *reinterpret_cast<const float4*>(s_sc + h * kScoreStride + score_at(e0 + 4 * q4));
            dist2[2 * q4] = ri_tc::add_f2(dist2[2 * q4], share(s4.x, s4.y, h));
            dist2[2 * q4 + 1] = ri_tc::add_f2(dist2[2 * q4 + 1], share(s4.z, s4.w, h));
          }
        }
#pragma unroll
      for (int i = 0; i < KEYS; ++i)
        if (i < n_mine) {
          float d0, d1;
          ri_tc::unpack_f2(dist2[i / 2], d0, d1);
          uint16_t b = Elem<DT>::bits(i & 1 ? d1 : d0);
          if (tc.cnt[i] == 0) b = DT == RI_BF16 ? 0xFF7Fu : 0xFBFFu;   // most negative finite value
          key[i] = ri_ordered_key(b);
          atomicAdd(&hist1[key[i] >> 8], 1u);
        }
      if (f.views)
#pragma unroll
        for (int q4 = 0; q4 < KEYS / 4; ++q4)
          if (4 * q4 < n_mine)
            *reinterpret_cast<uint2*>(a.dist_keys + gc + 4 * q4) =
                make_uint2(key[4 * q4] | ((uint32_t)key[4 * q4 + 1] << 16), key[4 * q4 + 2] | ((uint32_t)key[4 * q4 + 3] << 16));
    }
  }
  __syncthreads();
  RI_FT(3);

  // ---- high byte of the two cuts: thread tid looks after bin 255 - tid ----
#pragma unroll 1
  for (int dst = warp; dst < (MAXCL > 8 ? CL : min(CL, warp + 1)); dst += T / 32)      // a lane pushes eight bins
    push16(peer(smem_u32(rx_high + rank * 256 + lane * 8), dst), peer(bars + 8 * kMailHigh, dst), pack_counts(hist1 + lane * 8));
  const int K = a.P + a.E;
  const int my_bin = 255 - tid;
  await_mail(bars + 8 * kMailHigh, abort, 52);
  RI_FT(4);
  {
    const uint64_t v = bin_triple<MAXCL>(rx_high + my_bin, 256, CL, rank, hist1[my_bin]);
    uint64_t total;
    const uint64_t pre = block_scan<T, uint64_t, false>(v, warp_sums64[0], total);
    note_cut(&fk, my_bin, pre, v, K);
    note_cut(&fp, my_bin, pre, v, a.P);
    __syncthreads();
  }
  const int binK = fk.bin, binP = fp.bin;

  // ---- low byte ----
#pragma unroll
  for (int i = 0; i < KEYS; ++i)
    if (i < n_mine) {
      if ((key[i] >> 8) == binK) atomicAdd(&hist2[key[i] & 255], 1u);
      if ((key[i] >> 8) == binP) atomicAdd(&hist2[256 + (key[i] & 255)], 1u);
    }
  __syncthreads();
#pragma unroll 1
  for (int dst = warp; dst < (MAXCL > 8 ? CL : min(CL, warp + 1)); dst += T / 32)
#pragma unroll
    for (int u = 0; u < 2; ++u)
      push16(peer(smem_u32(rx_low + rank * 512 + u * 256 + lane * 8), dst), peer(bars + 8 * kMailLow, dst),
             pack_counts(hist2 + u * 256 + lane * 8));
  await_mail(bars + 8 * kMailLow, abort, 53);
  RI_FT(5);
  {
    const uint64_t va = bin_triple<MAXCL>(rx_low + my_bin, 512, CL, rank, hist2[my_bin]);
    const uint64_t vb = bin_triple<MAXCL>(rx_low + 256 + my_bin, 512, CL, rank, hist2[256 + my_bin]);
    uint64_t pa = va, pb = vb;
    block_scan2<T>(pa, pb, warp_sums2);
    note_cut(&lk, my_bin, pa, va, K - fk.above_g);
    note_cut(&lp, my_bin, pb, vb, a.P - fp.above_g);
    __syncthreads();
  }
  RI_FT(14);
  const uint16_t TK = (uint16_t)((binK << 8) | lk.bin), TP = (uint16_t)((binP << 8) | lp.bin);
  const int needK = K - fk.above_g - lk.above_g;      // how many keys equal to TK are taken (cluster-wide)
  const int needP = a.P - fp.above_g - lp.above_g;
  // the CTAs of lower rank: ties on each cut, and selected keys (those above the cut plus the ties they take)
  const int tieK_before = lk.at_l, tieP_before = lp.at_l;
  const int inK_before = fk.above_l + lk.above_l + min(needK, tieK_before);
  const int inP_before = fp.above_l + lp.above_l + min(needP, tieP_before);
  const int remK = max(needK - tieK_before, 0), remP = max(needP - tieP_before, 0);   // ties this CTA and later ones take

  // ---- ordered compaction ----
  uint32_t gtK = 0, eqK = 0, gtP = 0, eqP = 0;     // of this thread's keys: those above and on the two cuts
#pragma unroll
  for (int i = 0; i < KEYS; ++i)
    if (i < n_mine) {
      gtK |= (uint32_t)(key[i] > TK) << i; eqK |= (uint32_t)(key[i] == TK) << i;
      gtP |= (uint32_t)(key[i] > TP) << i; eqP |= (uint32_t)(key[i] == TP) << i;
    }
  // 16-bit counters: above K cut | on K cut | above P cut | on P cut
  uint64_t c4_total;
  const uint64_t pre = block_scan<T, uint64_t, false>(
      (uint64_t)(__popc(gtK) | (__popc(eqK) << 16)) | ((uint64_t)(__popc(gtP) | (__popc(eqP) << 16)) << 32), warp_sums64[1], c4_total);
  const int eqK0 = (int)((pre >> 16) & 0xffffu), eqP0 = (int)(pre >> 48);
  const int posP0 = (int)((pre >> 32) & 0xffffu) + min(eqP0, remP);        // taken keys before this thread's, in this CTA
  const int est0 = (int)(pre & 0xffffu) + min(eqK0, remK) - posP0;
  const uint32_t retrieved = gtP | lowest_bits(eqP, remP - eqP0), estimated = (gtK | lowest_bits(eqK, remK - eqK0)) & ~retrieved;
  const int my_ret = (int)((c4_total >> 32) & 0xffffu) + min((int)(c4_total >> 48), remP);
  const int my_est = (int)(c4_total & 0xffffu) + min((int)((c4_total >> 16) & 0xffffu), remK) - my_ret;
  RI_FT(6);
  auto size_bits = [&](int i) { return (tc.szw[i >> 1] >> (16 * (i & 1))) & 0xffffu; };
  {
    int pos = est0;
#pragma unroll
    for (int i = 0; i < KEYS; ++i)
      if (estimated >> i & 1u) {      // the scores follow below, one entry per thread
        if (pos < f.cap) est[pos] = (uint32_t)(e0 + i) | (size_bits(i) << 16);
        ++pos;
      }
  }
  if (retrieved) {
    int pos = posP0, off = tc.off0;
#pragma unroll
    for (int i = 0; i < KEYS; ++i) {
      if (retrieved >> i & 1u) {
        if (pos < a.P) own[pos] = make_uint4(((uint32_t)key[i] << 16) | (uint32_t)(0xffff - (lo + e0 + i)), (uint32_t)tc.cnt[i], (uint32_t)off, 0u);
        ++pos;
      }
      off += tc.cnt[i];
    }
  }
  if (tid < CL) push4(peer(smem_u32(rx_nest + rank), tid), peer(bars + 8 * kMailCandidates, tid), (uint32_t)my_est);
  meanwhile();
  __syncthreads();
  // the pushes in dense warps: st.async from a few lanes of every warp, key after key, took 9 us for 16 keys a thread
#pragma unroll 1
  for (int dst = warp; dst < (MAXCL > 8 ? CL : min(CL, warp + 1)); dst += T / 32)
    for (int j = lane; j < my_ret; j += 32)
      if (inP_before + j < a.P) push16(peer(smem_u32(cand + inP_before + j), dst), peer(bars + 8 * kMailCandidates, dst), own[j]);
  // log2-domain scores of the estimation entries, entry by entry (uniform work, consecutive stores)
  for (int j = tid; j < min(my_est, f.cap); j += T) {
    const int e = score_at((int)(est[j] & 0xffffu));
#pragma unroll
    for (int h = 0; h < kMaxHeads; ++h)
      if (h < gs) est_sc[h * f.cap + j] = s_sc[h * kScoreStride + e] * RI_LOG2E;
  }
  RI_FT(7);
  await_mail(bars + 8 * kMailCandidates, abort, 54);
  __syncthreads();
  if (*abort) return -1;
  RI_FT(16);

  // Page budget (wave_buffer_cpu.cpp:207-216): the clusters are taken in rank order while their pages fit.
  // When ALL P candidates fit — the usual case — the order plays no part in what is attended, so unless the
  // caller wants the ranked ids the ranking is skipped and the rows are laid out in cluster-id order: one scan.
  constexpr int kPer = 1024 / T;    // P <= 1024
  int pc[kPer], pages[kPer];
  // pages (low half) and rows (high half) of the candidates in id order, one packed scan
  uint64_t pr = 0;
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int i = tid * kPer + u;
    pc[u] = i < a.P ? (int)cand[i].y : 0;
    pages[u] = f.page_shift >= 0 ? (pc[u] + a.page - 1) >> f.page_shift : (pc[u] + a.page - 1) / a.page;
    pr += (uint64_t)(uint32_t)pages[u] | ((uint64_t)(uint32_t)pc[u] << 32);
  }
  uint64_t pr_total;
  const uint64_t pr_pre = block_scan<T, uint64_t, false>(pr, warp_sums64[2], pr_total);
  int keep, rows_kept;
  if (!f.views && (int)(uint32_t)pr_total <= a.buffer_pages) {
    // everything fits: id order serves as the order of the row list, each cluster starts at the rows before it
    keep = a.P;
    rows_kept = (int)(pr_total >> 32);
    uint32_t row_start = (uint32_t)(pr_pre >> 32);
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = tid * kPer + u;
      if (i < a.P) {
        dstart[i] = row_start;
        doff[i] = cand[i].z;
      }
      row_start += (uint32_t)pc[u];
    }
    RI_FT(17);
  } else {
    for (int i = tid; i < a.p_pad; i += T) cand_key[i] = i < a.P ? cand[i].x : 0u;   // padding compares below every real candidate
    __syncthreads();
    {
      // rank = number of larger candidates (distinct values: distinct ranks); four lanes share a candidate,
      // each counting over a quarter of the list
      const int quads = a.p_pad / 4, seg = tid & 3;
      const int q_lo = quads * seg / 4, q_hi = quads * (seg + 1) / 4;
      for (int base = 0; base < a.P; base += T / 4) {      // uniform trip count: the shuffles below need whole warps
        const int i = base + (tid >> 2);
        const uint32_t mine = i < a.P ? cand_key[i] : 0xffffffffu;
        int r0 = 0, r1 = 0;
        int q = q_lo;
        for (; q + 2 <= q_hi; q += 2) {
          const uint4 c0 = *reinterpret_cast<const uint4*>(cand_key + 4 * q), c1 = *reinterpret_cast<const uint4*>(cand_key + 4 * q + 4);
          r0 += (c0.x > mine) + (c0.y > mine) + (c0.z > mine) + (c0.w > mine);
          r1 += (c1.x > mine) + (c1.y > mine) + (c1.z > mine) + (c1.w > mine);
        }
        if (q < q_hi) {
          const uint4 c = *reinterpret_cast<const uint4*>(cand_key + 4 * q);
          r0 += (c.x > mine) + (c.y > mine) + (c.z > mine) + (c.w > mine);
        }
        int rk = r0 + r1;
        rk += __shfl_xor_sync(0xffffffffu, rk, 1);
        rk += __shfl_xor_sync(0xffffffffu, rk, 2);
        if (seg == 0 && i < a.P) {
          ranked[rk] = mine;
          rcnt[rk] = cand[i].y;
          roff[rk] = cand[i].z;
        }
      }
    }
    __syncthreads();
    uint32_t psum = 0, total;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = tid * kPer + u;
      pc[u] = i < a.P ? (int)rcnt[i] : 0;
      pages[u] = (pc[u] + a.page - 1) / a.page;
      psum += (uint32_t)pages[u];
    }
    uint32_t before = block_scan<T, uint32_t>(psum, warp_sums, total);
    RI_FT(17);
    // pages are non-negative, so the clusters that fit the budget form a prefix of the order
    bool fits[kPer];
    uint32_t nfit = 0, rsum = 0;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      before += (uint32_t)pages[u];
      fits[u] = tid * kPer + u < a.P && (int)before <= a.buffer_pages;
      nfit += fits[u] ? 1u : 0u;
      rsum += fits[u] ? (uint32_t)pc[u] : 0u;
    }
    // kept count (<= 1024) in the high 12 bits, kept rows (< 2^20) in the low 20
    uint32_t both_total;
    const uint32_t both_pre = block_scan<T, uint32_t>((nfit << 20) | rsum, warp_sums, both_total);
    uint32_t row_start = both_pre & 0xfffffu;
    keep = (int)(both_total >> 20);
    rows_kept = (int)(both_total & 0xfffffu);
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = tid * kPer + u;
      if (i < keep) {
        dstart[i] = row_start;
        doff[i] = roff[i];
      }
      row_start += fits[u] ? (uint32_t)pc[u] : 0u;
    }
  }
  if (tid == 0) dstart[keep] = (uint32_t)rows_kept;
  RI_FT(8);

  // ---- this CTA's share of the exact steps (every warp works it out: lane c stands for CTA c) ----
  // Level the cost units (kCostEst per estimation step a CTA already has,
  // kCostExact per exact step to hand out) so that sum_c max(0, level - e_c) >= X, then cut the exact steps at the
  // running sums.
  // Two rounds of levelling (CTAs above the first level drop out of the second) are enough in practice; whatever
  // imbalance is left only costs time.
  const int n_e = lane < CL ? (int)rx_nest[lane] : 0;
  {
    const int xs_total = (static_len + rows_kept + 15) / 16;
    const int X = f.att.cost_exact * xs_total;
    const int e_u = f.att.cost_est * ((n_e + 15) / 16);
    bool act = lane < CL;
    int level = 0;
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int sum_e = __reduce_add_sync(0xffffffffu, act ? e_u : 0);
      const int n = __popc(__ballot_sync(0xffffffffu, act));                             // >= 1: the least loaded CTA stays
      level = (int)__fdividef((float)(X + sum_e + n - 1), (float)n);
      act = act && e_u <= level;
    }
    const int x_u = lane < CL ? max(0, level - e_u) : 0;
    const int before = __reduce_add_sync(0xffffffffu, lane < rank ? x_u : 0);
    const int mine = __shfl_sync(0xffffffffu, x_u, rank);
    ll.x_lo = min(xs_total, (before + f.att.cost_exact - 1) / f.att.cost_exact);
    ll.x_hi = rank == CL - 1 ? xs_total : min(xs_total, (before + mine + f.att.cost_exact - 1) / f.att.cost_exact);
  }
  const bool local = __reduce_max_sync(0xffffffffu, n_e) <= f.cap;
  ll.est = est; ll.est_sc = est_sc;
  ll.cap = f.cap; ll.n_est = my_est; ll.slice_lo = lo;
  ll.dstart = dstart; ll.doff = doff; ll.keep = keep; ll.n_rows = rows_kept;
  __syncthreads();

  RI_FT(18);
  // ---- the global lists: for callers that asked for them, and for the attend steps when the lists above
  //      do not fit ----
  if (f.views || !local) {
    int pe = inK_before - inP_before + est0;        // behind the estimation entries in the CTAs of lower rank
#pragma unroll
    for (int i = 0; i < KEYS; ++i)
      if (estimated >> i & 1u) {
        if (pe < a.E) {
          a.est_ids[(int64_t)g * a.e_pad + pe] = lo + e0 + i;
          a.est_w[(int64_t)g * a.e_pad + pe] = Elem<DT>::from_bits((uint16_t)size_bits(i));
          for (int h = 0; h < gs; ++h)
            a.est_s2[((int64_t)g * kMaxHeads + h) * a.e_pad + pe] = s_sc[h * kScoreStride + score_at(e0 + i)] * RI_LOG2E;
          if (a.estimated_ids) a.estimated_ids[(int64_t)g * a.E + pe] = lo + e0 + i;
        }
        ++pe;
      }
    // the cluster's warps share the kept clusters out
    for (int i = rank * (T / 32) + warp; i < keep; i += CL * (T / 32)) {
      const int o = (int)doff[i], start = (int)dstart[i], n = (int)dstart[i + 1] - start;
      for (int j = lane; j < n; j += 32)
        if (start + j < a.max_rows) a.rows[(int64_t)g * a.max_rows + start + j] = o + j;
    }
    if (rank == 0) {
      if (tid == 0) {
        a.n_exact[g] = rows_kept;
        if (a.retrieved_kept) a.retrieved_kept[g] = keep;
      }
      if (a.retrieved_ids)
        for (int i = tid; i < a.P; i += T) a.retrieved_ids[(int64_t)g * a.P + i] = 0xffff - (int)(ranked[i] & 0xffffu);
    }
    __syncthreads();    // the arrays read above lie where a faster warp is about to fill the ring
  }
  if (!local) {         // the global lists are read by the other CTAs of the cluster in the next phase
    __threadfence();
    cluster_arrive();
    cluster_wait();
  }
  return local ? 1 : 0;
}

template <int DT, int KEYS, int MAXCL>
__global__ void __launch_bounds__(kFusedThreads, 1) wave_fused_kernel(FusedArgs f) {
  extern __shared__ __align__(128) uint8_t dyn[];
  __shared__ float s_max[kMaxHeads], s_inv[kMaxHeads];
  __shared__ float sm_m[kFusedWarps][kMaxHeads], sm_l[kFusedWarps][kMaxHeads];
  __shared__ __align__(8) uint64_t s_bars[kMails];
  __shared__ int s_abort;
  using Geo = Geom<KEYS>;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), CL = f.cl;
  const int g = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, t = lane & 3;
  const int C = f.sel.C, gs = f.sel.gs;
  const int lo = min(C, rank * f.sel.slice), hi = min(C, lo + f.sel.slice);
  float* s_sc = reinterpret_cast<float*>(dyn + f.scores_off);
  float2* rx_stat = reinterpret_cast<float2*>(dyn + f.mail_off);             // [CL][warps][heads] (max, sum)
  // partial outputs pushed to this CTA, which finishes chunks (4 channels of a head) first .. first + own - 1 of the group's
  const int per = chunks_per_cta(gs, CL), first = rank * per, own = min(max(gs * 32 - first, 0), per);
  float4* rx_out = reinterpret_cast<float4*>(rx_stat + CL * kFusedWarps * kMaxHeads);      // [CL][per]
  float2* rx_ml = reinterpret_cast<float2*>(rx_out + CL * per);                             // [CL][per] (max, sum)
  const uint32_t bars = smem_u32(s_bars);
  volatile int* abort = &s_abort;

  // one phase each; what will arrive is known from the start
  if (tid == 0) {
    s_abort = 0;
    const int bytes[kMails] = {CL * kFusedWarps * kMaxHeads * 8, CL * 512, CL * 1024, f.sel.P * 16 + CL * 4, own * CL * 24};
    for (int i = 0; i < kMails; ++i) ri_tc::mbar_init(bars + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int i = 0; i < kMails; ++i) ri_tc::mbar_arrive_expect_tx(bars + 8 * i, bytes[i]);
  }
  cluster_arrive();
  ri_pdl_trigger();
  // the scan's first rows on their way into L2 while the kernel in front ends (nothing is read before the wait)
  {
    const uint8_t* from = reinterpret_cast<const uint8_t*>(f.cent + ((int64_t)g * C + lo) * 16);
    const int lines = min((hi - lo) * 2, Geo::kScanRing / 128);
    for (int i = tid; i < lines; i += kFusedThreads) asm volatile("prefetch.global.L2 [%0];" ::"l"(from + (int64_t)i * 128));
  }
  ri_pdl_wait();

  int static_len;     // fetched now (not where the compiler would sink the load to: the middle of phase 2)
  asm volatile("ld.global.b32 %0, [%1];" : "=r"(static_len) : "l"(f.att.static_len));
  ThreadClusters<KEYS> tc;
  uint4 new_row = make_uint4(0u, 0u, 0u, 0u);        // this step's key (lanes 0..15) and value row: CTA 0's first warp
  const bool appends = f.att.new_k != nullptr && rank == 0 && warp == 0;

  // ---- phase 1: scores of this CTA's slice ----
  RI_FT(0);
  float m_run, s_run;
  scan_slice<DT, KEYS>(f, g, lo, hi, dyn, s_sc, m_run, s_run, [&] {
    tc.fetch(f.sel, g, lo, hi - lo);
    if (appends) {
      const uint4* from = (lane < 16 ? f.att.new_k : f.att.new_v) + (int64_t)g * 16 + (lane & 15);
      asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(new_row.x), "=r"(new_row.y), "=r"(new_row.z), "=r"(new_row.w) : "l"(from));
    }
  });
  RI_FT(1);
  cluster_wait();     // every CTA's barriers are set up (they arrived before their scans)
  for (int dst = t; dst < CL; dst += 4)
    push8(peer(smem_u32(rx_stat + (rank * kFusedWarps + warp) * kMaxHeads + r), dst), peer(bars + 8 * kMailStats, dst),
          __float_as_uint(m_run), __float_as_uint(s_run));
  if (warp < gs) {     // warp h: head h
    await_mail(bars + 8 * kMailStats, abort, 51);
    constexpr int kPer = MAXCL * kFusedWarps / 32;
    float m[kPer], M = -INFINITY, S = 0.f;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = u * 32 + lane;
      m[u] = i < CL * kFusedWarps ? rx_stat[i * kMaxHeads + warp].x : -INFINITY;
      M = fmaxf(M, m[u]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
#pragma unroll
    for (int u = 0; u < kPer; ++u)
      if (m[u] > -INFINITY) S += rx_stat[(u * 32 + lane) * kMaxHeads + warp].y * exp2f((m[u] - M) * RI_LOG2E);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) S += __shfl_xor_sync(0xffffffffu, S, o);
    if (lane == 0) { s_max[warp] = M; s_inv[warp] = 1.0f / S; }
  }

  // ---- phase 2: selection (its arrays lie where the scan's ring was) ----
  RI_FT(2);
  LocalLists ll;
  const int form = select_in_cluster<DT, KEYS, MAXCL>(f, g, rank, lo, hi - lo, dyn, s_sc, s_max, s_inv, static_len, tc, bars, abort, ll, [&] {
    // the steady zone gets the new token's rows; the attend steps of this kernel take them from where they came from
    if (appends && static_len >= 1 && static_len <= f.att.steady_stride)
      (lane < 16 ? f.steady_k_w : f.steady_v_w)[((int64_t)g * f.att.steady_stride + static_len - 1) * 16 + (lane & 15)] = new_row;
  });
  RI_FT(9);

  if (form >= 0) {
    // ---- phase 3: attention over the estimation and exact rows selected above ----
    uint8_t* ring = dyn + f.ring_off;
    Partial part;
    if (form == 1)
      attend_steps<DT, true, kFusedWarps, Geo::kAttendStages>(f.att, g, rank, CL, static_len, static_len + ll.n_rows, ring, &ll, part);
    else
      attend_steps<DT, false, kFusedWarps, Geo::kAttendStages>(f.att, g, rank, CL, static_len, static_len + ll.n_rows, ring, nullptr, part);

    // ---- merge the warps of this CTA (each parks its accumulator in its own idle ring region), a thread per chunk ----
    float l_run = part.l;
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
    if (t == 0) { sm_m[warp][r] = part.m; sm_l[warp][r] = l_run; }
    park_partial(part, reinterpret_cast<float*>(ring + warp * kStageBytes));
    __syncthreads();
    if (tid < gs * 32) {
      const int h = tid >> 5;
      float M = -INFINITY, L = 0.f;
      float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < kFusedWarps; ++w) M = fmaxf(M, sm_m[w][h]);
      const float Ms = M == -INFINITY ? 0.f : M;
#pragma unroll
      for (int w = 0; w < kFusedWarps; ++w) {
        const float x = exp2f(sm_m[w][h] - Ms);
        const float4 o = *reinterpret_cast<const float4*>(ring + w * kStageBytes + tid * 16);
        L += sm_l[w][h] * x;
        O.x += o.x * x; O.y += o.y * x; O.z += o.z * x; O.w += o.w * x;
      }
      const int dst = tid / per, slot = rank * per + tid - dst * per;
      const uint32_t bar = peer(bars + 8 * kMailOut, dst);
      push16(peer(smem_u32(rx_out + slot), dst), bar,
             make_uint4(__float_as_uint(O.x), __float_as_uint(O.y), __float_as_uint(O.z), __float_as_uint(O.w)));
      push8(peer(smem_u32(rx_ml + slot), dst), bar, __float_as_uint(M), __float_as_uint(L));
    }
    RI_FT(12);

    // ---- merge the partial results of the group's CTAs: this CTA finishes its chunks ----
    if (tid < own && await_mail(bars + 8 * kMailOut, abort, 55)) {
      float M = -INFINITY, L = 0.f;
      float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
      float2 ml[MAXCL];
#pragma unroll
      for (int c = 0; c < MAXCL; ++c) {
        ml[c] = c < CL ? rx_ml[c * per + tid] : make_float2(-INFINITY, 0.f);
        M = fmaxf(M, ml[c].x);
      }
      const float Ms = M == -INFINITY ? 0.f : M;
#pragma unroll
      for (int c = 0; c < MAXCL; ++c)
        if (c < CL) {
          const float x = exp2f(ml[c].x - Ms);
          const float4 o = rx_out[c * per + tid];
          L += ml[c].y * x;
          O.x += o.x * x; O.y += o.y * x; O.z += o.z * x; O.w += o.w * x;
        }
      const float inv[4] = {O.x, O.y, O.z, O.w};
      uint16_t bits[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) bits[i] = Elem<DT>::bits(L > 0.f ? inv[i] / L : 0.f);
      const int64_t at = (int64_t)g * gs * RI_HEAD_DIM + (first + tid) * 4;
      uint16_t* out = reinterpret_cast<uint16_t*>(f.att.out) + at;
      const uint2 all = make_uint2(bits[0] | ((uint32_t)bits[1] << 16), bits[2] | ((uint32_t)bits[3] << 16));
      auto store = [&](uint16_t* to, bool aligned) {
        if (aligned) {
          *reinterpret_cast<uint2*>(to) = all;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) to[i] = bits[i];
        }
      };
      store(out, f.out_aligned);
      for (int c = 0; c < f.att.n_copies; ++c) {    // several GPUs: every rank's gather buffer
        uint16_t* to = f.att.copies[c] + at;
        store(to, (uintptr_t)to % 8 == 0);
      }
    }
    RI_FT(13);
  }
  // A CTA leaves when all that was meant for it has arrived.  One that gave up does not know that: it waits here until the
  // others have left or gave up too (a CTA that has left counts as arrived).  Twice, because the others' next barrier may be the
  // one behind the global lists, after which they still push; and a while longer, for what a CTA pushed just before it left.
  __syncthreads();
  if (s_abort) {
    if (tid == 0) {
      *f.status = s_abort;
      if (f.gather_error) *f.gather_error = kSliceMissing;
    }
    cluster_arrive();
    cluster_wait();
    cluster_arrive();
    cluster_wait();
    for (int i = 0; i < 20; ++i) __nanosleep(1000);
  }
}

// After the decode kernel of the same stream: raise this rank's flag on every rank, then wait (bounded) until
// every rank's flag here holds this step's epoch.  Thread r looks after rank r.  Where the decode kernel left a slice out, no flag
// is raised: the other ranks' waits run out and say so too.
__global__ void gather_signal_wait_kernel(uint32_t* const* flag_slots, const uint32_t* flags, const uint32_t* epoch,
                                          int32_t* error, int n_ranks, long long limit_ns, unsigned long long* stamps) {
  ri_pdl_enter();
  const int r = threadIdx.x;
  unsigned long long t_in;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_in));
  const uint32_t expected = *epoch;
  if (__syncthreads_or(*error == kSliceMissing)) {     // both words are on their way at once
    if (r == 0) *error = 1;
    return;
  }
  if (r >= n_ranks) return;
  // the decode kernel has completed (stream order), so its stores to the other GPUs happen before this fence,
  // and the fence orders them before the flag at system scope
  asm volatile("fence.acq_rel.sys;" ::: "memory");
  asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(flag_slots[r]), "r"(expected) : "memory");
  unsigned long long t0;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  long long spins = 0;
  for (;;) {
    uint32_t v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flags + r) : "memory");
    if ((int32_t)(v - expected) >= 0) break;
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if ((long long)(now - t0) > limit_ns || ++spins > (1ll << 26)) { *error = 1; break; }   // give up: time or count
    __nanosleep(64);
  }
  if (stamps != nullptr) {       // entry | flags raised | last flag seen (the maximum over the threads)
    unsigned long long t_out;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_out));
    if (r == 0) { stamps[0] = t_in; stamps[1] = t0; }
    atomicMax(stamps + 2, t_out);      // the timer only grows, so the latest call's maximum wins
  }
}

// ---- host side ----------------------------------------------------------------------------------------------------
// Where things lie in the dynamic shared memory for clusters of `cl` CTAs; false where they do not fit.
int g_cap_limit = -1;   // ri_wave_test_local_cap

int slice_of(int n_centroids, int cl) { return ((n_centroids / 8 + cl - 1) / cl) * 8; }
int keys_of(int slice) { return slice <= 4 * kFusedThreads ? 4 : slice <= 8 * kFusedThreads ? 8 : 16; }

template <int KEYS>
bool lay_out(const ri_wave_layer& p, int cl, int budget, FusedArgs* f) {
  using Geo = Geom<KEYS>;
  const int p_pad = (int)ri_align_up(p.nprobe, 4), gs = p.group_size;
  const int mail_off = (budget - mail_bytes(gs, cl)) & ~127;
  const int scores_off = (mail_off - gs * Geo::kScoreStride * (int)sizeof(float)) & ~127;
  const int ring_off = (mail_off - Geo::kAttendRing) & ~127;
  const int room = (scores_off - temp_bytes(p_pad, cl) < ring_off ? scores_off - temp_bytes(p_pad, cl) : ring_off) - range_bytes(p_pad) - 16;
  if (slice_of(p.n_centroids, cl) > Geo::kMaxSlice || Geo::kScanRing > scores_off || room < 0) return false;
  int cap = room / entry_bytes(gs);
  if (g_cap_limit >= 0 && cap > g_cap_limit) cap = g_cap_limit;
  cap = (cap > Geo::kMaxSlice ? Geo::kMaxSlice : cap) & ~15;
  f->cap = cap;
  f->temp_off = (int)ri_align_up(range_bytes(p_pad) + (int64_t)cap * entry_bytes(gs), 16);
  f->scores_off = scores_off; f->ring_off = ring_off; f->mail_off = mail_off; f->cl = cl;
  f->sel.slice = slice_of(p.n_centroids, cl);
  return true;
}

// Per device: the shared memory the kernel's one CTA per SM may use, and how many clusters of each size the device can hold
// at once (clusters are placed inside one GPC, so that is less than SMs / size: a B200 with 148 SMs holds 15 clusters of
// 8 or 7 CTAs, 22 of 6, 26 of 5, 33 of 4).
struct Device { int budget; int fit[kMaxCluster + 1]; };   // fit: of up to MAXCL CTAs

template <int DT, int KEYS, int MAXCL>
int ask_device(Device* out) {
  static Device cached[64];
  static std::atomic<bool> known[64];
  int dev = 0;
  RI_CUDA_OK(cudaGetDevice(&dev));
  const bool track = dev >= 0 && dev < 64;
  if (track && known[dev].load(std::memory_order_acquire)) { *out = cached[dev]; return RI_OK; }
  static std::mutex lock;
  std::lock_guard<std::mutex> hold(lock);
  int per_sm = 0, reserved = 0, optin = 0, sms = 0;
  RI_CUDA_OK(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
  RI_CUDA_OK(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev));
  RI_CUDA_OK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  RI_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  cudaFuncAttributes fa;
  RI_CUDA_OK(cudaFuncGetAttributes(&fa, wave_fused_kernel<DT, KEYS, MAXCL>));
  if (MAXCL > 8)
    RI_CUDA_OK(cudaFuncSetAttribute(wave_fused_kernel<DT, KEYS, MAXCL>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  Device d;
  d.budget = ((per_sm - reserved < optin ? per_sm - reserved : optin) - (int)fa.sharedSizeBytes) & ~127;
  RI_CUDA_OK(cudaFuncSetAttribute(wave_fused_kernel<DT, KEYS, MAXCL>, cudaFuncAttributeMaxDynamicSharedMemorySize, d.budget));
  for (int cl = 0; cl <= kMaxCluster; ++cl) d.fit[cl] = 0;
  for (int cl = MAXCL > 8 ? 9 : 1; cl <= MAXCL; ++cl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cl, 64);
    cfg.blockDim = dim3(kFusedThreads);
    cfg.dynamicSmemBytes = (size_t)d.budget;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cl;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&d.fit[cl], wave_fused_kernel<DT, KEYS, MAXCL>, &cfg) != cudaSuccess || d.fit[cl] <= 0) {
      (void)cudaGetLastError();
      d.fit[cl] = cl > 8 ? 0 : sms / cl;       // the query is unavailable: the bound that ignores GPC boundaries
    }
  }
  if (track) {
    cached[dev] = d;
    known[dev].store(true, std::memory_order_release);
  }
  *out = d;
  return RI_OK;
}

template <int DT, int KEYS, int MAXCL = 8>
int launch(const ri_wave_layer& p, const Layout& L, int cl, cudaStream_t s, const ri_wave_gather* gather) {
  FusedArgs f;
  Device d;
  int rc = ask_device<DT, KEYS, MAXCL>(&d);
  if (rc != RI_OK || (rc = fill_select_args(p, L, f.sel)) != RI_OK) return rc;
  fill_attend_args(p, L, nullptr, f.att);
  f.cent = static_cast<const uint4*>(p.d_centroids);
  f.scores = reinterpret_cast<float*>(static_cast<uint8_t*>(p.d_scratch) + L.scores);
  f.status = ri_status_word();
  if (!f.status) return RI_ERR_CUDA;
  f.alpha = 0.08838834764831845f;
  f.views = p.d_retrieved_ids != nullptr;
  f.att.new_k = static_cast<const uint4*>(p.d_new_keys);
  f.att.new_v = static_cast<const uint4*>(p.d_new_values);
  f.steady_k_w = static_cast<uint4*>(const_cast<void*>(p.d_steady_keys));
  f.steady_v_w = static_cast<uint4*>(const_cast<void*>(p.d_steady_values));
  f.page_shift = -1;
  for (int i = 0; i < 20; ++i)
    if (p.page_size == 1 << i) f.page_shift = i;
  f.out_aligned = (uintptr_t)p.d_out % 8 == 0;
  f.gather_error = gather ? gather->d_error : nullptr;
  if (gather) {
    f.att.copies = reinterpret_cast<uint16_t* const*>(gather->d_out_slots);
    f.att.n_copies = gather->n_ranks;
  }
  RI_REQUIRE(lay_out<KEYS>(p, cl, d.budget, &f), "the single-kernel path does not take this geometry");
  RI_CUDA_OK(ri_launch_pdl_cluster(5, cl, wave_fused_kernel<DT, KEYS, MAXCL>, dim3(cl, p.groups), dim3(kFusedThreads), (size_t)d.budget, s, f));
  return RI_OK;
}

int cluster_size(const ri_wave_layer& p, const Device& d, const Device& big) {
  // The largest size with which all groups' clusters are resident at once (a cluster that has to wait for another one to
  // finish doubles the layer's time), as long as a CTA's slice is worth its share of the exchanges.  us a layer, one group of
  // 11776 centroids: 28.7 with 8 CTAs, 20.4 with 16; four groups of 992: 12.7 with 8, 13.6 with 16; eight of 512: 11.1 with 4,
  // 11.4 with 8, 15.8 with one.
  int cl = kMaxCluster;
  while (cl > 1 && p.groups > (cl > 8 ? big : d).fit[cl]) --cl;
  while (cl > 8 && p.n_centroids < 160 * cl) --cl;
  while (cl > 4 && p.n_centroids < 96 * cl) --cl;
  // a thread's keys limit the slice: more groups than fit at once take turns
  while (slice_of(p.n_centroids, cl) > Geom<16>::kMaxSlice) ++cl;
  return cl;
}

template <int DT>
int launch_fused_dt(const ri_wave_layer& p, const Layout& L, cudaStream_t s, const ri_wave_gather* gather) {
  Device d, big;
  int rc = ask_device<DT, 8, 8>(&d);
  if (rc != RI_OK || (rc = ask_device<DT, 4, 16>(&big)) != RI_OK) return rc;
  const int cl = cluster_size(p, d, big), keys = keys_of(slice_of(p.n_centroids, cl));
  if (cl > 8) return keys == 4 ? launch<DT, 4, 16>(p, L, cl, s, gather) : launch<DT, 8, 16>(p, L, cl, s, gather);
  switch (keys) {
    case 4: return launch<DT, 4>(p, L, cl, s, gather);
    case 8: return launch<DT, 8>(p, L, cl, s, gather);
    default: return launch<DT, 16>(p, L, cl, s, gather);
  }
}

}  // namespace

bool fused_supported(const ri_wave_layer& p) { return p.n_centroids <= kFusedMaxCentroids; }

// Test hook: cap the estimation entries a CTA keeps in shared memory (0 forces the global lists, a small value the
// mixed case); negative restores the default.  Not part of the decode interface.
extern "C" int ri_wave_test_local_cap(int cap) {
  g_cap_limit = cap;
  return RI_OK;
}

int launch_fused(const ri_wave_layer& p, const Layout& L, cudaStream_t s, const ri_wave_gather* gather) {
  return p.dtype == RI_BF16 ? launch_fused_dt<RI_BF16>(p, L, s, gather) : launch_fused_dt<RI_F16>(p, L, s, gather);
}

int launch_gather_wait(const ri_wave_gather& g, cudaStream_t s) {
  const long long limit_ns = (g.wait_limit_us > 0 ? (long long)g.wait_limit_us : 1000000ll) * 1000ll;
  RI_CUDA_OK(ri_launch_pdl_id(6, gather_signal_wait_kernel, dim3(1), dim3(64), 0, s, g.d_flag_slots, g.d_flags, g.d_epoch,
                              g.d_error, g.n_ranks, limit_ns, g.d_stamps));
  return RI_OK;
}

}  // namespace ri_wave
