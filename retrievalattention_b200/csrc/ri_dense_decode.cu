// Decoding with full attention over a dense head-major cache: the comparator's two steps.
//   ri_dense_append   one token's key and value rows of every request into the cache, at the request's own length;
//   ri_dense_decode   softmax(q.K^T / sqrt(d)).V over the request's valid rows, split over the whole chip.
// (reference: cache_hub/flash_attn_cache.py:133-151, attn_hub/flash_attn.py:17-30)
//
// Bound by the rows of K and V, read once.  The cache's 16-row steps, all groups behind one another (groups without rows
// take none), are cut into one equal contiguous range per SM and that again into one per warp, so uneven requests and
// group counts that do not divide the chip leave no SM idle; a cluster of eight CTAs per group, the earlier split, put 256
// CTAs of equal work on 148 SMs.  A warp streams its steps through its own three-stage ring, filled by TMA: sixteen 16-byte
// cp.async per lane and step, as the gathered rows of ri_wave_attend.cuh need them, held the kernel at 4.8 TB/s whatever
// the split.  It does not stop at a group's end: it stores that group's partial result and goes on.  A CTA whose range
// lies inside one group merges its warps in shared memory first.  A second kernel, its launch hidden behind the first,
// merges a group's partial results by log-sum-exp in a fixed order.
// Four requests of 27768 to 32768 tokens, 8 heads of 4, a layer with its append: 144 -> 91 us, 3.5 -> 5.4 TB/s (the
// append by indexing kernels and the lengths' own kernels were 22 us of it).
//
// A step in shared memory: K, then V, each as two halves of 64 channels x 16 rows in the 128-byte swizzle.  Lane
// (r = lane/4, t = lane%4) reads K row 8jj + s(r) and of V rows t + 4i the 16-byte pieces s(r) and 8 + s(r), where s
// rotates the three bits of r so that the eight lanes of a quarter read eight different bank groups.  Column n
// of the scores is therefore key 8jj + s(n), which makes a lane's two columns keys t and t + 4: the rows of V it holds.
#include <atomic>

#include "ri_tc.cuh"
#include "ri_wave_attend.cuh"

namespace ri_wave {
namespace {

using namespace ri_tc;

constexpr int kDenseWarps = 8;
constexpr int kDenseThreads = kDenseWarps * 32;
constexpr int kDenseMaxCtas = 160;                    // the grid is one CTA per SM, at most this many
constexpr int kDenseRing = kDenseWarps * kStages * kStageBytes;   // 192 KB, on a 1024-byte boundary
constexpr int kDenseSmem = 1024 + kDenseRing;
constexpr int kCombineThreads = 256;

struct DenseArgs {
  const uint4* q;
  const int32_t* valid;      // [batch]; a group attends valid[b] + extra rows, at most `stride`
  float* part_o;             // [slots][gs][128]
  float2* part_ml;           // [slots][gs]: (maximum in the log2 domain, sum)
  uint16_t* out;
  int* error_flag;           // 0, or which wait gave up
  int64_t stride;
  int batch, hk, gs, extra, max_ctas;
  float scale2;
};

__device__ __forceinline__ int rows_of(const DenseArgs& a, int b) {
  return (int)min((int64_t)max(a.valid[b] + a.extra, 0), a.stride);
}
__device__ __forceinline__ int steps_of(int rows) { return (rows + 15) >> 4; }

// All steps of the cache (whole warps).
__device__ __forceinline__ int count_steps(const DenseArgs& a) {
  int sum = 0;
  for (int b = threadIdx.x & 31; b < a.batch; b += 32) sum += steps_of(rows_of(a, b));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  return sum * a.hk;
}
// How many CTAs share `total` steps: at least a step per warp, at most one CTA per SM.
__device__ __forceinline__ int used_ctas(int total, int max_ctas) {
  return min(max_ctas, max(1, (total + kDenseWarps - 1) / kDenseWarps));
}
__device__ __forceinline__ int cta_start(int c, int total, int n) { return (int)((int64_t)c * total / n); }

// A place in the sequence of steps: group g, its first step in the sequence, its rows.
struct Place {
  int g, first, rows;
};
// The group that holds step s (whole warps; s < total).
__device__ __forceinline__ Place find_place(const DenseArgs& a, int s) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int b0 = 0; b0 < a.batch; b0 += 32) {
    const int b = b0 + lane;
    const int rows = b < a.batch ? rows_of(a, b) : 0, n = steps_of(rows) * a.hk;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, s < before + incl);
    if (hit) {
      const int src = __ffs(hit) - 1;
      const int r = __shfl_sync(0xffffffffu, rows, src), start = before + __shfl_sync(0xffffffffu, incl - n, src);
      const int per = steps_of(r), h = (s - start) / per;
      return {(b0 + src) * a.hk + h, start + h * per, r};
    }
    before += __shfl_sync(0xffffffffu, incl, 31);
  }
  return {0, 0, 0};
}
// The next group with rows (there is one: the caller has steps left).
__device__ __forceinline__ void next_place(const DenseArgs& a, Place& p) {
  p.first += steps_of(p.rows);
  ++p.g;
  if (p.g % a.hk == 0) {
    int b = p.g / a.hk;
    while ((p.rows = rows_of(a, b)) == 0 && b + 1 < a.batch) ++b;
    p.g = b * a.hk;
  }
}

template <int DT>
__global__ void __launch_bounds__(kDenseThreads, 1) dense_decode_kernel(const __grid_constant__ CUtensorMap map_k,
                                                                     const __grid_constant__ CUtensorMap map_v, DenseArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t s_full[kDenseWarps][kStages];
  __shared__ int s_abort;
  __shared__ float sm_m[kDenseWarps][kMaxHeads], sm_l[kDenseWarps][kMaxHeads];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = lane >> 2, t = lane & 3, gs = a.gs;
  const int sr = ((r & 1) << 2) | (r >> 1);              // s(r) above
  if (tid == 0) s_abort = 0;
  if (lane == 0) {                                       // a warp's barriers are set up and fed by the same lane
    for (int i = 0; i < kStages; ++i) mbar_init(smem_u32(&s_full[warp][i]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  volatile int* abort_flag = &s_abort;
  ri_pdl_enter();
  const int total = count_steps(a), n_ctas = used_ctas(total, a.max_ctas), c = (int)blockIdx.x;
  if (c >= n_ctas || total == 0) return;
  const int c_lo = cta_start(c, total, n_ctas), c_hi = cta_start(c + 1, total, n_ctas), c_n = c_hi - c_lo;
  const int lo = c_lo + c_n * warp / kDenseWarps, hi = c_lo + c_n * (warp + 1) / kDenseWarps;
  const Place c_first = find_place(a, c_lo);
  const bool merged = c_hi <= c_first.first + steps_of(c_first.rows);      // the CTA's range lies inside one group

  constexpr int kHalfStep = 2048, kStageStride = kDenseWarps * kStageBytes;      // ring: stage-major
  uint8_t* my_ring = ring + warp * kStageBytes;
  const uint32_t my_ring_u32 = smem_u32(my_ring), my_full = smem_u32(&s_full[warp][0]);

  float m_run = -INFINITY, l_run = 0.f;    // head r (l: this lane's share, reduced over the quad at the end)
  float acc[8][4];
  auto clear = [&] {
    m_run = -INFINITY;
    l_run = 0.f;
#pragma unroll
    for (int x = 0; x < 8; ++x)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[x][i] = 0.f;
  };
  auto reduce_sum = [&] {
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
  };
  // accumulators to rows of 128 floats, one per head (heads 2t and 2t+1 are this lane's)
  auto put = [&](float* o) {
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const int ch = (x < 4) ? 8 * sr + 2 * x : 64 + 8 * sr + 2 * (x - 4);
      if (2 * t < gs) *reinterpret_cast<float2*>(o + (2 * t) * RI_HEAD_DIM + ch) = make_float2(acc[x][0], acc[x][2]);
      if (2 * t + 1 < gs) *reinterpret_cast<float2*>(o + (2 * t + 1) * RI_HEAD_DIM + ch) = make_float2(acc[x][1], acc[x][3]);
    }
  };
  // Slots: along the sequence (warp, group) goes up by one of the two at a time, so their sum names a partial result.
  auto store_partial = [&](int g) {
    const int64_t slot = (int64_t)(c * kDenseWarps + warp) + g;
    reduce_sum();
    put(a.part_o + slot * gs * RI_HEAD_DIM);
    if (t == 0 && r < gs) a.part_ml[slot * gs + r] = make_float2(m_run, l_run);
  };

  clear();
  if (lo < hi) {
    Place at_issue = find_place(a, lo), at = at_issue;
    auto issue = [&](int s, int stage) {                 // rows behind the cache's end arrive as zeros
      while (s >= at_issue.first + steps_of(at_issue.rows)) next_place(a, at_issue);
      if (lane == 0) {
        const uint32_t dst = my_ring_u32 + stage * kStageStride, bar = my_full + 8 * stage;
        const int row = (int)((int64_t)at_issue.g * a.stride) + (s - at_issue.first) * 16;
        mbar_arrive_expect_tx(bar, kStageBytes);
        tma_load_3d(dst, &map_k, bar, 0, row, 0);
        tma_load_3d(dst + 2 * kHalfStep, &map_v, bar, 0, row, 0);
      }
    };
    int s_issue = lo;
#pragma unroll
    for (int st = 0; st < kStages; ++st)
      if (s_issue < hi) issue(s_issue++, st);
    uint4 qa[4];
    auto load_q = [&] {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        qa[kk] = r < gs ? ri_ldg16(a.q + ((int64_t)at.g * gs + r) * 16 + t + kk * 4) : make_uint4(0, 0, 0, 0);
    };
    load_q();
    int stage = 0, phase = 0;
    bool ok = true;
#pragma unroll 1
    for (int s = lo; s < hi; ++s) {
      if (s >= at.first + steps_of(at.rows)) {
        store_partial(at.g);
        clear();
        do next_place(a, at);
        while (s >= at.first + steps_of(at.rows));
        load_q();
      }
      const int base = (s - at.first) * 16;
      ok = __all_sync(0xffffffffu, mbar_wait(my_full + 8 * stage, phase, abort_flag, 41));
      if (!ok) break;
      const uint8_t* src = my_ring + stage * kStageStride;
      float s2[2][2];
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        float c1[4] = {0.f, 0.f, 0.f, 0.f}, c2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const uint4 kb = *reinterpret_cast<const uint4*>(src + (kk >> 1) * kHalfStep + (8 * jj + sr) * 128 +
                                                           (((t ^ sr) << 4) ^ ((kk & 1) << 6)));
          Elem<DT>::mma16816(c1, qa[kk].x, 0u, qa[kk].y, 0u, kb.x, kb.y);
          Elem<DT>::mma16816(c2, qa[kk].z, 0u, qa[kk].w, 0u, kb.z, kb.w);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
          s2[jj][e] = base + jj * 8 + t + 4 * e < at.rows ? (c1[e] + c2[e]) * a.scale2 : -INFINITY;
      }
      // online softmax for head r
      float mx = fmaxf(fmaxf(s2[0][0], s2[0][1]), fmaxf(s2[1][0], s2[1][1]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_new = fmaxf(m_run, mx), m_safe = m_new == -INFINITY ? 0.f : m_new;
      const float alpha = exp2f(m_run - m_safe);
      float p[2][2], psum = 0.f;
#pragma unroll
      for (int jj = 0; jj < 2; ++jj)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          p[jj][e] = exp2f(s2[jj][e] - m_safe);
          psum += p[jj][e];
        }
      l_run = l_run * alpha + psum;
      m_run = m_new;
      const float f0 = __shfl_sync(0xffffffffu, alpha, (2 * t) * 4), f1 = __shfl_sync(0xffffffffu, alpha, (2 * t + 1) * 4);
#pragma unroll
      for (int x = 0; x < 8; ++x) { acc[x][0] *= f0; acc[x][1] *= f1; acc[x][2] *= f0; acc[x][3] *= f1; }
      uint4 v[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint8_t* p = src + 2 * kHalfStep + (t + 4 * i) * 128 + (((sr ^ t) << 4) ^ ((i & 1) << 6));
        v[i][0] = *reinterpret_cast<const uint4*>(p);
        v[i][1] = *reinterpret_cast<const uint4*>(p + kHalfStep);
      }
      __syncwarp();
      if (s_issue < hi) issue(s_issue++, stage);      // the stage is in registers: refill it before the products
      if (base + 16 > at.rows) {                      // a group's last step: what lies behind its rows may be anything
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (base + t + 4 * i >= at.rows) v[i][0] = v[i][1] = make_uint4(0, 0, 0, 0);
      }
      pv_step<DT>(acc, v, Elem<DT>::pack2(p[0][0], p[0][1]), Elem<DT>::pack2(p[1][0], p[1][1]));
      if (++stage == kStages) { stage = 0; phase ^= 1; }
    }
    if (!ok) {               // leave a bounded chance to the copies in flight before their memory goes
      if (lane == 0) {
        for (int i = 0; i < kStages; ++i) mbar_wait(my_full + 8 * ((stage + i) % kStages), phase ^ (stage + i >= kStages), abort_flag, 42);
        *a.error_flag = s_abort;
      }
      __syncwarp();
    } else if (!merged) {
      store_partial(at.g);
    }
  }
  if (!merged) return;

  reduce_sum();
  if (t == 0) { sm_m[warp][r] = m_run; sm_l[warp][r] = l_run; }
  auto warp_o = [&](int w) { return reinterpret_cast<float*>(ring + w * kStageBytes); };
  put(warp_o(warp));
  __syncthreads();
  const int64_t slot = (int64_t)c * kDenseWarps + c_first.g;
  for (int idx = tid; idx < gs * RI_HEAD_DIM; idx += kDenseThreads) {
    const int h = idx >> 7;
    float M = -INFINITY, L = 0.f, O = 0.f;
#pragma unroll
    for (int w = 0; w < kDenseWarps; ++w) M = fmaxf(M, sm_m[w][h]);
    const float Ms = M == -INFINITY ? 0.f : M;
#pragma unroll
    for (int w = 0; w < kDenseWarps; ++w) {
      const float f = exp2f(sm_m[w][h] - Ms);
      L += sm_l[w][h] * f;
      O += warp_o(w)[idx] * f;
    }
    a.part_o[slot * gs * RI_HEAD_DIM + idx] = O;
    if ((idx & 127) == 0) a.part_ml[slot * gs + h] = make_float2(M, L);
  }
}

// One head of one group per block: the slots of its partial results in sequence order, then two halves of the block each
// sum every second one.
template <int DT>
__global__ void __launch_bounds__(kCombineThreads) dense_combine_kernel(DenseArgs a) {
  ri_pdl_enter();
  __shared__ int s_slot[kDenseMaxCtas * kDenseWarps];
  __shared__ float s_w[kDenseMaxCtas * kDenseWarps];
  __shared__ float s_red[2], s_o[RI_HEAD_DIM];
  __shared__ int s_n;
  const int tid = threadIdx.x, lane = tid & 31, h = blockIdx.x, g = blockIdx.y, gs = a.gs;
  uint16_t* out = a.out + ((int64_t)g * gs + h) * RI_HEAD_DIM;
  const int b = g / a.hk, n = steps_of(rows_of(a, b));
  if (n == 0) {
    if (tid < RI_HEAD_DIM) out[tid] = 0;
    return;
  }
  if (tid < 32) {
    int before = 0;
    for (int i = lane; i < b; i += 32) before += steps_of(rows_of(a, i));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    const int lo = before * a.hk + (g - b * a.hk) * n, hi = lo + n;
    const int total = count_steps(a), n_ctas = used_ctas(total, a.max_ctas);
    int c0 = (int)((int64_t)lo * n_ctas / total);           // the CTA that holds step lo
    while (c0 > 0 && cta_start(c0, total, n_ctas) > lo) --c0;
    while (cta_start(c0 + 1, total, n_ctas) <= lo) ++c0;
    int count = 0;
    for (int c_base = c0; c_base < n_ctas && cta_start(c_base, total, n_ctas) < hi; c_base += 4) {      // 4 CTAs a warp step
      const int c = c_base + (lane >> 3), w = lane & 7;
      bool mine = false;
      if (c < n_ctas) {
        const int c_lo = cta_start(c, total, n_ctas), c_n = cta_start(c + 1, total, n_ctas) - c_lo;
        if (c_lo >= lo && c_lo + c_n <= hi) {
          mine = w == 0;
        } else {
          const int w_lo = c_lo + c_n * w / kDenseWarps, w_hi = c_lo + c_n * (w + 1) / kDenseWarps;
          mine = max(w_lo, lo) < min(w_hi, hi);
        }
      }
      const unsigned votes = __ballot_sync(0xffffffffu, mine);
      if (mine) s_slot[count + __popc(votes & ((1u << lane) - 1))] = c * kDenseWarps + w + g;
      count += __popc(votes);
    }
    __syncwarp();
    float M = -INFINITY, L = 0.f;
    for (int i = lane; i < count; i += 32) M = fmaxf(M, a.part_ml[(int64_t)s_slot[i] * gs + h].x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    const float Ms = M == -INFINITY ? 0.f : M;
    for (int i = lane; i < count; i += 32) {
      const float2 ml = a.part_ml[(int64_t)s_slot[i] * gs + h];
      const float f = exp2f(ml.x - Ms);
      s_w[i] = f;
      L += ml.y * f;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
    if (lane == 0) { s_red[0] = L; s_n = count; }
  }
  __syncthreads();
  const int ch = tid & (RI_HEAD_DIM - 1), half = tid >> 7, count = s_n;
  float O = 0.f;
#pragma unroll 8
  for (int i = half; i < count; i += 2) O += a.part_o[((int64_t)s_slot[i] * gs + h) * RI_HEAD_DIM + ch] * s_w[i];
  if (half) s_o[ch] = O;
  __syncthreads();
  if (!half) {
    const float L = s_red[0];
    out[ch] = Elem<DT>::bits(L > 0.f ? (O + s_o[ch]) / L : 0.f);
  }
}

__global__ void __launch_bounds__(256) dense_append_kernel(const uint4* __restrict__ k, const uint4* __restrict__ v, uint4* keys,
                                                           uint4* values, const int32_t* __restrict__ valid, int* error_flag,
                                                           int hk, int pieces, int64_t stride) {
  ri_pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;      // one 16-byte piece of K and of V
  if (i >= pieces) return;
  const int g = i >> 4;
  const int64_t row = valid[g / hk];
  if (row < 0 || row >= stride) {      // a replayed graph may come here: the host does not see the lengths
    if ((i & 15) == 0) *error_flag = RI_STATUS_CACHE_FULL;
    return;
  }
  keys[(g * stride + row) * 16 + (i & 15)] = k[i];
  values[(g * stride + row) * 16 + (i & 15)] = v[i];
}

int64_t dense_slots(int64_t groups) { return (int64_t)kDenseMaxCtas * kDenseWarps + groups; }

// Rows of 128 channels as (64 channels, row, half): a box of 16 rows lies in shared memory as two swizzled half tiles.
int make_step_map(CUtensorMap* map, const void* base, int64_t rows, int dtype) {
  EncodeTiledFn enc;
  const int rc = get_encode_fn(&enc);
  if (rc != RI_OK) return rc;
  const cuuint64_t dims[3] = {64, (cuuint64_t)rows, 2}, strides[2] = {256, 128};
  const cuuint32_t box[3] = {64, 16, 2}, estr[3] = {1, 1, 1};
  const CUresult r = enc(map, dtype == RI_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                         const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  RI_REQUIRE(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with code %d", (int)r);
  return RI_OK;
}

template <int DT>
int launch_dense(const DenseArgs& a, const CUtensorMap& map_k, const CUtensorMap& map_v, cudaStream_t s) {
  static std::atomic<bool> known[64];                   // per device; asked for again where it is not remembered
  int dev = 0;
  RI_CUDA_OK(cudaGetDevice(&dev));
  const bool track = dev >= 0 && dev < 64;
  if (!track || !known[dev].load(std::memory_order_relaxed)) {
    RI_CUDA_OK(cudaFuncSetAttribute(dense_decode_kernel<DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDenseSmem));
    if (track) known[dev].store(true, std::memory_order_relaxed);
  }
  RI_CUDA_OK(ri_launch_pdl_id(11, dense_decode_kernel<DT>, dim3(a.max_ctas), dim3(kDenseThreads), (size_t)kDenseSmem, s,
                              map_k, map_v, a));
  RI_CUDA_OK(ri_launch_pdl_id(11, dense_combine_kernel<DT>, dim3(a.gs, a.batch * a.hk), dim3(kCombineThreads), 0, s, a));
  return RI_OK;
}

}  // namespace
}  // namespace ri_wave

extern "C" int64_t ri_dense_decode_scratch_bytes(int32_t batch, int32_t kv_heads, int32_t group_size) {
  if (batch < 1 || kv_heads < 1 || group_size < 1 || group_size > ri_wave::kMaxHeads || (int64_t)batch * kv_heads > 65535)
    return RI_ERR_INVALID;
  return ri_wave::dense_slots((int64_t)batch * kv_heads) * group_size * (RI_HEAD_DIM + 2) * 4;
}

extern "C" int ri_dense_decode(const void* d_q, const void* d_k, const void* d_v, const int32_t* d_valid_length, int32_t extra,
                               void* d_out, void* d_scratch, int32_t* d_error, int32_t batch, int32_t kv_heads, int32_t group_size,
                               int64_t rows_stride, int32_t dtype, void* stream) {
  using namespace ri_wave;
  RI_REQUIRE(d_q && d_k && d_v && d_valid_length && d_out && d_scratch && d_error, "ri_dense_decode: null pointer");
  RI_REQUIRE(batch >= 1 && kv_heads >= 1 && (int64_t)batch * kv_heads <= 65535 && group_size >= 1 && group_size <= kMaxHeads &&
                 rows_stride >= 1 && rows_stride < (1ll << 31) && extra >= 0,
             "ri_dense_decode: bad sizes");
  RI_REQUIRE((int64_t)batch * kv_heads * rows_stride < (1ll << 31) - 16, "ri_dense_decode: too large");
  RI_REQUIRE(dtype == RI_BF16 || dtype == RI_F16, "dtype=%d unsupported", dtype);
  RI_REQUIRE(((uintptr_t)d_q | (uintptr_t)d_k | (uintptr_t)d_v | (uintptr_t)d_scratch) % 16 == 0,
             "q, k, v and the scratch must be 16-byte aligned");
  DenseArgs a = {};
  a.q = static_cast<const uint4*>(d_q);
  a.error_flag = d_error;
  a.valid = d_valid_length;
  a.part_o = static_cast<float*>(d_scratch);
  a.part_ml = reinterpret_cast<float2*>(a.part_o + dense_slots((int64_t)batch * kv_heads) * group_size * RI_HEAD_DIM);
  a.out = static_cast<uint16_t*>(d_out);
  a.stride = rows_stride;
  a.batch = batch; a.hk = kv_heads; a.gs = group_size; a.extra = extra;
  a.scale2 = RI_LOG2E * 0.08838834764831845f;
  int sms = 0, rc;
  if ((rc = ri_sm_count(&sms)) != RI_OK) return rc;
  a.max_ctas = sms < kDenseMaxCtas ? sms : kDenseMaxCtas;
  const int64_t rows = (int64_t)batch * kv_heads * rows_stride;
  CUtensorMap map_k, map_v;
  if ((rc = make_step_map(&map_k, d_k, rows, dtype)) != RI_OK || (rc = make_step_map(&map_v, d_v, rows, dtype)) != RI_OK) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return dtype == RI_BF16 ? launch_dense<RI_BF16>(a, map_k, map_v, s) : launch_dense<RI_F16>(a, map_k, map_v, s);
}

extern "C" int ri_dense_append(const void* d_k, const void* d_v, void* d_keys, void* d_values, const int32_t* d_valid_length,
                               int32_t* d_error, int32_t batch, int32_t kv_heads, int64_t rows_stride, void* stream) {
  RI_REQUIRE(d_k && d_v && d_keys && d_values && d_valid_length && d_error, "ri_dense_append: null pointer");
  RI_REQUIRE(batch >= 1 && kv_heads >= 1 && (int64_t)batch * kv_heads < (1ll << 26) && rows_stride >= 1, "ri_dense_append: bad sizes");
  RI_REQUIRE(((uintptr_t)d_k | (uintptr_t)d_v | (uintptr_t)d_keys | (uintptr_t)d_values) % 16 == 0,
             "ri_dense_append: tensors must be 16-byte aligned");
  const int pieces = batch * kv_heads * 16;
  RI_CUDA_OK(ri_launch_pdl_id(11, ri_wave::dense_append_kernel, dim3((pieces + 255) / 256), dim3(256), 0,
                              static_cast<cudaStream_t>(stream), static_cast<const uint4*>(d_k), static_cast<const uint4*>(d_v),
                              static_cast<uint4*>(d_keys), static_cast<uint4*>(d_values), d_valid_length, d_error, kv_heads,
                              pieces, rows_stride));
  return RI_OK;
}
