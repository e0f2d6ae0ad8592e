// HBM-bound support kernels of the MegaMoE layer for sm_100a: input quantiser, route ordering, pool plan and
// placement, top-k combine.  All integer work here is deterministic (no order-dependent atomics), so the dispatch
// layout is reproducible run to run.
#include <stddef.h>
#include <stdlib.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include <cuda_fp4.h>

#include "mmoe_common.cuh"

namespace mmoe {

// ---------------------------------------------------------------------------------------------------------------------
// Host side of the chained (programmatic dependent) launches.  MMOE_DISABLE_CHAINED_LAUNCH=1 in the environment turns
// the attribute off for the whole process (every launch then waits for the full completion of its predecessor).
// ---------------------------------------------------------------------------------------------------------------------
namespace {
thread_local bool g_chain_scope = false;   // inside a ChainScope(true) of this thread
bool chaining_enabled() {
  static const bool on = [] {
    const char* v = getenv("MMOE_DISABLE_CHAINED_LAUNCH");
    return !(v != nullptr && v[0] != '\0' && v[0] != '0');
  }();
  return on;
}
}  // namespace

ChainScope::ChainScope(bool on) : saved_(g_chain_scope) { g_chain_scope = on && chaining_enabled(); }
ChainScope::~ChainScope() { g_chain_scope = saved_; }

bool chained() { return g_chain_scope; }

// =====================================================================================================================
// Kernel (a): BF16 -> MXFP8 E4M3 with one UE8M0 scale per 32 elements, four scale bytes per int32 word.
// Follows the reference quantiser (backend/staging.py:36-82): scale = 2^ceil(log2(max(amax, 1e-4) / 448)), exponent
// clamped to [1, 254]; values multiplied by the exact reciprocal and rounded to nearest even.
// A warp takes segments of 128 vectors of 8 elements: four independent 16-byte loads per lane, 4 lanes share a scale, 16 a
// scale word.  HBM-bound: 3840 x 5120 (60 MB) took 30 us with one division per vector and single-value conversions.
// =====================================================================================================================
constexpr int kStageSegVec = 128;

__device__ __forceinline__ void stage_vector(const uint4& raw, uint2* __restrict__ q_out, uint32_t* word_out) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
  float v[8];
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = __bfloat1622float2(p[j]);
    v[2 * j] = f.x;
    v[2 * j + 1] = f.y;
    amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
  }
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  amax = fmaxf(amax, 1e-4f);
  // ceil(log2(amax / 448)), 448 = 1.75 * 2^8: the exponent of amax, one more if its mantissa exceeds 1.75 (the carry of the
  // addition), less 8.  An infinite amax gets the largest exponent.
  const uint32_t bits = __float_as_uint(amax);
  const int e = bits == 0x7F800000u ? 254 : static_cast<int>((bits + (0x7FFFFFu - (0x60u << 16))) >> 23) - 8;
  const float inv = __uint_as_float(e == 254 ? 0x00400000u : static_cast<uint32_t>(254 - e) << 23);   // exactly 2^(127 - e)
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    w[j] = __nv_cvt_float2_to_fp8x2(make_float2(__fmul_rn(v[2 * j], inv), __fmul_rn(v[2 * j + 1], inv)), __NV_SATFINITE, __NV_E4M3);
  *q_out = make_uint2(w[0] | (w[1] << 16), w[2] | (w[3] << 16));
  // the four exponents of a 16-lane group, one per byte, in every lane of the group
  uint32_t word = static_cast<uint32_t>(e) << (8 * ((threadIdx.x >> 2) & 3));
  word |= __shfl_xor_sync(0xffffffffu, word, 4);
  word |= __shfl_xor_sync(0xffffffffu, word, 8);
  *word_out = word;
}

// Router in front of the quantiser (one warp per token): the k largest gate logits (ties: the lower expert id), weights =
// softmax over the selected logits, and -- when a replica table is given -- the physical copy `(token + slot) % copies`
// of every selected logical expert, which is the choice a serving engine makes before it calls the layer.
struct RouterArgs {
  const float* logits;           // [m, num_logical] or NULL: ids / weights are given and only repacked
  int num_logical;
  const int32_t* replica_count;  // [num_logical] or NULL: logical id == physical id
  const int32_t* replica_slots;  // [num_logical, max_copies]
  int max_copies;
};

__device__ void route_token(const RouterArgs& r, int64_t t, int k, bool is_pad, int64_t* __restrict__ ids_out,
                            float* __restrict__ w_out) {
  const int lane = threadIdx.x & 31;
  const float* row = r.logits + t * r.num_logical;
  uint64_t taken = 0;                               // bit j: this lane's element lane + 32 j has been selected
  float best_val = 0.f, sum = 0.f;
  float my_val = 0.f;                               // lane s < k keeps the s-th selection
  int my_idx = -1;
  for (int s = 0; s < k; ++s) {
    float v = -INFINITY;
    int idx = 0x7fffffff;
    for (int e = lane, j = 0; e < r.num_logical; e += 32, ++j) {
      const float x = row[e];
      if (!((taken >> j) & 1ull) && (x > v || (x == v && e < idx))) { v = x; idx = e; }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, v, d);
      const int oi = __shfl_xor_sync(0xffffffffu, idx, d);
      if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    if ((idx & 31) == lane && idx < r.num_logical) taken |= 1ull << (idx >> 5);
    if (s == 0) best_val = v;
    const float ex = expf(v - best_val);
    sum += ex;
    if (lane == s) { my_val = ex; my_idx = idx; }
  }
  if (lane < k) {
    int64_t id = my_idx;
    if (r.replica_count != nullptr && my_idx >= 0 && my_idx < r.num_logical) {
      const int copies = max(1, r.replica_count[my_idx]);
      id = r.replica_slots[(int64_t)my_idx * r.max_copies + static_cast<int>((t + lane) % copies)];
    }
    ids_out[t * k + lane] = is_pad ? -1 : id;
    w_out[t * k + lane] = is_pad ? 0.f : __fdiv_rn(my_val, sum);
  }
}

// Four blocks to an SM (53 registers): with five (48) the blocks of the placement behind it start so early that they crowd some SMs, 1021 tokens
// skewed 481 -> 488 us.
__global__ void __launch_bounds__(256, 1) stage_kernel(
    const uint4* __restrict__ hidden, uint2* __restrict__ x_q, int32_t* __restrict__ x_sf,
    int32_t* __restrict__ shared_sf, int64_t shared_rows, int shared_bm,
    const void* __restrict__ ids_in, int ids64, const float* __restrict__ w_in, const uint8_t* __restrict__ pad,
    int64_t* __restrict__ ids_out, float* __restrict__ w_out, int m, int h, int k, RouterArgs router) {
  chain_begin();
  const int vec_per_row = h / 8, words = h / kTileK;
  const uint32_t segs = (vec_per_row + kStageSegVec - 1) / kStageSegVec, total = m * segs;
  const int lane = threadIdx.x & 31;
  const uint32_t stride = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
  for (uint32_t seg = tid >> 5; seg < total; seg += stride >> 5) {
    const int t = static_cast<int>(seg / segs);
    const int v0 = static_cast<int>(seg - t * segs) * kStageSegVec + lane;
    const uint4* row = hidden + (int64_t)t * vec_per_row;
    uint4 raw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) raw[u] = v0 + 32 * u < vec_per_row ? __ldcs(row + v0 + 32 * u) : make_uint4(0, 0, 0, 0);
    // row of token t in the BLOCK_M-dependent shared-expert scale layout (backend/staging.py:85-95)
    const int mm = shared_bm > 0 ? t % shared_bm : 0;
    const int64_t shared_row = shared_bm > 0 ? (int64_t)(t / shared_bm) * ((shared_bm + 127) / 128 * 128) + (mm / 128) * 128 + (mm % 32) * 4 + (mm % 128) / 32 : 0;
#pragma unroll 1          // a third of the code, which lies in DRAM when a call begins: one token 38.7 -> 38.4 us, 2 to 3840 tokens the same
    for (int v = v0; v < v0 + 128 && v < vec_per_row; v += 32) {      // rows are whole multiples of 32 vectors: a warp is in or out together
      uint2 q;
      uint32_t word;
      stage_vector(raw[0], &q, &word);
#pragma unroll
      for (int u = 0; u < 3; ++u) raw[u] = raw[u + 1];
      x_q[(int64_t)t * vec_per_row + v] = q;
      if ((lane & 15) == 0) {
        x_sf[(int64_t)t * words + v / 16] = static_cast<int32_t>(word);
        if (shared_bm > 0) shared_sf[(int64_t)(v / 16) * shared_rows + shared_row] = static_cast<int32_t>(word);
      }
    }
  }
  if (router.logits != nullptr) {
    for (int t = tid >> 5; t < m; t += stride >> 5) route_token(router, t, k, pad != nullptr && pad[t] != 0, ids_out, w_out);
    return;
  }
  // routing repack (backend/staging.py:244-251)
  const uint32_t routes = m * k;
  for (uint32_t r = tid; r < routes; r += stride) {
    const bool is_pad = pad != nullptr && pad[r / k] != 0;
    const int64_t id = ids64 ? static_cast<const int64_t*>(ids_in)[r] : static_cast<const int32_t*>(ids_in)[r];
    ids_out[r] = is_pad ? -1 : id;
    w_out[r] = is_pad ? 0.f : w_in[r];
  }
}

cudaError_t launch_stage(const Ctx& c, const void* hidden, const void* ids, int ids64, const float* w,
                         const uint8_t* pad, int m, int shared_bm, cudaStream_t s) {
  return launch_route_stage(c, hidden, ids, ids64, w, nullptr, 0, nullptr, nullptr, 0, pad, m, shared_bm, s);
}

cudaError_t launch_route_stage(const Ctx& c, const void* hidden, const void* ids, int ids64, const float* w,
                               const float* logits, int num_logical, const int32_t* replica_count,
                               const int32_t* replica_slots, int max_copies, const uint8_t* pad, int m, int shared_bm,
                               cudaStream_t s) {
  if (m == 0) return cudaSuccess;
  const int h = c.geo.hidden;
  const int64_t segs = (int64_t)m * ((h / 8 + kStageSegVec - 1) / kStageSegVec);      // one warp each
  int blocks = static_cast<int>(std::min<int64_t>((segs + 7) / 8, 148 * 8));
  if (blocks < 1) blocks = 1;
  const RouterArgs router{logits, num_logical, replica_count, replica_slots, max_copies};
  return launch_chained(stage_kernel, dim3(blocks), dim3(256), 0, s, static_cast<const uint4*>(hidden),
      c.at<uint2>(c.lay.x), c.at<int32_t>(c.lay.x_sf), c.at<int32_t>(c.lay.shared_x_sf), c.lay.shared_sf_rows, c.geo.num_shared_experts > 0 ? shared_bm : 0, ids, ids64, w,
      pad, c.at<int64_t>(c.lay.topk_idx), c.at<float>(c.lay.topk_weights), m, h, c.geo.num_topk, router);
}

// =====================================================================================================================
// NVFP4 activation staging: BF16 -> packed E2M1 with one E4M3 scale per 16 elements and a per-tensor FP32 scale (the
// two-level NVFP4 recipe).  The serving engine's hook names such a staging call next to the MXFP8 one
// (patches/vllm-megamoe-plugin.patch:10, `prepare_megamoe_nvfp4_inputs`); the reference plugin itself never implements
// it.  Per block of 16:  s = e4m3_rn(amax * global_scale / 6);  q_i = e2m1_rn(x_i * global_scale / s)  (0 when s == 0);
// x is recovered as q * s / global_scale.  Low nibble = even K, as in the MXFP4 weights.  One thread owns a block (two
// 16-byte loads, one 8-byte store, one scale byte).
// =====================================================================================================================
__global__ void __launch_bounds__(256) stage_nvfp4_kernel(const uint4* __restrict__ hidden, uint2* __restrict__ q_out,
                                                          uint8_t* __restrict__ sf_out, float global_scale, int64_t blocks16) {
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < blocks16; b += (int64_t)gridDim.x * blockDim.x) {
    const uint4 raw[2] = {hidden[2 * b], hidden[2 * b + 1]};
    float v[16];
    float amax = 0.f;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw[u]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(p[j]);
        v[8 * u + 2 * j] = f.x;
        v[8 * u + 2 * j + 1] = f.y;
        amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
      }
    }
    const float s = fminf(__fdiv_rn(__fmul_rn(amax, global_scale), 6.0f), 448.0f);
    const uint8_t s8 = float_to_e4m3(s);
    const float sf = e4m3_to_float(s8);
    const float inv = sf != 0.f ? __fdiv_rn(global_scale, sf) : 0.f;
    uint32_t w[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t byte = __nv_cvt_float2_to_fp4x2(make_float2(__fmul_rn(v[2 * j], inv), __fmul_rn(v[2 * j + 1], inv)), __NV_E2M1,
                                                     cudaRoundNearest);
      w[j >> 2] |= (byte & 0xFFu) << (8 * (j & 3));
    }
    q_out[b] = make_uint2(w[0], w[1]);
    sf_out[b] = s8;
  }
}

cudaError_t launch_stage_nvfp4(const void* hidden, void* q_out, void* sf_out, float global_scale, int64_t num_tokens, int hidden_size,
                               cudaStream_t s) {
  const int64_t blocks16 = num_tokens * hidden_size / 16;
  if (blocks16 == 0) return cudaSuccess;
  const int grid = static_cast<int>(std::min<int64_t>((blocks16 + 255) / 256, 148 * 16));
  return launch_plain(stage_nvfp4_kernel, dim3(grid), dim3(256), 0, s, static_cast<const uint4*>(hidden), static_cast<uint2*>(q_out),
                      static_cast<uint8_t*>(sf_out), global_scale, blocks16);
}

// =====================================================================================================================
// Route ordering: a stable counting sort of the routes (token*k + slot) by destination expert in three passes over
// chunks of 128 tokens.  Replaces the atomics-ordered slot assignment of the reference (backend/kernel/dispatch.py:
// 348-410) with a deterministic order; the per-expert counts are the same numbers.
// =====================================================================================================================
// ---------------------------------------------------------------------------------------------------------------------
// small block-level building blocks of the route ordering and the plan
// ---------------------------------------------------------------------------------------------------------------------
// Exclusive prefix sum of `in[0..n)` into `out[0..n]` (out[n] = total), n <= 1024, whole block (>= 32 threads, a
// multiple of 32) participates; `in` and `out` may not alias.  Ends with a barrier.
__device__ void block_exclusive_scan(const int32_t* in, int32_t* out, int n) {
  __shared__ int32_t warp_tot[33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  __syncthreads();
  int carry = 0;
  for (int base = 0; base < n; base += blockDim.x) {
    const int i = base + threadIdx.x;
    int v = i < n ? in[i] : 0;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += t;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      int w = lane < nwarps ? warp_tot[lane] : 0;
      int wi = w;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, wi, d);
        if (lane >= d) wi += t;
      }
      warp_tot[lane] = wi - w;                 // exclusive offset of each warp
      if (lane == 31) warp_tot[32] = wi;       // block total of this round
    }
    __syncthreads();
    if (i < n) out[i] = carry + warp_tot[warp] + incl - v;
    carry += warp_tot[32];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = carry;
  __syncthreads();
}

// Stable rank of every route among the routes of the same expert, by ONE warp walking the routes in order, 32 at a
// time: lanes with the same expert find each other with match.any, the lowest such lane owns the running counter.
// `ids[i]` (-1 = masked) in shared memory, `count[e]` zeroed shared counters; writes rank[i] (or -1).
__device__ void warp_rank_routes(const int32_t* ids, int n, int32_t* count, int32_t* rank) {
  const int lane = threadIdx.x & 31;
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    const int e = i < n ? ids[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, e);
    int r = -1;
    if (e >= 0) {
      const int before = __popc(peers & ((1u << lane) - 1u));
      const int start = count[e];
      r = start + before;
    }
    __syncwarp();
    if (e >= 0 && (peers & ((1u << lane) - 1u)) == 0u) count[e] += __popc(peers);   // lowest lane of each expert group
    __syncwarp();
    if (i < n) rank[i] = r;
  }
}

constexpr int kSortThreads = 256;

// pass A: per chunk, local rank of every route among the chunk's routes to the same expert + per-chunk expert counts
__global__ void __launch_bounds__(kSortThreads) sort_local_kernel(
    const int64_t* __restrict__ topk_idx, int32_t* __restrict__ route_pos, int32_t* __restrict__ chunk_count,
    int32_t* __restrict__ status, int m, int k, int num_experts) {
  chain_begin();
  extern __shared__ int32_t sm[];
  int32_t* ids = sm;                                // [chunk routes]
  int32_t* hist = sm + kSortChunkTokens * k;        // [num_experts]
  const int chunk = blockIdx.x;
  const int r0 = chunk * kSortChunkTokens * k;
  const int n = min(kSortChunkTokens * k, m * k - r0);
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x) hist[e] = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    int64_t id = topk_idx[r0 + i];
    if (id >= num_experts) { if (status != nullptr) report_bad_index(status); id = -1; }
    ids[i] = id < 0 ? -1 : static_cast<int32_t>(id);
  }
  __syncthreads();
  if (threadIdx.x < 32) warp_rank_routes(ids, n, hist, route_pos + r0);
  __syncthreads();
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x) chunk_count[(int64_t)chunk * num_experts + e] = hist[e];
}

// pass B: one block; per expert an exclusive scan over chunks, then an exclusive scan over experts
__global__ void __launch_bounds__(1024) sort_scan_kernel(
    int32_t* __restrict__ chunk_count, int32_t* __restrict__ send_count, int32_t* __restrict__ send_offset,
    int32_t* __restrict__ recv_count_if_single, int num_chunks, int num_experts) {
  chain_begin();
  __shared__ int32_t totals[2048 + 1];
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x) {
    int run = 0;
    for (int c = 0; c < num_chunks; ++c) {
      const int v = chunk_count[(int64_t)c * num_experts + e];
      chunk_count[(int64_t)c * num_experts + e] = run;
      run += v;
    }
    totals[e] = run;
    send_count[e] = run;
    if (recv_count_if_single != nullptr) recv_count_if_single[e] = run;
  }
  __shared__ int32_t offs[2048 + 1];
  block_exclusive_scan(totals, offs, num_experts);
  for (int e = threadIdx.x; e <= num_experts; e += blockDim.x) send_offset[e] = offs[e];
}

// pass C: final position of every route, and the inverse map
__global__ void __launch_bounds__(kSortThreads) sort_place_kernel(
    const int64_t* __restrict__ topk_idx, const int32_t* __restrict__ chunk_base,
    const int32_t* __restrict__ send_offset, int32_t* __restrict__ route_pos, int32_t* __restrict__ sorted_route,
    int m, int k, int num_experts) {
  chain_begin();
  const int64_t total = (int64_t)m * k;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < total; r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t id = topk_idx[r];
    int pos = -1;
    if (id >= 0 && id < num_experts) {
      const int chunk = static_cast<int>(r / (kSortChunkTokens * k));
      pos = send_offset[id] + chunk_base[(int64_t)chunk * num_experts + id] + route_pos[r];
      sorted_route[pos] = static_cast<int32_t>(r);
    }
    route_pos[r] = pos;
  }
}

cudaError_t launch_count_sort(const Ctx& c, int m, cudaStream_t s) {
  const int k = c.geo.num_topk, e = c.geo.num_experts;
  const int chunks = max(1, (m + kSortChunkTokens - 1) / kSortChunkTokens);
  int32_t* chunk_count = c.at<int32_t>(c.lay.sort_scratch);
  const size_t smem = (size_t)(kSortChunkTokens * k + e) * sizeof(int32_t);
  cudaError_t err = launch_chained(sort_local_kernel, dim3(chunks), dim3(kSortThreads), smem, s, c.at<int64_t>(c.lay.topk_idx),
                                   c.at<int32_t>(c.lay.route_pos), chunk_count, c.at<int32_t>(c.lay.status), m, k, e);
  if (err == cudaSuccess)
    err = launch_chained(sort_scan_kernel, dim3(1), dim3(1024), 0, s, chunk_count, c.at<int32_t>(c.lay.send_count), c.at<int32_t>(c.lay.send_offset),
                         c.geo.num_ranks == 1 ? c.at<int32_t>(c.lay.recv_count) : nullptr, chunks, e);
  if (err == cudaSuccess && m > 0) {
    const int blocks = static_cast<int>(std::min<int64_t>(((int64_t)m * k + kSortThreads - 1) / kSortThreads, 148 * 8));
    err = launch_chained(sort_place_kernel, dim3(blocks), dim3(kSortThreads), 0, s, c.at<int64_t>(c.lay.topk_idx), chunk_count,
                         c.at<int32_t>(c.lay.send_offset), c.at<int32_t>(c.lay.route_pos), c.at<int32_t>(c.lay.sorted_route), m, k, e);
  }
  return err;
}

// ---------------------------------------------------------------------------------------------------------------------
// Route ordering without any allocation.  The per-chunk expert counts, the only scratch the three passes need, live in
// a file-scope device array: every GPU that loads this library holds these 64 KB until the process exits.  Host code
// may only use the array's *address*, obtained once per device with cudaGetSymbolAddress while that device is current
// (the bare symbol name is a host-side stand-in, not a device pointer).
// ---------------------------------------------------------------------------------------------------------------------
constexpr int kStaticMaxTokens = 4096;                                   // 32 chunks of 128 tokens
constexpr int kStaticMaxExperts = 512;
constexpr int kStaticScratchInts = (kStaticMaxTokens / kSortChunkTokens) * kStaticMaxExperts;
static __device__ __align__(256) int32_t g_route_order_scratch[kStaticScratchInts];

namespace {
constexpr int kMaxDevices = 64;
// Written by the first call on a device; every writer stores the same address, so the only requirement is that the
// store and the loads are not torn or reordered: relaxed atomics.
std::atomic<int32_t*> g_scratch_ptr[kMaxDevices] = {};
}

cudaError_t route_order_static(const int64_t* topk_idx, int m, int k, int num_experts, int32_t* send_count,
                               int32_t* send_offset, int32_t* route_pos, int32_t* sorted_route, cudaStream_t s) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  int32_t* chunk_count = g_scratch_ptr[dev].load(std::memory_order_relaxed);
  if (chunk_count == nullptr) {                  // set-up: first call on this device
    // Resolving the symbol may load the module, which a capturing stream forbids: refuse instead of breaking the capture.
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    e = cudaStreamIsCapturing(s, &capturing);
    if (e != cudaSuccess) return e;
    if (capturing != cudaStreamCaptureStatusNone) return cudaErrorStreamCaptureUnsupported;
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_route_order_scratch);
    if (e != cudaSuccess) return e;
    chunk_count = static_cast<int32_t*>(ptr);
    g_scratch_ptr[dev].store(chunk_count, std::memory_order_relaxed);
  }
  // nothing in the scratch has to start at zero: pass A overwrites every (chunk, expert) cell that passes B and C read
  const int chunks = std::max(1, (m + kSortChunkTokens - 1) / kSortChunkTokens);
  const size_t smem = (size_t)(kSortChunkTokens * k + num_experts) * sizeof(int32_t);
  e = launch_plain(sort_local_kernel, dim3(chunks), dim3(kSortThreads), smem, s, topk_idx, route_pos, chunk_count, nullptr, m, k, num_experts);
  if (e == cudaSuccess) e = launch_plain(sort_scan_kernel, dim3(1), dim3(1024), 0, s, chunk_count, send_count, send_offset, nullptr, chunks, num_experts);
  if (e == cudaSuccess && m > 0) {
    const int blocks = static_cast<int>(std::min<int64_t>(((int64_t)m * k + kSortThreads - 1) / kSortThreads, 148 * 8));
    e = launch_plain(sort_place_kernel, dim3(blocks), dim3(kSortThreads), 0, s, topk_idx, chunk_count, send_offset, route_pos, sorted_route, m, k,
                     num_experts);
  }
  return e;
}

int route_order_static_max_tokens() { return kStaticMaxTokens; }
int route_order_static_max_experts() { return kStaticMaxExperts; }

// =====================================================================================================================
// EP > 1: gather the rows, scale words and weights of this rank's routes into send order (sorted by destination
// expert, hence by destination rank), ready for the all-to-allv.
// =====================================================================================================================
__global__ void __launch_bounds__(256) pack_kernel(
    const uint4* __restrict__ x, const int32_t* __restrict__ x_sf, const float* __restrict__ topk_w,
    const int32_t* __restrict__ sorted_route, const int32_t* __restrict__ send_offset, uint4* __restrict__ send_x,
    int32_t* __restrict__ send_sf, float* __restrict__ send_w, int h, int k, int num_experts) {
  const int total = send_offset[num_experts];
  const int vec = h / 16, words = h / kTileK;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int p = warp; p < total; p += nwarps) {
    const int route = sorted_route[p];
    const int t = route / k;
    for (int v = lane; v < vec; v += 32) send_x[(int64_t)p * vec + v] = x[(int64_t)t * vec + v];
    for (int w = lane; w < words; w += 32) send_sf[(int64_t)p * words + w] = x_sf[(int64_t)t * words + w];
    if (lane == 0) send_w[p] = topk_w[route];
  }
}

cudaError_t launch_pack(const Ctx& c, int m, cudaStream_t s) {
  if (m == 0) return cudaSuccess;
  return launch_plain(pack_kernel, dim3(148 * 4), dim3(256), 0, s, c.at<uint4>(c.lay.x), c.at<int32_t>(c.lay.x_sf), c.at<float>(c.lay.topk_weights),
                      c.at<int32_t>(c.lay.sorted_route), c.at<int32_t>(c.lay.send_offset), c.at<uint4>(c.lay.send_x),
                      c.at<int32_t>(c.lay.send_sf), c.at<float>(c.lay.send_w), c.geo.hidden, c.geo.num_topk, c.geo.num_experts);
}

// =====================================================================================================================
// Pool plan.  Pool order: local experts ascending, each expert starting on a BLOCK_M boundary
// (backend/kernel/dispatch.py:431-447); inside an expert, source ranks ascending and each source's routes in its send
// order (token, slot) -- a fixed order where the reference's is arrival order.
// =====================================================================================================================
struct PlanArgs {
  int e_local, num_ranks, block_m, pair_above, m, has_shared, shared_above, shared_cap;
};

// Exclusive prefix of one value pair per thread over the block (a multiple of 32 threads, at most 1024), with the totals.
struct ScanPair {
  uint64_t a;      // pool blocks | weights-as-A tiles << 21 | pair tiles << 42
  int32_t b;       // rows
};
__device__ ScanPair block_scan_pair(ScanPair v, ScanPair* total) {
  __shared__ uint64_t warp_a[33];
  __shared__ int32_t warp_b[33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  uint64_t a = v.a;
  int32_t b = v.b;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint64_t ta = __shfl_up_sync(0xffffffffu, a, d);
    const int32_t tb = __shfl_up_sync(0xffffffffu, b, d);
    if (lane >= d) { a += ta; b += tb; }
  }
  __syncthreads();                                   // an earlier scan's totals have been read
  if (lane == 31) { warp_a[warp] = a; warp_b[warp] = b; }
  __syncthreads();
  if (warp == 0) {
    const uint64_t wa = lane < nwarps ? warp_a[lane] : 0;
    const int32_t wb = lane < nwarps ? warp_b[lane] : 0;
    uint64_t sa = wa;
    int32_t sb = wb;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t ta = __shfl_up_sync(0xffffffffu, sa, d);
      const int32_t tb = __shfl_up_sync(0xffffffffu, sb, d);
      if (lane >= d) { sa += ta; sb += tb; }
    }
    warp_a[lane] = sa - wa;
    warp_b[lane] = sb - wb;
    if (lane == 31) { warp_a[32] = sa; warp_b[32] = sb; }
  }
  __syncthreads();
  *total = ScanPair{warp_a[32], warp_b[32]};
  return ScanPair{warp_a[warp] + a - v.a, warp_b[warp] + b - v.b};
}

// The tiles of one expert (or of the shared expert) behind `out`.
__device__ void emit_tiles(Tile* out, int expert, int row_base, int n, Cut cut, int chunk0) {
  for (int j = 0; j < cut.parts; ++j) {
    const int rows = max(0, min(cut.step, n - j * cut.step));
    out[j] = Tile{expert, rows > 0 ? row_base + j * cut.step : row_base, rows, rows > 0 ? chunk0 + j : chunk0, j, cut.parts, {0, 0}};
  }
}

// What the placement of an expert's rows needs, thread e holding expert e.
struct ExpertPlan {
  int block_off;     // first pool block
  int row_off;       // rows of the experts before it
  Cut cut;
};

// Builds the plan from the rows `n` of every expert, thread e holding expert e (0 past the last; e_local <= blockDim.x): tile
// table, offsets and header, written by the blocks that pass `write`.  The whole block takes part.
__device__ ExpertPlan build_plan(const PlanView& pv, int n, const PlanArgs& a, bool write) {
  const int e = threadIdx.x;
  __shared__ int s_rows, s_tiles;
  if (threadIdx.x == 0) {
    s_rows = 16;
    s_tiles = 0;
  }
  // With pair tiles in the call or rows from other ranks, weights-as-A tiles of 112 rows (four stages fit the shared memory) only
  // when enough experts gain a tile by it, else of 80 (five stages).
  const bool may_be_small = n > 0 && !on_pairs(n, a.pair_above, kSmallTileRows);
  const bool wide = may_be_small && ((n > kDeepTileRows && n <= kSmallTileRows) || n > 2 * kDeepTileRows);
  const int num_small = __syncthreads_count(may_be_small), num_wide = __syncthreads_count(wide);
  const bool no_pairs = a.pair_above == kNeverPair && a.num_ranks == 1;
  int cap = no_pairs ? small_only_cap(a.m, a.block_m, a.e_local) : (num_wide * 8 > num_small ? kSmallTileRows : kDeepTileRows);
  if (no_pairs && cap == kSixStageRows) {
    const int tiles = __reduce_add_sync(0xffffffffu, cut_rows(n, false, kSixStageRows).parts << 16 | cut_rows(n, false, kDeepTileRows).parts);
    if ((threadIdx.x & 31) == 0 && tiles != 0) atomicAdd(&s_tiles, tiles);
    __syncthreads();
    if (wide_tiles(s_tiles >> 16, s_tiles & 0xFFFF)) cap = kDeepTileRows;
  }
  const bool small = n > 0 && !on_pairs(n, a.pair_above, cap);
  const Cut cut = cut_rows(n, n > 0 && !small, cap);
  Cut sh_cut = shared_cut(a.has_shared ? a.m : 0, a.shared_above, a.shared_cap);
  const bool shared_small = a.m <= a.shared_above;
  const int blocks = (n + a.block_m - 1) / a.block_m;
  ScanPair total;
  const ScanPair at = block_scan_pair(
      ScanPair{static_cast<uint64_t>(blocks) | (static_cast<uint64_t>(small ? cut.parts : 0) << 21) |
                   (static_cast<uint64_t>(small ? 0 : cut.parts) << 42), n}, &total);
  const int block_off = static_cast<int>(at.a & 0x1FFFFF);
  const int small_total = static_cast<int>((total.a >> 21) & 0x1FFFFF), pair_total = static_cast<int>(total.a >> 42);
  if (write) {
    const int rows = small ? cut.step : 0;
    const int warp_rows = __reduce_max_sync(0xffffffffu, rows);
    if ((threadIdx.x & 31) == 0 && warp_rows > 0) atomicMax(&s_rows, warp_rows);
    const int first_tile = small ? static_cast<int>((at.a >> 21) & 0x1FFFFF) : small_total + static_cast<int>(at.a >> 42);
    if (e < a.e_local) {
      pv.expert_total[e] = n;
      pv.expert_block_off[e] = block_off;
      pv.expert_tile_off[e] = first_tile;
      emit_tiles(pv.tiles + first_tile, e, block_off * a.block_m, n, cut, block_off * chunks_per_block(a.block_m));
    }
    __syncthreads();
    // Behind pair launches the shared expert's cut is taken from the plan: where the routed tiles have larger slots anyway, its
    // tiles are as large (256 tokens of 384 experts, skewed, 234 -> 228 us; even 1077, 1104 with tiles of 80 rows in any case).
    if (shared_small && !no_pairs && a.num_ranks == 1 && s_rows > a.shared_cap) sh_cut = shared_cut(a.has_shared ? a.m : 0, a.shared_above, kDeepTileRows);
    if (threadIdx.x == 0) {
      PlanHeader& h = *pv.hdr;
      h.num_routed_tiles = small_total + pair_total;
      h.num_shared_tiles = sh_cut.parts;
      h.num_pool_blocks = static_cast<int>(total.a & 0x1FFFFF);
      h.total_recv = total.b;
      h.block_m = a.block_m;
      h.num_tokens = a.m;
      h.num_small_tiles = small_total;
      h.small_cap = cap;
      h.small_rows = max(s_rows, shared_small && a.has_shared ? sh_cut.step : 16);
      h.shared_step = sh_cut.step;
      h.shared_pairs = a.has_shared && !shared_small ? 1 : 0;
      pv.expert_block_off[a.e_local] = h.num_pool_blocks;
      pv.expert_tile_off[a.e_local] = h.num_routed_tiles;
    }
    const SharedTiles shared{sh_cut.parts, sh_cut.step, a.m};
    for (int j = threadIdx.x; j < sh_cut.parts; j += blockDim.x) pv.tiles[small_total + pair_total + j] = shared.at(j);
  }
  return ExpertPlan{block_off, at.b, cut};
}

// Scale words of the call's own tokens in the chunks of the shared expert's tiles (chunk j = tile j), whole warps: a warp takes
// one word of all rows of a tile, so that its 128 words leave as one line (positions 4 (i % 32) + i / 32, see chunk_pos).  A warp
// per token, which scattered the token's 40 words over as many lines, eight tokens one after the other, took 8-16 us of the
// counting launch.
struct SharedScales {
  const int32_t* x_sf;
  int32_t* out;          // nullptr: no shared expert
  int64_t rows;
  Cut cut;
};
__device__ void place_shared_scales(const SharedScales& s, int m, int words, int warp, int warps) {
  const int lane = threadIdx.x & 31;
  for (int task = warp; task < s.cut.parts * words; task += warps) {
    const int j = task / words, w = task - j * words;
    int32_t v[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int i = lane + 32 * a, t = j * s.cut.step + i;
      v[a] = i < s.cut.step && t < m ? s.x_sf[(int64_t)t * words + w] : 0;
    }
    *reinterpret_cast<int4*>(s.out + w * s.rows + (int64_t)j * kChunkRows + 4 * lane) = make_int4(v[0], v[1], v[2], v[3]);
  }
}

// The shared expert's tiles depend only on the token count: with its scale chunks written it can run before the routed
// experts' receive counts are known.
__global__ void __launch_bounds__(256) shared_plan_kernel(int m, SharedScales scales, int words) {
  chain_begin();
  place_shared_scales(scales, m, words, static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5), static_cast<int>((gridDim.x * blockDim.x) >> 5));
}

// General plan (any number of source ranks), one block: rows per expert from the receive counts, and for every (expert,
// source) segment where it starts in the pool and in receive order.
constexpr int kPlanThreads = 512;      // one thread per local expert
__global__ void __launch_bounds__(kPlanThreads) plan_kernel(char* __restrict__ plan_base, const int32_t* __restrict__ recv_count,
                                                            int32_t* __restrict__ stats, PlanArgs a) {
  chain_begin();
  PlanView pv = plan_view(plan_base, a.e_local, a.num_ranks);
  const int e = threadIdx.x;
  int n = 0;
  if (e < a.e_local)
    for (int r = 0; r < a.num_ranks; ++r) n += recv_count[r * a.e_local + e];
  if (stats != nullptr && e < a.e_local) stats[e] += n;      // cumulative per-expert receive statistics (dispatch.py:644-650)
  const ExpertPlan ep = build_plan(pv, n, a, true);
  int rank_off = 0, pool_row = ep.block_off * a.block_m;
  for (int r = 0; r < a.num_ranks; ++r) {
    const int c = e < a.e_local ? recv_count[r * a.e_local + e] : 0;
    ScanPair total;
    const ScanPair at = block_scan_pair(ScanPair{0, c}, &total);
    if (e < a.e_local) {
      pv.seg_recv_start[e * a.num_ranks + r] = rank_off + at.b;
      pv.seg_pool_start[e * a.num_ranks + r] = pool_row;
    }
    if (e == 0) pv.rank_off[r] = rank_off;
    rank_off += total.b;
    pool_row += c;
  }
  if (e == 0) pv.rank_off[a.num_ranks] = rank_off;
}

// =====================================================================================================================
// One GPU: route ordering, plan and placement without the detour over receive counts.  Same results as
// sort_local/scan/place + plan_kernel + place_kernel (tested against them).
// =====================================================================================================================
constexpr int kRouteThreads = 512;     // one thread per expert in the plan, 16 warps that rank routes
constexpr int kRouteWarps = kRouteThreads / 32;

// Stable rank of up to kSmallRoutes routes (or kSortChunkTokens * k) among the routes of the same expert, by the whole block: every warp ranks
// a run of its own against its own counters (lanes with the same expert find each other with match.any), then each
// expert's counters are summed over the warps.  ids[i] (0xFFFF = masked) -> rank[i]; returns thread e's expert total.
// (One warp walking all routes took 10 us for 768; 16 warps take 2.)
__device__ int block_rank_routes(const uint16_t* ids, int n, uint16_t* rank, uint16_t* warp_count, int num_experts) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < kRouteWarps * num_experts; i += kRouteThreads) warp_count[i] = 0;
  __syncthreads();                                   // ids are in place too
  const int run = ((n + kRouteWarps - 1) / kRouteWarps + 31) & ~31;
  uint16_t* mine = warp_count + warp * num_experts;
  const int end = min(n, (warp + 1) * run);
  for (int base = warp * run; base < end; base += 32) {
    const int i = base + lane;
    const int e = i < end ? ids[i] : 0xFFFF;
    const unsigned peers = __match_any_sync(0xffffffffu, e);
    const int before = __popc(peers & ((1u << lane) - 1u));
    const int start = e != 0xFFFF ? mine[e] : 0;
    __syncwarp();
    if (e != 0xFFFF && before == 0) mine[e] = static_cast<uint16_t>(start + __popc(peers));
    __syncwarp();
    if (i < end) rank[i] = static_cast<uint16_t>(start + before);
  }
  __syncthreads();
  int total = 0;
  if ((int)threadIdx.x < num_experts)
#pragma unroll
    for (int w = 0; w < kRouteWarps; ++w) {
      const int c = warp_count[w * num_experts + threadIdx.x];
      warp_count[w * num_experts + threadIdx.x] = static_cast<uint16_t>(total);
      total += c;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kRouteThreads)
    if (ids[i] != 0xFFFF) rank[i] = static_cast<uint16_t>(rank[i] + warp_count[(i / run) * num_experts + ids[i]]);
  __syncthreads();
  return total;
}

struct RouteArgs {
  const int64_t* topk_idx;
  int32_t* route_pos;
  int32_t* sorted_route;
  int32_t* send_count;
  int32_t* send_offset;
  int32_t* recv_count;
  int32_t* chunk_count;      // [chunks][E]
  int32_t* stats;
  int32_t* status;
  char* plan;
  const uint4* x;
  const int32_t* x_sf;
  const float* w;
  uint4* pool_x;
  int32_t* pool_sf;
  float* pool_w;
  int32_t* pool_dst;
  int64_t pool_sf_rows;
  SharedScales shared;
  int h, k;
  PlanArgs a;
};

// everything of the plan that is the same for every caller with one source rank
__device__ void write_single_rank_plan(const RouteArgs& r, const PlanView& pv, int n, const ExpertPlan& ep) {
  const int e = threadIdx.x;
  if (e < r.a.e_local) {
    r.send_count[e] = n;
    r.recv_count[e] = n;
    r.send_offset[e] = ep.row_off;
    pv.seg_pool_start[e] = ep.block_off * r.a.block_m;
    pv.seg_recv_start[e] = ep.row_off;
    if (r.stats != nullptr) r.stats[e] += n;         // cumulative per-expert receive statistics (dispatch.py:644-650)
    if (e == r.a.e_local - 1) {
      r.send_offset[r.a.e_local] = ep.row_off + n;
      pv.rank_off[0] = 0;
      pv.rank_off[1] = ep.row_off + n;
    }
  }
}

// Calls of at most kSmallRoutes routes: ONE launch.  Every block ranks the routes and builds the plan for itself in shared memory
// (2-3 us, less than a second launch behind a grid-wide hand-over), block 0 writes it out, and the others place the
// routes, one warp per route (block 0 with its share of them came in 0.5-1 us late).  The shared expert's scales are not placed: its GEMM1 gathers them itself.
// The ranking and the plan are a chain of barriers in code that lies in DRAM.  Walking it once on masked routes in front of the wait saved 0 to 1 us
// of calls in a row (128 tokens of 32 experts 132.1 -> 131.7, 32 tokens 113.3 -> 112.8) and cost 1 to 2 where the staging had ended
// already, as it has in every call that finds the GPU idle (142.3 -> 143.6 from event to event, 131.0 -> 132.2).
__global__ void __launch_bounds__(kRouteThreads) route_small_kernel(const RouteArgs r) {
  chain_wait();
  chain_release();       // in this order: the GEMM1 launch starts knowing that the staging has completed
  extern __shared__ int32_t sm[];
  const int E = r.a.e_local, n = r.a.m * r.k, n_even = (n + 1) & ~1;
  int32_t* s_block = sm;                             // [E] first pool block
  int32_t* s_off = s_block + E;                      // [E] send offset
  int32_t* s_step = s_off + E;                       // [E] rows per tile
  uint16_t* ids = reinterpret_cast<uint16_t*>(s_step + E);
  uint16_t* rank = ids + n_even;
  uint16_t* warp_count = rank + n_even;              // [16][E]
  for (int i = threadIdx.x; i < n; i += kRouteThreads) {
    int64_t id = r.topk_idx[i];
    if (id >= E) { if (blockIdx.x == 0) report_bad_index(r.status); id = -1; }
    ids[i] = id < 0 ? 0xFFFF : static_cast<uint16_t>(id);
  }
  const int total = block_rank_routes(ids, n, rank, warp_count, E);
  const PlanView pv = plan_view(r.plan, E, 1);
  const ExpertPlan ep = build_plan(pv, total, r.a, blockIdx.x == 0);
  if ((int)threadIdx.x < E) {
    s_block[threadIdx.x] = ep.block_off;
    s_off[threadIdx.x] = ep.row_off;
    s_step[threadIdx.x] = ep.cut.step;
  }
  if (blockIdx.x == 0) {
    write_single_rank_plan(r, pv, total, ep);
    return;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warps = (gridDim.x - 1) * kRouteWarps;
  const int vec = r.h / 16, words = r.h / kTileK, cpb = chunks_per_block(r.a.block_m);
  for (int i = (blockIdx.x - 1) * kRouteWarps + (threadIdx.x >> 5); i < n; i += warps) {
    const int e = ids[i];
    if (e == 0xFFFF) {
      if (lane == 0) r.route_pos[i] = -1;
      continue;
    }
    const int j = rank[i], t = i / r.k;
    const int p = s_block[e] * r.a.block_m + j, part = j / s_step[e];
    const uint4* src = r.x + (int64_t)t * vec;
    uint4* dst = r.pool_x + (int64_t)p * vec;
    for (int v0 = lane; v0 < vec; v0 += 128) {
      uint4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (v0 + 32 * u < vec) q[u] = src[v0 + 32 * u];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (v0 + 32 * u < vec) dst[v0 + 32 * u] = q[u];
    }
    const int64_t pos = (int64_t)(s_block[e] * cpb + part) * kChunkRows + chunk_pos(j - part * s_step[e]);
    for (int wd = lane; wd < words; wd += 32) r.pool_sf[wd * r.pool_sf_rows + pos] = r.x_sf[(int64_t)t * words + wd];
    if (lane == 0) {
      r.pool_w[p] = r.w[i];
      r.pool_dst[p] = s_off[e] + j;
      r.route_pos[i] = s_off[e] + j;
      r.sorted_route[s_off[e] + j] = i;
    }
  }
}

// Larger calls, and those whose shared expert runs on CTA pairs, first of two launches: one block per 128 tokens ranks its routes; the last block to finish sums the chunks
// and builds the plan.  Further blocks place the shared expert's scales, which GEMM1 starts with while the next launch still places.
__host__ __device__ inline int route_chunks(int m) { return m > kSortChunkTokens ? (m + kSortChunkTokens - 1) / kSortChunkTokens : 1; }

// Three blocks per SM, for 40 registers: its blocks start beside the staging's last ones (with 64, 3840 tokens of 48 experts 956 -> 960 us).
__global__ void __launch_bounds__(kRouteThreads, 3) route_count_kernel(const RouteArgs r) {
  chain_begin();
  extern __shared__ int32_t sm[];
  const int chunks = route_chunks(r.a.m);
  if ((int)blockIdx.x >= chunks) {
    place_shared_scales(r.shared, r.a.m, r.h / kTileK, (blockIdx.x - chunks) * kRouteWarps + (threadIdx.x >> 5), (gridDim.x - chunks) * kRouteWarps);
    return;
  }
  const int E = r.a.e_local, r0 = blockIdx.x * kSortChunkTokens * r.k;
  const int n = max(0, min(kSortChunkTokens * r.k, r.a.m * r.k - r0)), n_even = (kSortChunkTokens * r.k + 1) & ~1;
  uint16_t* ids = reinterpret_cast<uint16_t*>(sm);
  uint16_t* rank = ids + n_even;
  uint16_t* warp_count = rank + n_even;
  for (int i = threadIdx.x; i < n; i += kRouteThreads) {
    int64_t id = r.topk_idx[r0 + i];
    if (id >= E) { report_bad_index(r.status); id = -1; }
    ids[i] = id < 0 ? 0xFFFF : static_cast<uint16_t>(id);
  }
  int total = block_rank_routes(ids, n, rank, warp_count, E);
  for (int i = threadIdx.x; i < n; i += kRouteThreads) r.route_pos[r0 + i] = ids[i] == 0xFFFF ? -1 : rank[i];
  const int e = threadIdx.x;
  if (e < E) r.chunk_count[(int64_t)blockIdx.x * E + e] = total;
  const PlanView pv = plan_view(r.plan, E, 1);
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&pv.hdr->ticket, 1) == chunks - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x == 0) pv.hdr->ticket = 0;
  total = 0;
  if (e < E)
    for (int c0 = 0; c0 < chunks; c0 += 8) {         // eight independent loads in flight
      int v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = c0 + u < chunks ? __ldcg(&r.chunk_count[(int64_t)(c0 + u) * E + e]) : 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (c0 + u < chunks) r.chunk_count[(int64_t)(c0 + u) * E + e] = total;
        total += v[u];
      }
    }
  const ExpertPlan ep = build_plan(pv, total, r.a, true);
  write_single_rank_plan(r, pv, total, ep);
}

// Second launch: one warp per token.  The token's FP8 row is read once and stored to the pool rows of all its routes; lane s
// works out where route s goes.
__global__ void __launch_bounds__(256) route_place_kernel(const RouteArgs r) {
  chain_wait();
  chain_release();       // in this order: the GEMM1 launch starts knowing that staging, counting and plan have completed
  const PlanView pv = plan_view(r.plan, r.a.e_local, 1);
  const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
  const int vec = r.h / 16, words = r.h / kTileK, cpb = chunks_per_block(r.a.block_m);
  const int cap = pv.hdr->small_cap;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < r.a.m; t += warps) {
    int row = -1, sf_pos = 0;                          // lane s: pool row and scale position of route s
    if (lane < r.k) {
      const int i = t * r.k + lane;
      const int64_t id = r.topk_idx[i];
      int pos = -1;
      if (id >= 0 && id < r.a.e_local) {
        const int e = static_cast<int>(id);
        const int j = r.chunk_count[(int64_t)(t / kSortChunkTokens) * r.a.e_local + e] + r.route_pos[i];
        const int block = pv.expert_block_off[e];
        const int total = pv.expert_total[e];
        const Cut cut = cut_rows(total, on_pairs(total, r.a.pair_above, cap), cap);
        const int part = j / cut.step;
        pos = r.send_offset[e] + j;
        row = block * r.a.block_m + j;
        sf_pos = (block * cpb + part) * kChunkRows + chunk_pos(j - part * cut.step);
        r.sorted_route[pos] = i;
        r.pool_w[row] = r.w[i];
        r.pool_dst[row] = pos;
      }
      r.route_pos[i] = pos;
    }
    const uint4* src = r.x + (int64_t)t * vec;
    for (int base = 0; base < vec; base += 160) {
      const int v0 = base + lane;
      uint4 q[5];
#pragma unroll
      for (int u = 0; u < 5; ++u)
        if (v0 + 32 * u < vec) q[u] = src[v0 + 32 * u];
      for (int s = 0; s < r.k; ++s) {
        const int p = __shfl_sync(0xffffffffu, row, s);
        if (p < 0) continue;
        uint4* dst = r.pool_x + (int64_t)p * vec;
#pragma unroll
        for (int u = 0; u < 5; ++u)
          if (v0 + 32 * u < vec) dst[v0 + 32 * u] = q[u];
      }
    }
    for (int w0 = 0; w0 < words; w0 += 32) {
      const int wd = w0 + lane;
      const int32_t v = wd < words ? r.x_sf[(int64_t)t * words + wd] : 0;
      for (int s = 0; s < r.k; ++s) {
        const int p = __shfl_sync(0xffffffffu, row, s), pos = __shfl_sync(0xffffffffu, sf_pos, s);
        if (p >= 0 && wd < words) r.pool_sf[wd * r.pool_sf_rows + pos] = v;
      }
    }
  }
}

// Place: one warp per pool row of every routed tile: copy the FP8 row, scatter its scale words into the chunk layout,
// record the top-k weight and the receive-order row that takes the expert output.  A block takes 32 rows of a tile at a
// time (a tile has at most 4 such slices), so the grid stays busy whatever the number of tiles, and every lane keeps
// four 16-byte loads in flight.
__global__ void __launch_bounds__(256) place_kernel(
    char* __restrict__ plan_base, const uint4* __restrict__ src_x, const int32_t* __restrict__ src_sf,
    const float* __restrict__ src_w, const int32_t* __restrict__ sorted_route, uint4* __restrict__ pool_x,
    int32_t* __restrict__ pool_sf, float* __restrict__ pool_w, int32_t* __restrict__ pool_dst, int64_t pool_sf_rows,
    int e_local, int num_ranks, int h, int k, int direct, SharedScales shared) {
  chain_begin();
  PlanView pv = plan_view(plan_base, e_local, num_ranks);
  const int ntiles = pv.hdr->num_routed_tiles;
  const int block_m = pv.hdr->block_m;
  const int vec = h / 16, words = h / kTileK;
  const int warp_in_block = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  if (shared.out != nullptr) {
    const int m = pv.hdr->num_tokens;
    place_shared_scales(shared, m, words, blockIdx.x * warps + warp_in_block, gridDim.x * warps);
  }
  constexpr int kSlices = kPairTileRows / 32;
  for (int task = blockIdx.x; task < ntiles * kSlices; task += gridDim.x) {
    const int slice = task / ntiles, t = task - slice * ntiles;   // slice-major: the first slices are the populated ones
    const Tile tile = pv.tiles[t];
    const int i_end = min(tile.n_valid, 32 * slice + 32);
    if (32 * slice >= i_end) continue;
    const int e = tile.expert;
    const int expert_row0 = pv.expert_block_off[e] * block_m;
    for (int i = 32 * slice + warp_in_block; i < i_end; i += warps) {
      const int p = tile.row0 + i;
      const int j = p - expert_row0;           // index of this row among the expert's routes
      int r = 0, acc = 0;
      for (; r < num_ranks - 1; ++r) {          // source rank that owns the j-th route
        const int next = pv.seg_pool_start[e * num_ranks + r + 1] - expert_row0;
        if (j < next) break;
      }
      acc = pv.seg_pool_start[e * num_ranks + r] - expert_row0;
      const int recv_row = pv.seg_recv_start[e * num_ranks + r] + (j - acc);
      int64_t src_row = recv_row;
      float w;
      if (direct) {                              // EP1: read the staged inputs in place
        const int route = sorted_route[recv_row];
        src_row = route / k;
        w = src_w[route];
      } else {
        w = src_w[recv_row];
      }
      const uint4* src = src_x + src_row * vec;
      uint4* dst = pool_x + (int64_t)p * vec;
      for (int v0 = lane; v0 < vec; v0 += 128) {
        uint4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (v0 + 32 * u < vec) q[u] = src[v0 + 32 * u];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (v0 + 32 * u < vec) dst[v0 + 32 * u] = q[u];
      }
      const int pos = tile.sf_chunk * kChunkRows + chunk_pos(i);
      for (int wd = lane; wd < words; wd += 32) pool_sf[(int64_t)wd * pool_sf_rows + pos] = src_sf[src_row * words + wd];
      if (lane == 0) {
        pool_w[p] = w;
        pool_dst[p] = recv_row;
      }
    }
  }
}

namespace {
PlanArgs plan_args(const Ctx& c, int m, int block_m) {
  return PlanArgs{c.e_local, c.geo.num_ranks, block_m, c.pair_above_for(m), m, c.geo.num_shared_experts > 0 && m > 0 ? 1 : 0,
                  c.shared_above_for(m), c.shared_cap_for(m, block_m)};
}

// (on the weights-as-A kernels GEMM1 gathers them itself)
SharedScales shared_scales(const Ctx& c, int m, int pair_above) {
  const bool on = c.geo.num_shared_experts > 0 && m > pair_above;
  return SharedScales{c.at<int32_t>(c.lay.x_sf), on ? c.at<int32_t>(c.lay.shared_tile_sf) : nullptr, shared_chunk_rows(c.geo.num_max_tokens),
                      shared_cut(m, pair_above, kDeepTileRows)};
}

RouteArgs route_args(const Ctx& c, int m, int block_m, int32_t* stats) {
  RouteArgs r{};
  r.topk_idx = c.at<int64_t>(c.lay.topk_idx);
  r.route_pos = c.at<int32_t>(c.lay.route_pos);
  r.sorted_route = c.at<int32_t>(c.lay.sorted_route);
  r.send_count = c.at<int32_t>(c.lay.send_count);
  r.send_offset = c.at<int32_t>(c.lay.send_offset);
  r.recv_count = c.at<int32_t>(c.lay.recv_count);
  r.chunk_count = c.at<int32_t>(c.lay.sort_scratch);
  r.stats = stats;
  r.status = c.at<int32_t>(c.lay.status);
  r.plan = c.ws + c.lay.plan;
  r.x = c.at<uint4>(c.lay.x);
  r.x_sf = c.at<int32_t>(c.lay.x_sf);
  r.w = c.at<float>(c.lay.topk_weights);
  r.pool_x = c.at<uint4>(c.lay.pool_x);
  r.pool_sf = c.at<int32_t>(c.lay.pool_sf);
  r.pool_w = c.at<float>(c.lay.pool_w);
  r.pool_dst = c.at<int32_t>(c.lay.pool_dst);
  r.pool_sf_rows = c.lay.pool_sf_rows;
  r.shared = shared_scales(c, m, c.shared_above_for(m));
  r.h = c.geo.hidden;
  r.k = c.geo.num_topk;
  r.a = plan_args(c, m, block_m);
  return r;
}
}  // namespace

cudaError_t launch_route_small(const Ctx& c, int m, int block_m, int32_t* stats, cudaStream_t s) {
  const int n = m * c.geo.num_topk, e = c.geo.num_experts;
  const size_t smem = (size_t)3 * e * 4 + (size_t)2 * ((n + 1) & ~1) * 2 + (size_t)kRouteWarps * e * 2;
  return launch_chained(route_small_kernel, dim3(1 + std::min((n + kRouteWarps - 1) / kRouteWarps, 147)), dim3(kRouteThreads), smem, s,
                        route_args(c, m, block_m, stats));
}

cudaError_t launch_route_large(const Ctx& c, int m, int block_m, int32_t* stats, cudaStream_t s) {
  const RouteArgs r = route_args(c, m, block_m, stats);
  const int chunks = route_chunks(m);
  const int scale_blocks = r.shared.out == nullptr ? 0 : std::min((r.shared.cut.parts * (r.h / kTileK) + kRouteWarps - 1) / kRouteWarps, 148);
  const size_t smem = (size_t)2 * ((kSortChunkTokens * r.k + 1) & ~1) * 2 + (size_t)kRouteWarps * r.a.e_local * 2;
  cudaError_t e = launch_chained(route_count_kernel, dim3(chunks + scale_blocks), dim3(kRouteThreads), smem, s, r);
  if (e == cudaSuccess && m > 0) e = launch_chained(route_place_kernel, dim3(std::min((m + 7) / 8, 148 * 8)), dim3(256), 0, s, r);
  return e;
}

cudaError_t launch_shared_plan(const Ctx& c, int m, cudaStream_t s) {
  if (m <= c.pair_above || c.geo.num_shared_experts == 0) return cudaSuccess;
  return launch_chained(shared_plan_kernel, dim3(std::max(1, std::min((m + 7) / 8, 148 * 2))), dim3(256), 0, s, m, shared_scales(c, m, c.pair_above),
                        c.geo.hidden / kTileK);
}

cudaError_t launch_plan_place(const Ctx& c, int m, int block_m, int32_t* stats, cudaStream_t s) {
  const int R = c.geo.num_ranks;
  cudaError_t e = launch_chained(plan_kernel, dim3(1), dim3(kPlanThreads), 0, s, c.ws + c.lay.plan, c.at<int32_t>(c.lay.recv_count), stats,
                                 plan_args(c, m, block_m));
  if (e != cudaSuccess) return e;
  const bool direct = R == 1;
  return launch_chained(place_kernel, dim3(148 * 8), dim3(256), 0, s, c.ws + c.lay.plan, direct ? c.at<uint4>(c.lay.x) : c.at<uint4>(c.lay.recv_x),
      direct ? c.at<int32_t>(c.lay.x_sf) : c.at<int32_t>(c.lay.recv_sf),
      direct ? c.at<float>(c.lay.topk_weights) : c.at<float>(c.lay.recv_w), c.at<int32_t>(c.lay.sorted_route),
      c.at<uint4>(c.lay.pool_x), c.at<int32_t>(c.lay.pool_sf), c.at<float>(c.lay.pool_w), c.at<int32_t>(c.lay.pool_dst),
      c.lay.pool_sf_rows, c.e_local, R, c.geo.hidden, c.geo.num_topk, direct ? 1 : 0, shared_scales(c, m, c.shared_above_for(m)));
}

// =====================================================================================================================
// Combine: y[t] = bf16_rn(sum of the token's valid slots in ascending slot order, shared expert last), sequential FP32
// additions starting from zero (backend/kernel/combine.py:128-199).  One thread owns 8 consecutive output elements.
// =====================================================================================================================
__device__ __forceinline__ void add_bf16x8(float (&acc)[8], const uint4& v) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = __bfloat1622float2(p[j]);
    acc[2 * j] = __fadd_rn(acc[2 * j], f.x);
    acc[2 * j + 1] = __fadd_rn(acc[2 * j + 1], f.y);
  }
}

// The counters of a launch of both GEMMs, by a block more: in the call's last kernel nothing waits for that.  No block lets
// the next launch start before they are zero, so that the next such launch may claim its tasks at once.  True for that block.
__device__ __forceinline__ bool combine_zeroes(char* plan_base, int e_local) {
  if (plan_base == nullptr || blockIdx.x != gridDim.x - 1) {
    chain_release();
    return false;
  }
  const PlanView pv = plan_view(plan_base, e_local, 1);
  if (threadIdx.x == 0) {
    pv.hdr->routed = 0;
    pv.hdr->next_task = 0;
    pv.hdr->layer1_done = 0;
  }
  for (int e = threadIdx.x; e < e_local + 4; e += blockDim.x) pv.done[e] = 0;      // and `pair_tasks`, `pairs_open` behind it
  __threadfence();
  __syncthreads();
  chain_release();
  return true;
}

// What the serving engine's separate BF16 addition leaves: the layer output rounded to BF16 first, then the sum of the two BF16 values
// rounded once more.
__device__ __forceinline__ __nv_bfloat162 add_residual(__nv_bfloat162 o, __nv_bfloat162 r) {
  const float2 a = __bfloat1622float2(o), b = __bfloat1622float2(r);
  return __floats2bfloat162_rn(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}

// Calls of at most kNarrowTokens tokens, where latency and code on its way from DRAM are all there is to wait for: two outputs per
// thread, a quarter of the instructions.  Wide and narrow: 1 token 38.1 and 38.4 us, 2 54.0 and 53.4, 4 84.3 and 84.4, 8 149.0 and 148.7, 16 of 32
// experts 102.7 and 102.4; past the line 17 108.2 and 107.9, 48 118.1 and 117.5, 64 119.9 and 119.6, 128 130.9 and 130.5, within 0.5 us of
// each other: little hangs on where it lies.
constexpr int kNarrowTokens = 16;
__global__ void __launch_bounds__(256) combine_narrow_kernel(
    const uint32_t* __restrict__ rows, const int32_t* __restrict__ route_pos, const uint32_t* __restrict__ shared_out,
    const uint32_t* __restrict__ residual, uint32_t* __restrict__ y, int m, int h, int k, char* plan_base, int e_local) {
  chain_wait();
  if (combine_zeroes(plan_base, e_local)) return;
  const uint32_t pairs = h / 2, i = blockIdx.x * blockDim.x + threadIdx.x, t = i / pairs;
  if (t >= static_cast<uint32_t>(m)) return;
  const uint32_t sh = shared_out != nullptr ? shared_out[i] : 0u, res = residual != nullptr ? residual[i] : 0u;
  const int32_t* pos = route_pos + t * k;
  const uint32_t* col = rows + (i - t * pairs);
  float lo = 0.f, hi = 0.f;
  auto add = [&](uint32_t v) {
    lo = __fadd_rn(lo, __uint_as_float(v << 16));
    hi = __fadd_rn(hi, __uint_as_float(v & 0xFFFF0000u));
  };
#pragma unroll 1
  for (int s0 = 0; s0 < k; s0 += 8) {
    int p[8];
    uint32_t q[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) p[s] = s0 + s < k ? pos[s0 + s] : -1;
#pragma unroll
    for (int s = 0; s < 8; ++s) q[s] = p[s] >= 0 ? col[(int64_t)p[s] * pairs] : 0u;
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (p[s] >= 0) add(q[s]);
  }
  if (shared_out != nullptr) add(sh);
  __nv_bfloat162 out = __floats2bfloat162_rn(lo, hi);
  if (residual != nullptr) out = add_residual(out, *reinterpret_cast<const __nv_bfloat162*>(&res));
  y[i] = *reinterpret_cast<const uint32_t*>(&out);
}

// A warp takes 64 vectors of 8 outputs of one token; a lane has the rows of up to eight slots of its two vectors in flight at
// once (with one dependent load after the other 3840 x 5120 top-6, 315 MB, took 63 us).
constexpr int kCombineSegVec = 64;
__global__ void __launch_bounds__(256) combine_kernel(
    const uint4* __restrict__ rows, const int32_t* __restrict__ route_pos, const uint4* __restrict__ shared_out,
    const uint4* __restrict__ residual, uint4* __restrict__ y, int m, int h, int k, char* plan_base, int e_local) {
  chain_wait();
  if (combine_zeroes(plan_base, e_local)) return;
  const int blocks = plan_base != nullptr ? gridDim.x - 1 : gridDim.x;
  const int vec = h / 8, lane = threadIdx.x & 31;
  const uint32_t segs = (vec + kCombineSegVec - 1) / kCombineSegVec, total = m * segs, warps = (blocks * blockDim.x) >> 5;
  for (uint32_t seg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; seg < total; seg += warps) {
    const int t = static_cast<int>(seg / segs);
    const int v0 = static_cast<int>(seg - t * segs) * kCombineSegVec + lane;
    const bool both = v0 + 32 < vec;                 // rows are whole multiples of 32 vectors
    const int my_pos = lane < k ? route_pos[(int64_t)t * k + lane] : -1;
    const int64_t i = (int64_t)t * vec + v0;
    uint4 sh[2], res[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      sh[u] = res[u] = make_uint4(0, 0, 0, 0);
      if (u == 0 || both) {
        if (shared_out != nullptr) sh[u] = __ldcs(shared_out + i + 32 * u);
        if (residual != nullptr) res[u] = residual[i + 32 * u];
      }
    }
    float acc[2][8] = {};
    for (int s0 = 0; s0 < k; s0 += 8) {
      uint4 q[8][2];
      bool valid[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const int pos = __shfl_sync(0xffffffffu, my_pos, (s0 + s) & 31);
        valid[s] = s0 + s < k && pos >= 0;           // warp-uniform
        if (valid[s]) {
          const uint4* row = rows + (int64_t)pos * vec + v0;
          q[s][0] = __ldcs(row);
          if (both) q[s][1] = __ldcs(row + 32);
        }
      }
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (valid[s]) {
          add_bf16x8(acc[0], q[s][0]);
          if (both) add_bf16x8(acc[1], q[s][1]);
        }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (u == 1 && !both) break;
      if (shared_out != nullptr) add_bf16x8(acc[u], sh[u]);
      uint4 out;
      __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = __floats2bfloat162_rn(acc[u][2 * j], acc[u][2 * j + 1]);
      if (residual != nullptr) {
        const __nv_bfloat162* r = reinterpret_cast<const __nv_bfloat162*>(&res[u]);
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = add_residual(o[j], r[j]);
      }
      y[i + 32 * u] = out;
    }
  }
}

cudaError_t launch_combine(const Ctx& c, void* y, const void* residual, int m, cudaStream_t s) {
  if (m == 0) return cudaSuccess;
  const int h = c.geo.hidden;
  const bool one_rank = c.geo.num_ranks == 1;
  const void* rows = c.ws + (one_rank ? c.lay.ret : c.lay.ret_recv);
  const void* shared = c.geo.num_shared_experts > 0 ? c.ws + c.lay.shared_out : nullptr;
  char* plan = one_rank ? c.ws + c.lay.plan : nullptr;
  auto launch = [&](auto kernel, auto* out, int64_t blocks) {
    using T = std::remove_pointer_t<decltype(out)>;
    return launch_chained(kernel, dim3(static_cast<unsigned>(blocks) + (one_rank ? 1 : 0)), dim3(256), 0, s, static_cast<const T*>(rows),
                          c.at<int32_t>(c.lay.route_pos), static_cast<const T*>(shared), static_cast<const T*>(residual), out, m, h, c.geo.num_topk,
                          plan, c.e_local);
  };
  if (m <= kNarrowTokens) return launch(combine_narrow_kernel, static_cast<uint32_t*>(y), ((int64_t)m * (h / 2) + 255) / 256);
  const int64_t segs = (int64_t)m * ((h / 8 + kCombineSegVec - 1) / kCombineSegVec);      // one warp each
  return launch(combine_kernel, static_cast<uint4*>(y), std::min<int64_t>((segs + 7) / 8, 148 * 8));
}

cudaError_t zero_counters(const Ctx& c, cudaStream_t s) {
  const PlanView pv = plan_view(c.ws + c.lay.plan, c.e_local, c.geo.num_ranks);
  const size_t first = offsetof(PlanHeader, routed), end = offsetof(PlanHeader, layer1_done) + sizeof pv.hdr->layer1_done;
  cudaError_t e = cudaMemsetAsync(reinterpret_cast<char*>(pv.hdr) + first, 0, end - first, s);      // `claims` lies between, zero already
  if (e == cudaSuccess) e = cudaMemsetAsync(pv.done, 0, (c.e_local + 4) * sizeof *pv.done, s);
  return e;
}

// =====================================================================================================================
// Scalar validation engine (tests only): the same plan, pool, epilogues and output addressing as the tensor-core
// kernels, with the two block-scaled GEMMs written as plain FP32 dot products.  One warp = one 32-channel scale group.
// =====================================================================================================================
template <bool kFp8Weights>
__device__ __forceinline__ float dot_group(const uint8_t* __restrict__ xrow, const uint8_t* __restrict__ wrow) {
  // 32 K elements: xrow -> 32 e4m3 bytes; wrow -> 16 packed bytes (FP4) or 32 e4m3 bytes
  float acc = 0.f;
  if (kFp8Weights) {
#pragma unroll 8
    for (int j = 0; j < 32; ++j) acc = fmaf(e4m3_to_float(xrow[j]), e4m3_to_float(wrow[j]), acc);
  } else {
#pragma unroll 8
    for (int j = 0; j < 16; ++j) {
      const uint32_t b = wrow[j];
      acc = fmaf(e4m3_to_float(xrow[2 * j]), e2m1_to_float(b & 15u), acc);
      acc = fmaf(e4m3_to_float(xrow[2 * j + 1]), e2m1_to_float(b >> 4), acc);
    }
  }
  return acc;
}

// scale byte of weight row `row` (within its matrix of n_rows rows), K group g, in the 4x32-transposed MN-major layout
__device__ __forceinline__ uint32_t weight_sf_byte(const int32_t* __restrict__ sf, int n_rows, int row, int g) {
  const int blk = row / 128, in = row % 128;
  const int pos = blk * 128 + chunk_pos(in);
  const uint32_t word = static_cast<uint32_t>(sf[(int64_t)(g / 4) * n_rows + pos]);
  return (word >> (8 * (g % 4))) & 0xFFu;
}

__device__ __forceinline__ uint32_t token_sf_byte(const int32_t* __restrict__ sf, int64_t sf_rows, const Tile& tile,
                                                  int i, int g) {
  const int pos = tile.sf_chunk * kChunkRows + chunk_pos(i);
  const uint32_t word = static_cast<uint32_t>(sf[(int64_t)(g / 4) * sf_rows + pos]);
  return (word >> (8 * (g % 4))) & 0xFFu;
}

// address of weight row `row` (0..rows_per_expert) of expert e, for plain and two-slice weight tensors
__device__ __forceinline__ const uint8_t* weight_row_ptr(const uint8_t* base, int e, int row, int rows_per_expert,
                                                         int64_t row_bytes, int64_t slice_stride) {
  if (slice_stride > 0) {
    const int half = rows_per_expert / 2;
    return base + (row / half) * slice_stride + ((int64_t)e * half + row % half) * row_bytes;
  }
  return base + ((int64_t)e * rows_per_expert + row) * row_bytes;
}

__global__ void __launch_bounds__(128) simt_l1_kernel(
    char* __restrict__ plan_base, int e_local, int num_ranks, int first_tile, int num_tiles_from_hdr_shared,
    const uint8_t* __restrict__ tok_x, const int32_t* __restrict__ tok_sf, int64_t tok_sf_rows,
    const float* __restrict__ tok_w, const uint8_t* __restrict__ w13, const int32_t* __restrict__ w13_sf,
    uint8_t* __restrict__ act_x, uint8_t* __restrict__ act_sf, int64_t act_sf_rows, int h, int inter, float clamp,
    int fast_math, int fp8_weights, int64_t slice_stride) {
  PlanView pv = plan_view(plan_base, e_local, num_ranks);
  const int ntiles = num_tiles_from_hdr_shared ? pv.hdr->num_shared_tiles : pv.hdr->num_routed_tiles;
  const int base = num_tiles_from_hdr_shared ? pv.hdr->num_routed_tiles : 0;
  const int groups = inter / 32;
  const int lane = threadIdx.x & 31;
  const int64_t work = (int64_t)ntiles * groups;
  const int64_t wstride = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t wi = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); wi < work; wi += wstride) {
    const Tile tile = pv.tiles[base + wi / groups];
    const int g_out = static_cast<int>(wi % groups);
    const int c = g_out * 32 + lane;
    const bool shared = tile.expert == kSharedExpert;
    const int e = shared ? 0 : tile.expert;
    const int64_t wrow_bytes = fp8_weights ? h : h / 2;
    // stored W13 rows: [g0..7, u0..7, g8..15, u8..15, ...]
    const int row_g = 16 * (c / 8) + (c % 8), row_u = row_g + 8;
    const uint8_t* wg = weight_row_ptr(w13, e, row_g, 2 * inter, wrow_bytes, slice_stride);
    const uint8_t* wu = weight_row_ptr(w13, e, row_u, 2 * inter, wrow_bytes, slice_stride);
    const int32_t* wsf = w13_sf + (int64_t)e * (h / 128) * 2 * inter;
    for (int i = 0; i < tile.n_valid; ++i) {
      const uint8_t* xr = tok_x + (int64_t)(tile.row0 + i) * h;
      float accg = 0.f, accu = 0.f;
      for (int g = 0; g < h / 32; ++g) {
        // (the shared expert's tokens: the staged scale rows themselves)
        const float sx = ue8m0_to_float(shared ? (static_cast<uint32_t>(tok_sf[(int64_t)(tile.row0 + i) * (h / kTileK) + g / 4]) >> (8 * (g % 4))) & 0xFFu
                                               : token_sf_byte(tok_sf, tok_sf_rows, tile, i, g));
        const float sg = ue8m0_to_float(weight_sf_byte(wsf, 2 * inter, row_g, g));
        const float su = ue8m0_to_float(weight_sf_byte(wsf, 2 * inter, row_u, g));
        float dg, du;
        if (fp8_weights) {
          dg = dot_group<true>(xr + g * 32, wg + g * 32);
          du = dot_group<true>(xr + g * 32, wu + g * 32);
        } else {
          dg = dot_group<false>(xr + g * 32, wg + g * 16);
          du = dot_group<false>(xr + g * 32, wu + g * 16);
        }
        accg = fmaf(dg, sx * sg, accg);
        accu = fmaf(du, sx * su, accu);
      }
      const float wt = shared ? 1.0f : tok_w[tile.row0 + i];
      const float act = swiglu_act(accg, accu, wt, clamp, fast_math != 0);
      const float amax = warp_max_nonneg(fabsf(act));
      const int sf_exp = ue8m0_exp_of_amax(amax);
      act_x[(int64_t)(tile.row0 + i) * inter + c] = float_to_e4m3(__fmul_rn(act, ue8m0_inv(sf_exp)));
      if (lane == 0) {
        const int pos = tile.sf_chunk * kChunkRows + chunk_pos(i);
        act_sf[((int64_t)(g_out / 4) * act_sf_rows + pos) * 4 + (g_out % 4)] = static_cast<uint8_t>(sf_exp);
      }
    }
  }
}

__global__ void __launch_bounds__(128) simt_l2_kernel(
    char* __restrict__ plan_base, int e_local, int num_ranks, int use_shared_tiles,
    const uint8_t* __restrict__ act_x, const int32_t* __restrict__ act_sf, int64_t act_sf_rows,
    const uint8_t* __restrict__ w2, const int32_t* __restrict__ w2_sf, const int32_t* __restrict__ pool_dst,
    __nv_bfloat16* __restrict__ out, int h, int inter, int fp8_weights, int64_t slice_stride) {
  PlanView pv = plan_view(plan_base, e_local, num_ranks);
  const int ntiles = use_shared_tiles ? pv.hdr->num_shared_tiles : pv.hdr->num_routed_tiles;
  const int base = use_shared_tiles ? pv.hdr->num_routed_tiles : 0;
  const int groups = h / 32;
  const int lane = threadIdx.x & 31;
  const int64_t work = (int64_t)ntiles * groups;
  const int64_t wstride = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t wi = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); wi < work; wi += wstride) {
    const Tile tile = pv.tiles[base + wi / groups];
    const int row = static_cast<int>(wi % groups) * 32 + lane;   // output feature
    const bool shared = tile.expert == kSharedExpert;
    const int e = shared ? 0 : tile.expert;
    const int64_t wrow_bytes = fp8_weights ? inter : inter / 2;
    const uint8_t* wr = weight_row_ptr(w2, e, row, h, wrow_bytes, slice_stride);
    const int32_t* wsf = w2_sf + (int64_t)e * (inter / 128) * h;
    for (int i = 0; i < tile.n_valid; ++i) {
      const uint8_t* xr = act_x + (int64_t)(tile.row0 + i) * inter;
      float acc = 0.f;
      for (int g = 0; g < inter / 32; ++g) {
        const float sx = ue8m0_to_float(token_sf_byte(act_sf, act_sf_rows, tile, i, g));
        const float sw = ue8m0_to_float(weight_sf_byte(wsf, h, row, g));
        const float d = fp8_weights ? dot_group<true>(xr + g * 32, wr + g * 32) : dot_group<false>(xr + g * 32, wr + g * 16);
        acc = fmaf(d, sx * sw, acc);
      }
      const int64_t dst = shared ? (tile.row0 + i) : pool_dst[tile.row0 + i];
      out[dst * h + row] = __float2bfloat16_rn(acc);
    }
  }
}

cudaError_t launch_experts_simt(const Ctx& c, const MmoeWeights& w, const MmoeOptions& o, int m, int block_m,
                                cudaStream_t s) {
  const int h = c.geo.hidden, inter = c.geo.intermediate;
  const int blocks = 148 * 8;
  char* plan = c.ws + c.lay.plan;
  const dim3 g(blocks), b(128);
  cudaError_t e = launch_plain(simt_l1_kernel, g, b, 0, s, plan, c.e_local, c.geo.num_ranks, 0, 0, c.at<uint8_t>(c.lay.pool_x),
                               c.at<int32_t>(c.lay.pool_sf), c.lay.pool_sf_rows, c.at<float>(c.lay.pool_w),
                               static_cast<const uint8_t*>(w.w13), static_cast<const int32_t*>(w.w13_sf),
                               c.at<uint8_t>(c.lay.act_x), c.at<uint8_t>(c.lay.act_sf), c.lay.pool_sf_rows, h,
                               inter, o.activation_clamp, o.fast_math, 0, w.w13_slice_stride);
  if (e == cudaSuccess)
    e = launch_plain(simt_l2_kernel, g, b, 0, s, plan, c.e_local, c.geo.num_ranks, 0, c.at<uint8_t>(c.lay.act_x),
                     c.at<int32_t>(c.lay.act_sf), c.lay.pool_sf_rows, static_cast<const uint8_t*>(w.w2),
                     static_cast<const int32_t*>(w.w2_sf), c.at<int32_t>(c.lay.pool_dst), c.at<__nv_bfloat16>(c.lay.ret), h, inter, 0,
                     w.w2_slice_stride);
  if (c.geo.num_shared_experts > 0 && m > 0) {
    if (e == cudaSuccess)
      e = launch_plain(simt_l1_kernel, g, b, 0, s, plan, c.e_local, c.geo.num_ranks, 0, 1, c.at<uint8_t>(c.lay.x),
                       c.at<int32_t>(c.lay.x_sf), 0, nullptr, static_cast<const uint8_t*>(w.shared_w13),
                       static_cast<const int32_t*>(w.shared_w13_sf), c.at<uint8_t>(c.lay.shared_act_x),
                       c.at<uint8_t>(c.lay.shared_act_sf), c.lay.shared_sf_rows, h, inter, o.activation_clamp, o.fast_math, 1, 0);
    if (e == cudaSuccess)
      e = launch_plain(simt_l2_kernel, g, b, 0, s, plan, c.e_local, c.geo.num_ranks, 1, c.at<uint8_t>(c.lay.shared_act_x),
                       c.at<int32_t>(c.lay.shared_act_sf), c.lay.shared_sf_rows, static_cast<const uint8_t*>(w.shared_w2),
                       static_cast<const int32_t*>(w.shared_w2_sf), nullptr, c.at<__nv_bfloat16>(c.lay.shared_out), h, inter, 1, 0);
  }
  return e;
}

}  // namespace mmoe
