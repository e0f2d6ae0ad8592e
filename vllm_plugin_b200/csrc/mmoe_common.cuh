// Shared definitions of the sm_100a MegaMoE kernels: plan tables, number-format helpers and the two epilogue
// functions (SwiGLU + requantisation, BF16 store) that both the tcgen05 kernels and the scalar validation kernels call.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../include/mmoe.h"

namespace mmoe {

constexpr int kGroupK = 32;        // K elements per UE8M0 scale
constexpr int kTileK = 128;        // K elements per pipeline stage = one packed scale word
constexpr int kTileRows = 128;     // weight rows per tile (UMMA M)
constexpr int kChunkRows = 128;    // token rows per scale-factor chunk (one 512-byte tcgen05.cp source per K stage)
constexpr int kSmallTileRows = 112;      // largest token tile of the weights-as-A kernels (UMMA N): four accumulators of 112 TMEM columns
constexpr int kPairTileRows = 128;       // largest token tile of the tokens-as-A kernels (half of a CTA pair's 256 rows)
constexpr int kNeverPair = 0x7fffffff;
// The shared expert of a call on one GPU that may have pair tiles: on the pairs past this many tokens, else in tiles of the
// weights-as-A kernels, which need no scale chunks, so that one launch orders and places the routes (up to kSmallRoutes of them).  On
// pairs -> in tiles: 200 tokens of 48 experts 204 -> 195 us, of 16 (top-3) 105 -> 94, 256 of 384 1081 -> 1078, of 128 (top-3) 407 -> 400,
// of 48 206 -> 198, of 32 163 -> 155, of 16 110 -> 100; skewed popularity, 200 of 384 203 -> 194, 256 of 384 224 -> 228, of 128 144 ->
// 146, of 97 217 -> 217, of 48 199 -> 199, of 16 114 -> 108.  384 tokens 1158 -> 1166, 512 1179 -> 1202.
constexpr int kSharedPairsAbove = 256;

// Rows of a weights-as-A tile: five stages of up to 80 rows fit the shared memory, four of 112.
constexpr int kDeepTileRows = 80;

// Which kernels run a routed expert depends on the rows it received in this call: above `pair_above` (see kPairAbove) the CTA
// pairs, except where they would start a second task for at most 80 rows and the weights-as-A kernels, whose tiles have up to
// `small_cap` rows in this call, take at most four tiles instead.  A pair task takes 2 x 562 clk of SM time per stage however few
// its rows, a tile 430-500.  Three tiles of 112: 280 rows on each of 48 experts 727 -> 608 us, 336 rows 789 -> 667; at 400
// rows four lose (930 -> 957).  Four tiles of 80, a few such experts among cold ones: 12 x 280 rows among 97 experts
// 463.5 -> 453.6, 40 x 300 among 384 1745 -> 1647, 5 x 320 among 48 281.7 -> 258.7.  Five tiles, 321 to 336 rows, lose: 12 x 322
// among 97 477.2 -> 484.6, 12 x 336 479.3 -> 489.3; 40 among 384 and 5 among 48 within 2 %.
__host__ __device__ inline bool on_pairs(int n, int pair_above, int small_cap) {
  const int few_tiles = small_cap >= kSmallTileRows ? 3 * kSmallTileRows : 4 * kDeepTileRows;
  return n > pair_above && (pair_above == 0 || n <= 2 * kPairTileRows || n > few_tiles);
}

// How the n rows of an expert are cut into tiles.  Weights-as-A kernels: ceil(n / small_cap) equal tiles (rounded up to 16
// rows).  Pairs: an even number of tiles of at most 128 rows, the two halves of CTA-pair tasks; the second half
// of a single pair is empty when everything fits the first.  Cuts ignore the BLOCK_M boundaries of the pool.
struct Cut {
  int32_t parts, step;
};
__host__ __device__ inline Cut cut_rows(int n, bool pairs, int small_cap) {
  if (n <= 0) return Cut{0, 16};
  if (pairs) {
    if (n <= kPairTileRows) return Cut{2, kPairTileRows};
    const int parts = 2 * ((n + 2 * kPairTileRows - 1) / (2 * kPairTileRows));
    return Cut{parts, ((n + parts - 1) / parts + 15) & ~15};
  }
  const int parts = (n + small_cap - 1) / small_cap;
  return Cut{parts, ((n + parts - 1) / parts + 15) & ~15};
}
// GEMM1 of a call of at most this many tokens on one GPU multiplies every expert that is hit with all staged tokens and orders
// the routes itself (an UMMA takes 16 token columns at least); see staged_tokens().
constexpr int kStagedTokens = 16;
// Token slots with which a call without pair tiles starts, known to the host because its launch starts before the plan is complete;
// also the cut of its shared expert.  Slots of up to 32 rows leave room for six stages, of up to 80 for five.  Six are worth 3 % where
// a call reads many experts for a few rows each, and a tile more per 32 rows of the others costs its CTA a task:
//   BLOCK_M 16, slots of 80 -> 32: 64 tokens of 384 experts 696 -> 674 us, 192 tokens 1044 -> 1012, 192 of 128 (top-3) 383 -> 375; with
//     Zipf(1.2) popularity and two hot experts, 64 tokens of 384 127 -> 128, but 128 tokens 154 -> 165 and 192 tokens 185 -> 206.  Those
//     start with 32, and the plan decides whether they stay there (wide_tiles()).
//   BLOCK_M 32, 10 to 24 rows expected: 192 tokens of 97 experts 319 -> 312, skewed 189 -> 210, like the above.  Few experts: up to 64
//     tokens of 32 and 16 121 -> 119 and 66 -> 64; past that there is little to gain, 192 tokens of 48, 128 of 32 and 96 of 16 (top-3)
//     181 -> 182, 129 -> 129, 76.8 -> 75.7, and skewed 170 -> 193, 123 -> 134, 75 -> 76: those keep slots of 80.
// An expert of any size fits the scale chunks of its pool blocks either way, see chunks_per_block().
constexpr int kSixStageRows = 32;
constexpr int kFewExperts = 64, kFewExpertsTokens = 64;
__host__ __device__ inline int small_only_cap(int m, int block_m, int e_local) {
  if (block_m == 16 && m <= 16) return 16;
  return block_m == 16 || (block_m == 32 && (m <= kFewExpertsTokens || e_local >= kFewExperts)) ? kSixStageRows : kDeepTileRows;
}
// Whether the experts of a call that starts with slots of 32 rows are cut at 80, from the number of tiles that either makes.  The CTAs
// then drain their pipeline and start over (see sa_scheduler), which has to be earned back.  Zipf(1.2) and two hot experts: 18 tiles
// fewer of 70, 192 tokens of 384 and of 97 experts 206 -> 194 and 212 -> 202 us; ten of 57 and of 37, 128 of 384 165 -> 161, 192 of 128
// (top-3) 120 -> 118; eight of 46, 96 of 384 140.7 -> 140.5; five of 23, 96 of 128 89 -> 92.  One in eight: a call that only waits for HBM
// has 3 % to gain from the sixth stage however many tiles it has.
__host__ __device__ inline bool wide_tiles(int tiles32, int tiles80) {
  const int fewer = tiles32 - tiles80;
  return fewer >= 8 && 8 * fewer > tiles32;
}
// The cut of the shared expert's m tokens, known to the host as well, so that its tiles need no plan.  `cap`: rows of its tiles if
// it is not on pairs.
__host__ __device__ inline Cut shared_cut(int m, int pair_above, int cap) { return cut_rows(m, m > pair_above, cap); }

// Scale-factor chunks (128 token rows each) reserved per pool block of a BLOCK_M variant: at least as many as the non-empty
// tiles an expert's rows are cut into (small_cap >= 16 for BLOCK_M 16, >= 32 for 32, >= 64 for 64, >= 80 for 192 and 240).
__host__ __device__ inline int chunks_per_block(int block_m) { return block_m <= 64 ? 1 : (block_m <= 128 ? 2 : 3); }
constexpr int kSortChunkTokens = 128;
// Routes that one block orders by itself (see route_small_kernel).  Against two launches: 160 tokens of 32 experts 140.5 -> 134.0
// us, 130 of 384 978 -> 970, 192 of 384 1074 -> 1068.
constexpr int kSmallRoutes = 4096;
constexpr int kSharedExpert = -2;  // MmoeTile::expert of a shared-expert tile

// One unit of token rows handed to the grouped GEMMs: `n_valid` rows starting at `row0` of the token matrix (pool rows for
// routed experts, token indices for the shared expert), whose scales live in chunk `sf_chunk`.
struct Tile {
  int32_t expert;    // local expert index, or kSharedExpert
  int32_t row0;
  int32_t n_valid;
  int32_t sf_chunk;
  int32_t part, parts;   // this tile is the part-th of the `parts` tiles of its expert
  int32_t pad[2];
};
static_assert(sizeof(Tile) == 32, "tile record is 32 bytes");

struct PlanHeader {
  int32_t num_routed_tiles;
  int32_t num_shared_tiles;
  int32_t num_pool_blocks;     // sum over experts of ceil(n_e / BLOCK_M)
  int32_t total_recv;          // routes received by this rank
  int32_t block_m;
  int32_t num_tokens;
  int32_t num_small_tiles;     // the first of the routed tiles: those of the weights-as-A kernels; the others are pair tiles
  int32_t small_cap;           // rows a weights-as-A tile of this call may have
  int32_t small_rows;          // rows of the largest one, rounded up to 16
  int32_t ticket;              // blocks of the route-counting launch that have finished; zero between launches
  int32_t routed;              // 1 once a GEMM launch that orders the routes itself has the plan complete; zero between calls
  uint32_t claims;             // CTAs of that launch that have asked to do it, modulo its grid: zero between launches
  uint32_t next_task;          // tasks of a launch of both GEMMs that have been claimed: zero between calls
  int32_t layer1_done;         // finished parts of GEMM1 of a launch of both GEMMs, all experts (not those on CTA pairs): zero between calls
  int32_t shared_step;         // rows of the shared expert's tiles ...
  int32_t shared_pairs;        // ... and 1 if they run on CTA pairs (neither is written where the launch orders the routes itself)
};
static_assert(sizeof(PlanHeader) == 64, "plan header is 64 bytes");

// Plan region: header | expert_total[E_l] | expert_block_off[E_l+1] | expert_tile_off[E_l+1] | rank_off[R+1] |
// seg_pool_start[E_l*R] | seg_recv_start[E_l*R] | done[E_l+1] | pair_tasks[2] | pairs_open | tiles[max_tiles]
struct PlanView {
  PlanHeader* hdr;
  int32_t* expert_total;
  int32_t* expert_block_off;
  int32_t* expert_tile_off;
  int32_t* rank_off;
  int32_t* seg_pool_start;
  int32_t* seg_recv_start;
  int32_t* done;               // one GPU, both GEMMs: finished parts of GEMM1 per expert, the shared one last; zero between calls
  int32_t* pair_tasks;         // ... the tasks of either layer that CTA pairs have claimed, likewise
  int32_t* pairs_open;         // ... and the CTA pairs of GEMM1 that have seen everything in front of them complete (see open_chain), likewise
  Tile* tiles;
};

__host__ __device__ inline int64_t align_up(int64_t a, int64_t b) { return (a + b - 1) / b * b; }

// The shared expert's tiles of a launch, in front of the routed ones and without a tile record.
struct SharedTiles {
  int32_t parts, step, m;       // parts 0: none in this launch
  __host__ __device__ Tile at(int j) const {
    const int rows = m - j * step < step ? m - j * step : step;
    return rows > 0 ? Tile{kSharedExpert, j * step, rows, j, j, parts, {0, 0}} : Tile{kSharedExpert, 0, 0, 0, j, parts, {0, 0}};
  }
};

// scale chunks of the shared expert's tokens: one per tile, whatever the cut
__host__ __device__ inline int64_t shared_chunk_rows(int64_t max_tokens) { return (max_tokens / 64 + 2) * 128; }

// tile records reserved for the shared expert of a call with at most `max_tokens` tokens
__host__ __device__ inline int64_t shared_tile_capacity(int64_t max_tokens) { return (max_tokens / 16 + 2) * 2; }

__host__ __device__ inline int64_t plan_bytes(int e_local, int num_ranks, int64_t max_tiles) {
  int64_t ints = e_local + 3 * (e_local + 1) + (num_ranks + 1) + 2 * (int64_t)e_local * num_ranks + 3;
  return 64 + align_up(ints * 4, 32) + max_tiles * (int64_t)sizeof(Tile);
}

__host__ __device__ inline PlanView plan_view(void* base, int e_local, int num_ranks) {
  PlanView v;
  char* p = static_cast<char*>(base);
  v.hdr = reinterpret_cast<PlanHeader*>(p);
  int32_t* q = reinterpret_cast<int32_t*>(p + 64);
  v.expert_total = q;            q += e_local;
  v.expert_block_off = q;        q += e_local + 1;
  v.expert_tile_off = q;         q += e_local + 1;
  v.rank_off = q;                q += num_ranks + 1;
  v.seg_pool_start = q;          q += (int64_t)e_local * num_ranks;
  v.seg_recv_start = q;          q += (int64_t)e_local * num_ranks;
  v.done = q;                    q += e_local + 1;
  v.pair_tasks = q;              q += 2;
  v.pairs_open = q;              q += 1;
  int64_t ints = q - reinterpret_cast<int32_t*>(p + 64);
  v.tiles = reinterpret_cast<Tile*>(p + 64 + align_up(ints * 4, 32));
  return v;
}

// Row of a 128-row scale chunk that holds token row i of the chunk: the layout `tcgen05.cp.32x128b.warpx4` expects
// (lane i%32 receives the four 32-row groups side by side).
__host__ __device__ inline int chunk_pos(int i) { return (i & 31) * 4 + ((i >> 5) & 3); }

// Device status words (int32[8]): [0] != 0 means a bounded wait expired; [1] kernel id, [2] role, [3] block,
// [4] bad-argument counter (e.g. an expert id out of range seen by the dispatch).
// Kernel ids: 1, 2 weights-as-A, one layer (role: warp); 4 weights-as-A, both layers; 10 + b barrier b of the exchange (role: the rank
// that did not come); 21, 22 CTA pairs, one layer.
constexpr int kStatusBothLayers = 4, kStatusPairs = 20;
enum { kStatusTimeout = 0, kStatusKernel = 1, kStatusRole = 2, kStatusBlock = 3, kStatusBadIndex = 4 };

#ifdef __CUDACC__
// ---------------------------------------------------------------------------------------------------------------
// number formats
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float e4m3_to_float(uint8_t v) {
  __half_raw h = __nv_cvt_fp8_to_halfraw(v, __NV_E4M3);
  return __half2float(__half(h));
}

__device__ __forceinline__ uint8_t float_to_e4m3(float v) {
  return static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
}

__device__ __forceinline__ float e2m1_to_float(uint32_t nib) {
  // 0, .5, 1, 1.5, 2, 3, 4, 6 with the sign in bit 3
  const uint32_t mag = nib & 7u;
  float v = mag < 4u ? 0.5f * mag : (mag == 4u ? 2.f : (mag == 5u ? 3.f : (mag == 6u ? 4.f : 6.f)));
  return (nib & 8u) ? -v : v;
}

__device__ __forceinline__ float ue8m0_to_float(uint32_t b) { return __uint_as_float(b << 23); }

__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// ---------------------------------------------------------------------------------------------------------------
// L1 epilogue for one (token, channel): BF16 rounding of both accumulators, clamp (upper only for the gate),
// sigmoid, (gate*sig)*up*weight.  Operation order and roundings follow the reference's epilogue
// (backend/kernel/epilogue.py:190-221).
// ---------------------------------------------------------------------------------------------------------------
template <bool kFast>
__device__ __forceinline__ float swiglu_act_t(float gate_acc, float up_acc, float weight, float clamp) {
  float g = bf16_round(gate_acc);
  float u = bf16_round(up_acc);
  g = fminf(g, clamp);                       // clamp is a BF16-representable value (or +inf)
  u = fminf(fmaxf(u, -clamp), clamp);
  float gated;
  if (kFast) {
    float e, r;
    const float t = __fmul_rn(-g, 1.4426950408889634f);
    asm("ex2.approx.f32 %0, %1;" : "=f"(e) : "f"(t));
    const float d = __fadd_rn(1.0f, e);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    gated = __fmul_rn(g, r);
  } else {
    gated = __fdiv_rn(g, __fadd_rn(1.0f, expf(-g)));
  }
  return __fmul_rn(__fmul_rn(gated, u), weight);
}
__device__ __forceinline__ float swiglu_act(float gate_acc, float up_acc, float weight, float clamp, bool fast_math) {
  return fast_math ? swiglu_act_t<true>(gate_acc, up_acc, weight, clamp) : swiglu_act_t<false>(gate_acc, up_acc, weight, clamp);
}

// UE8M0 exponent of a non-negative amax by the integer-carry method (backend/kernel/ptx_g.py:235-241).
__device__ __forceinline__ int ue8m0_exp_of_amax(float amax) {
  const uint32_t bits = __float_as_uint(amax);
  const int rounded = static_cast<int>((bits + (0x7FFFFFu - (0x60u << 16))) >> 23);
  return max(rounded, 105 + 8) - 8;
}

__device__ __forceinline__ float ue8m0_inv(int sf_exp) { return __uint_as_float(static_cast<uint32_t>(254 - sf_exp) << 23); }

// max over the warp of non-negative floats (IEEE bits of non-negative floats order like unsigned integers)
__device__ __forceinline__ float warp_max_nonneg(float v) {
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}

__device__ __forceinline__ void report_bad_index(int32_t* status) { atomicAdd(&status[kStatusBadIndex], 1); }
#endif  // __CUDACC__

// kernels and launchers implemented in the .cu files ------------------------------------------------------------------
struct Ctx {             // resolved pointers of one call
  MmoeGeometry geo;
  MmoeLayout lay;
  char* ws;
  int e_local;
  int kmax;              // min(k, E/R)
  int32_t* stats = nullptr;               // cumulative receive counts, for a GEMM1 launch that orders the routes itself ...
  bool route_in_gemm = false;             // ... which it does when this is set
  bool both_layers = false;               // the combine that follows zeroes the counters which a launch of both GEMMs leaves
  const void* const* peer_ws = nullptr;   // set by the call that fuses the write-back into GEMM2 (EP > 1)
  int tile_select = 0;                    // 0: every tile of the plan, 1: routed tiles only, 2: the early shared tiles only
  int pair_above = kNeverPair;            // experts with more rows than this run on CTA pairs ...
  // ... in a call of m tokens on this rank: in a small one none does, and the call needs no pair launch.  On one GPU a call is
  // small when no expert can have that many rows (but for tokens that name one twice).
  // With several ranks the host knows only its own tokens and takes the others to have as many, as the choice of BLOCK_M does;
  // a rank without tokens knows nothing.  Two empty pair launches cost 7.3 us, which hot experts have to earn back.  GEMMs of
  // one rank of 8, 48 experts each, Zipf(1.2) / even popularity, never -> with pairs: 64 tokens 164 -> 172 / 171 -> 178 us,
  // 256: 208 -> 217 / 198 -> 216, 512: 254 -> 271 / 215 -> 230, 1024: 357 -> 354 / 330 -> 340, 1920: 545 -> 477 / 525 -> 442.
  // One of 2 (192 experts), 512 tokens: 624 -> 625 / 616 -> 626.  16 experts, top-3, 512 tokens (96 rows each): 135 -> 145 /
  // 139 -> 142.  A rank that misjudges the others is slower by the same measure, not wrong.
  static constexpr int kFewRoutes = 3072, kFewRows = 96;
  int pair_above_for(int m) const {
    if (geo.num_ranks == 1) return m <= pair_above ? kNeverPair : pair_above;
    const int64_t routes = (int64_t)m * geo.num_topk;
    return pair_above > 0 && m > 0 && routes <= kFewRoutes && routes <= (int64_t)kFewRows * e_local ? kNeverPair : pair_above;
  }
  // The shared expert of such a call runs on CTA pairs past this many tokens ...
  int shared_above_for(int m) const {
    const int above = tile_select == 2 ? pair_above : pair_above_for(m);
    return geo.num_ranks == 1 && tile_select != 2 && above > 0 && above < kSharedPairsAbove ? kSharedPairsAbove : above;
  }
  // ... and up to it in tiles of so many rows, which the plan of a call that may have pair tiles raises to kDeepTileRows.
  int shared_cap_for(int m, int block_m) const {
    if (geo.num_ranks > 1 || tile_select == 2) return kDeepTileRows;
    return pair_above_for(m) == kNeverPair ? small_only_cap(m, block_m, e_local) : kSixStageRows;
  }
  template <typename T> T* at(int64_t off) const { return reinterpret_cast<T*>(ws + off); }
  bool fused() const { return peer_ws != nullptr && geo.num_ranks > 1 && tile_select != 2; }
};

// The GEMM launches of a call of m tokens: on CTA pairs, on the weights-as-A kernels, or both in this order.
struct GemmForms {
  bool pairs, small;
};
inline GemmForms gemm_forms(const Ctx& c, int m, bool with_shared) {
  // the shared expert by itself takes one launch in either form
  if (c.tile_select == 2) return GemmForms{with_shared && m > c.pair_above, with_shared && m <= c.pair_above};
  const int pair_above = c.pair_above_for(m);
  return GemmForms{pair_above != kNeverPair, pair_above > 0};
}

// Whether GEMM1 of such a call, in one launch with GEMM2, takes the staged tokens as they are instead of the rows of the pool.  With more than one rank the
// rows come from other ranks and the route table names experts of all of them: only one GPU's call may.
inline bool staged_tokens(const Ctx& c, int m, int block_m) {
  return c.geo.num_ranks == 1 && c.tile_select != 2 && c.pair_above_for(m) == kNeverPair && m > 0 && m <= kStagedTokens &&
         block_m <= kStagedTokens;
}


// ---------------------------------------------------------------------------------------------------------------------
// Programmatic dependent launch.  The kernels of one call form a chain on a stream.  chain_release() lets the NEXT kernel of
// the stream be scheduled as soon as every block of this one has come to it or ended (so that kernel's launch latency and
// set-up -- barrier initialisation, tensor-memory allocation -- overlap this kernel's run); chain_wait() waits until
// everything BEFORE this kernel in the stream has completed and its memory is visible.  Most kernels begin with both, in this
// order (chain_begin()), and touch no global memory before.  The wait is transitive: the next kernel's wait ends only when
// this grid has completed, and this grid completes only after its own wait has.  Nothing is taken to be complete about a kernel from
// elsewhere, which may release as early as it likes.  Both instructions do nothing in a kernel that was launched without the
// attribute below.
//
// A kernel of this library that waits first and releases then tells its successor more: what precedes IT has completed when the
// successor starts, which may use that without waiting for IT.  But visibility is promised to a grid that waits, and to no other.  So
//   * what follows the pairs' GEMM1 (their GEMM2, and the launch of both GEMMs) is told in memory: GEMM1 counts a release (open_chain)
//     between its wait and its chain_release(), and every thread of the launches behind acquires it or, where it finds nothing, waits
//     for all of GEMM1 after all (chain_opened);
//   * a GEMM launch behind the route ordering starts with the staged tokens alone.  Nobody counts for it: it relies on the ordering's
//     wait having brought the staged rows and scales to the L2, and reads them there: by bulk copies, and the scales behind a fence that
//     leaves nothing older in the L1.
// What one launch of a call writes for another (pool_w, pool_dst, scales) is never read through the read-only path (__ldg), which is for
// memory that nobody writes while the kernel runs.
// ---------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void open_chain(int32_t* word) {
  asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(word) : "memory");
}
__device__ __forceinline__ bool chain_opened(const int32_t* word) {
  int32_t v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
  return v > 0;
}
__device__ __forceinline__ void chain_begin() {
  chain_release();
  chain_wait();
}

// The entry points of single-GPU calls open a ChainScope; every launch outside one is an ordinary one.  A GEMM CTA holds an SM
// to itself, so what starts early there is the next launch's CTA on an SM that has run out of tasks.  Chain plus shared
// expert first, measured together: 7 tokens 163 -> 141 us, 128 tokens / 32 experts 155 -> 144, 3840 / 384 1784 -> 1683.
struct ChainScope {
  explicit ChainScope(bool on);
  ~ChainScope();
  ChainScope(const ChainScope&) = delete;
  ChainScope& operator=(const ChainScope&) = delete;
 private:
  bool saved_;
};
bool chained();   // true: launch with the attribute

// The three forms of a launch.  Each returns the status of this launch alone: cudaGetLastError() behind one also returns what an
// earlier call left on the thread, and a kernel that does run would be taken for one that does not.
template <typename... KArgs, typename... Args>
cudaError_t launch_plain(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(std::forward<Args>(args))...);
}

// as part of the chain
template <typename... KArgs, typename... Args>
cudaError_t launch_chained(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chained() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(std::forward<Args>(args))...);
}

// ... and a kernel of CTA clusters
template <typename... KArgs, typename... Args>
cudaError_t launch_clustered(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, int cluster, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chained() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(std::forward<Args>(args))...);
}

cudaError_t launch_stage(const Ctx& c, const void* hidden, const void* ids, int ids64, const float* w,
                         const uint8_t* pad, int m, int shared_bm, cudaStream_t s);
cudaError_t launch_route_stage(const Ctx& c, const void* hidden, const void* ids, int ids64, const float* w,
                               const float* logits, int num_logical, const int32_t* replica_count,
                               const int32_t* replica_slots, int max_copies, const uint8_t* pad, int m, int shared_bm,
                               cudaStream_t s);
cudaError_t launch_stage_nvfp4(const void* hidden, void* q_out, void* sf_out, float global_scale, int64_t num_tokens, int hidden_size,
                               cudaStream_t s);
cudaError_t launch_count_sort(const Ctx& c, int m, cudaStream_t s);
cudaError_t launch_pack(const Ctx& c, int m, cudaStream_t s);
cudaError_t launch_route_small(const Ctx& c, int m, int block_m, int32_t* stats, cudaStream_t s);
cudaError_t launch_route_large(const Ctx& c, int m, int block_m, int32_t* stats, cudaStream_t s);
cudaError_t launch_plan_place(const Ctx& c, int m, int block_m, int32_t* stats, cudaStream_t s);
cudaError_t launch_shared_plan(const Ctx& c, int m, cudaStream_t s);
cudaError_t launch_combine(const Ctx& c, void* y, const void* residual, int m, cudaStream_t s);
cudaError_t zero_counters(const Ctx& c, cudaStream_t s);   // what the combine of a single-GPU call zeroes, for a call whose combine was not launched
cudaError_t launch_experts_simt(const Ctx& c, const MmoeWeights& w, const MmoeOptions& o, int m, int block_m, cudaStream_t s);
cudaError_t launch_experts_umma(const Ctx& c, const MmoeWeights& w, const MmoeOptions& o, int m, int block_m, cudaStream_t s);
int prepare_umma(const MmoeGeometry& geo);   // returns an MMOE_* code
bool tc_ready();                             // prepare_umma() has run on the current device
void set_tuning(int max_stages, int orientation);
int tuned_orientation();                     // 0: per expert, 1: weights-as-A, 2 and 3: tokens-as-A on CTA pairs
cudaError_t route_order_static(const int64_t* topk_idx, int m, int k, int num_experts, int32_t* send_count,
                               int32_t* send_offset, int32_t* route_pos, int32_t* sorted_route, cudaStream_t s);
int route_order_static_max_tokens();
int route_order_static_max_experts();
cudaError_t launch_interleave_rows(const void* src, void* dst, int groups, int rows, int row_bytes, cudaStream_t s);
cudaError_t launch_scale_layout(const int32_t* src, int32_t* dst, int groups, int rows, int row_stride, int kwords,
                                int interleave, cudaStream_t s);
cudaError_t launch_split_halves(const void* src, void* dst, int groups, int64_t half_bytes, int64_t slice_stride, cudaStream_t s);
int ep_sync_bytes();
int ep_totals_offset();                      // byte offset of the [32][32] route-total table inside the ep_sync region
cudaError_t launch_ep_signal_return(const Ctx& c, const void* const* peer_ws, int64_t timeout_ns, cudaStream_t s);
cudaError_t launch_ep_dispatch(const Ctx& c, const void* const* peer_ws, int m, int64_t timeout_ns, cudaStream_t s);
cudaError_t launch_ep_return(const Ctx& c, const void* const* peer_ws, int64_t timeout_ns, cudaStream_t s);

}  // namespace mmoe
