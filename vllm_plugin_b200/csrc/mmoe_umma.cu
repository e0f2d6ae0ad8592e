// Grouped block-scaled GEMMs of the MegaMoE layer on the sm_100a tensor cores.
//
//   layer 1:  acc[ch, tok] = sum_k W13[e][ch, k] * x[tok, k]   (gate rows and up rows of one 128-channel tile in two
//             TMEM accumulators) -> SwiGLU, x top-k weight, per-32-channel UE8M0 requantisation to E4M3
//   layer 2:  acc[h, tok]  = sum_i W2[e][h, i] * act[tok, i]   -> BF16 rows of the return buffer
//
// Weights are the UMMA "A" operand (M = 128 rows), tokens the "B" operand (N = 16..112 tokens), so a small token
// count costs a small N instead of a padded M: `tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale`, MXFP4 (E2M1) or
// E4M3 weights x E4M3 activations with UE8M0 scales per 32 K.  The same roles exist in the reference's kernel
// (backend/kernel/tma_warps.py, mma_warp.py, epilogue.py, scheduler.py); the structure here is B200's:
//
//   warp 0     producer: one thread issues the TMA tile loads (packed FP4 expands to byte containers on the way into
//              shared memory; no cluster multicast) and 512-byte bulk copies of the scale chunks, per 128-K stage
//   warps 1,6  MMA: one warp per weight tile of the stage; an elected lane copies the scales into TMEM (tcgen05.cp) and
//              issues 4 UMMAs per stage, committing the stage's shared memory back to the producer and the finished
//              accumulator to the epilogue
//   warps 2-5  epilogue: TMEM -> registers (thread = weight row, columns = tokens), fused math, global stores
//   warp 7     layer 1: brings a stage's weight scales from stored into tensor-memory order ahead of the MMA warps
//   warp 8     both layers in one launch: claims the CTA's next task (scheduler)
//
// A call on one GPU runs both layers in one launch (moe_kernel) of persistent CTAs, one per SM, that claim their tasks (tile, 256
// weight rows) from a counter; with several ranks, and where a caller asks for one layer, umma_kernel walks a list dealt out
// beforehand.  TMEM accumulators are double buffered so the epilogue of task i overlaps the loads and MMAs of task i+1.  Every
// wait is bounded: when the budget expires the CTA records {kernel, role, block} in the status words, lets its in-flight copies
// land, frees its TMEM and returns; nothing traps.
//
// Expert parallelism: layer 2 has a second form (kFused) whose epilogue stores every BF16 row straight into the buffer
// of the rank the token came from (plain peer stores over NVLink, no TMA from or to peer memory), and `tile_select`
// restricts a launch to the routed tiles or to the shared expert's, so that the shared expert can run while the dispatch is still in flight on another stream.
#include <string.h>

#include <memory>
#include <type_traits>

#include "mmoe_plan_cache.h"
#include "mmoe_tc.cuh"

namespace mmoe {

namespace {

constexpr int kThreads = 256;   // producer, MMA 0, 4 epilogue warps, MMA 1, scale arranger (layer 1)
constexpr int both_threads(bool staged) { return kThreads + (staged ? 64 : 32); }   // a scheduler, and a warp that places rows

constexpr int kNumBoxes = kSmallTileRows / 16;

struct UmmaParams {
  CUtensorMap map_w_routed;    // FP4 weights, box 128 K x 256 rows (layer 1: the 5-D de-interleaving form)
  CUtensorMap map_w_shared;    // E4M3 weights of the shared expert
  const char* plan;
  const int32_t* wsf_routed;   // [E_l][K/128][rows_per_expert] scale words, 4x32 transposed per 128 rows
  const int32_t* wsf_shared;
  const int32_t* tsf_routed;   // token scale chunks: word w of chunk row r at w * tsf_rows + r
  const int32_t* tsf_shared;   // layer 2 only
  int64_t tsf_rows_routed, tsf_rows_shared;
  // layer-1 outputs
  uint8_t* act_routed;
  uint8_t* act_shared;
  uint8_t* act_sf_routed;      // byte view of the activation scale chunks
  uint8_t* act_sf_shared;
  int64_t act_sf_rows_routed, act_sf_rows_shared;
  float* pool_w;
  // layer-2 outputs
  __nv_bfloat16* ret;
  __nv_bfloat16* shared_out;
  int32_t* pool_dst;
  SharedTiles shared_tiles;    // run first
  int shared_in_plan;          // 1: their cut is the plan's, which is complete when the launch starts
  int with_routed;             // 0: only those
  int tile_rows;               // > 0: rows of the token slots that the launch starts with; 0: those of the call's largest tile, in the plan
  int early;                   // both layers: 1 when the launch in front lets this one start with the staged tokens complete, not the plan
  int behind_pairs;            // both layers: 1 when the launches in front are the pairs', of which this one needs nothing (see chain_opened)
  const int32_t* x_sf;         // layer 1: the staged tokens' scale words [T][K/128], gathered for tiles of staged tokens
  // calls of at most kStagedTokens tokens: every routed tile of layer 1 is the staged tokens themselves (see TaskQueue)
  const int64_t* topk_idx;
  int32_t* sorted_route;
  int num_routes, topk;
  // ... and with route_here the launch also orders the routes, builds the plan and places the rows
  int route_here;
  const float* topk_weights;
  int32_t* route_pos;
  int32_t* send_count;
  int32_t* send_offset;
  int32_t* recv_count;
  int32_t* stats;
  const uint4* x;
  uint4* pool_x;
  int32_t* pool_sf;
  int64_t pool_sf_rows;
  // layer 2 at EP > 1 with the write-back fused in: an output row goes straight into the `ret_recv` of the rank its
  // token came from (plain peer stores over NVLink), at that rank's send position
  int ep_me;
  const int32_t* ep_totals;    // [32][32]: totals[s][d] = routes rank s sent to rank d in this call
  __nv_bfloat16* ep_ret_recv[32];
  int32_t* status;
  int64_t timeout_ns;
  int e_local, num_ranks;
  int k_dim;                   // reduction length: H (layer 1) or I (layer 2)
  int rows_per_expert;         // 2I (layer 1) or H (layer 2)
  int routed_sliced;           // 1: routed weights are [2, E_l, rows/2, K/2] (two slices), 0: [E_l, rows, K/2]
  int routed_halves;           // layer 2: 1 when a slice is not whole 256-row blocks; the map's box is 128 rows then
  int n_blocks;                // 128-row weight blocks per tile: I/128 (layer 1) or H/128 (layer 2)
  int hidden, inter;
  float clamp;
  int fast_math;
  int max_stages;              // > 0: cap on the shared-memory pipeline depth
  CUtensorMap map_tok_routed_box[kNumBoxes];   // token maps with boxes of 16, 32, ... 112 rows
  CUtensorMap map_tok_shared_box[kNumBoxes];
};

// A task as the scheduler hands it to the other roles of its CTA.
struct QueueSlot {
  Tile tile;
  int32_t nb, layer;      // 256-row weight block; 0 in place of the layer: no more tasks
  int32_t ready;          // layer 2: the token rows are complete
};
constexpr int kQueue = 4;

// Both layers of a single-GPU call in one launch.
struct MoeParams {
  UmmaParams layer[2];
};

struct Control {          // lives at the start of shared memory
  uint64_t full[8];       // producer -> MMA warps: the stage's copies have landed
  uint64_t empty[8];      // MMA -> producer: the stage's shared memory may be overwritten
  uint64_t sf_full[8];    // layer 1, producer -> scale arranger: the stage's weight scales have landed (in stored order)
  uint64_t sf_ready[8];   // layer 1, scale arranger -> MMA warps: ... and are in tensor-memory order
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  volatile int32_t abort_flag;
  uint32_t routes_here;   // staged tokens: this CTA orders the routes
  int32_t next_rows;      // both layers: > 0 when the roles are to start over with token slots of so many rows
  union {
    struct {              // both layers in the launch
      uint64_t q_full[kQueue];    // scheduler -> the other roles: a task
      uint64_t q_empty[kQueue];   // ... which all of them have read
      uint64_t q_want;            // producer -> scheduler: the next one, please
      QueueSlot slots[kQueue];
      uint32_t hit[16];   // staged tokens: bit e = some token is routed to expert e
    };
    struct {              // layer 2 with the write-back fused in: where output rows go
      __nv_bfloat16* out_base[33];   // slot s < 32: `ret_recv` of source rank s, slot 32: the shared expert's (local) output
      int32_t rank_off[33];          // first receive-order row of each source rank
      int32_t home_base[32];         // ... and the send position on that rank of the first row it sent here
    };
  };
};
static_assert(sizeof(Control) <= 1024, "control block");

// Every task multiplies TWO 128-row weight tiles with one token tile: layer 1 the gate rows and the up rows of 128
// channels, layer 2 two consecutive 128-row blocks of W2.  Two tiles per stage halve the per-byte cost of everything
// that is paid per stage (barrier hand-offs, token tile, token scales) and give the two MMA-issuing warps one
// accumulator each.
//
// The token slot of a stage is as large as the largest tile of the call (rounded up to 16 rows), which the plan records, so
// one kernel serves every call: 6 stages up to 32 rows, 5 up to 80, 4 at 96 and 112.
template <int kLayer>
struct Shape {
  static constexpr int kABytes = 2 * kTileRows * kTileK;           // byte containers in shared memory
  // scale area of a stage: weight scales of the two tiles, 2 x 512, and token scales, 512.  Layer 1 receives the weight scales in
  // stored (gate/up interleaved) order, and the scale arranger rewrites them in place: with 1 KB more for the stored order, token
  // slots of 32 rows had five stages instead of six (24 tokens of 384 experts 370 -> 360 us, 1000 tokens 1284 -> 1249).
  static constexpr int kSfBytes = 3 * 512;
  static constexpr int kMaxStages = 8;
  static constexpr int kRingBytes = kSmemBudget - 1024;
  static constexpr int kSmemBytes = 1024 + kRingBytes + 1024;      // control block + stages + alignment slack
  static constexpr int kNCap = kSmallTileRows;                     // accumulator columns per weight tile
  static constexpr int kAccCols = 2 * kNCap;                       // TMEM columns of one accumulator stage
  static constexpr int kSfCol = 2 * kAccCols;                      // scale region: A0, A1, token scales (one copy per MMA warp)
  __host__ __device__ static int stages(int tile_rows) {
    const int n = kRingBytes / (kABytes + tile_rows * kTileK + kSfBytes);
    return n < kMaxStages ? n : kMaxStages;
  }
  static_assert(kSfCol + 16 <= (int)kTmemCols, "TMEM budget");
  static_assert(kRingBytes / (kABytes + kSmallTileRows * kTileK + kSfBytes) >= 4, "pipeline too shallow");
  static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
};

// ---------------------------------------------------------------------------------------------------------------
// The roles, each a function of (layer, stage layout L).
// ---------------------------------------------------------------------------------------------------------------
struct RoleState {                 // pipeline position of a role
  uint32_t stage = 0, phase = 0;   // position in the shared-memory ring
  uint32_t it = 0;                 // tasks this CTA has started: selects the accumulator buffer and its barrier phase
  bool ok = true;                  // false once the call is being abandoned
};

struct Cta {                       // where a role finds the CTA's resources
  Control* ctl;
  uint8_t* a_base;
  uint8_t* b_base;
  uint8_t* sf_base;
  uint32_t tmem_base;
  uint32_t num_stages;
  uint32_t b_bytes;                // token slot of a stage
};

// Tile by tile, or for an expert with several tiles weight block by weight block, so that the tiles of a block read its weights
// while they are in L2.
__device__ __forceinline__ void locate_task(const Tile* tiles, int task, int n_blocks, Tile* tile, int* nb) {
  const int i = task / n_blocks;
  *tile = tiles[i];
  *nb = task - i * n_blocks;
  if (tile->parts > 1) {
    const int first = i - tile->part, local = task - first * n_blocks;
    *nb = local / tile->parts;
    *tile = tiles[first + local - *nb * tile->parts];
  }
}

__device__ __forceinline__ SharedTiles sa_shared_tiles(const UmmaParams& p) {
  if (!p.shared_in_plan || p.shared_tiles.parts == 0) return p.shared_tiles;
  const PlanHeader* hdr = plan_view(const_cast<char*>(p.plan), p.e_local, p.num_ranks).hdr;
  return SharedTiles{hdr->num_shared_tiles, hdr->shared_step, p.shared_tiles.m};
}

// The task list of one CTA as a role walks it in a launch of one layer.  First the shared expert's tasks, which need nothing but
// the staged tokens and the host's count of them; then -- after what precedes this launch in the stream has completed -- the
// routed tiles of the plan.  After the first round the CTAs take their tasks in the opposite order: the first ones, whose shared
// tasks have twice the weight bytes, are not also the ones with a task more in the last round.
template <int kLaunchLayer>
struct TaskWalk {
  static constexpr bool kBoth = false;
  static constexpr int kLayer = kLaunchLayer;
  const UmmaParams& p;
  const SharedTiles shared;
  int shared_tasks, routed_tasks, round;
  bool waited;
  const Tile* tiles;
  Tile tile;               // current task
  int nb;
  // `plan_ready`: the plan is complete, without a wait
  __device__ __forceinline__ TaskWalk(const UmmaParams& params, bool plan_ready)
      : p(params), shared(sa_shared_tiles(params)), shared_tasks(shared.parts * params.n_blocks), routed_tasks(0), round(0), waited(false), tiles(nullptr) {
    if (plan_ready) load_plan(true);
  }
  __device__ __forceinline__ void load_plan(bool ready) {
    if (!ready) chain_wait();
    const PlanView pv = plan_view(const_cast<char*>(p.plan), p.e_local, p.num_ranks);
    tiles = pv.tiles;
    routed_tasks = p.with_routed ? pv.hdr->num_small_tiles * p.n_blocks : 0;
    waited = true;
  }
  // true: tile and nb are the next task's
  __device__ __forceinline__ bool next(Waiter&) {
    int task = round == 0 ? blockIdx.x : (round + 1) * gridDim.x - 1 - blockIdx.x;
    ++round;
    if (task < shared_tasks) {
      nb = task / shared.parts;
      tile = shared.at(task - nb * shared.parts);
      return true;
    }
    task -= shared_tasks;
    if (!waited) load_plan(false);
    if (task >= routed_tasks) return false;
    locate_task(tiles, task, p.n_blocks, &tile, &nb);
    return true;
  }
};

// Both layers in one launch: the tasks as the scheduler hands them on.
template <bool kOneLanePolls>
struct TaskFeed {
  static constexpr bool kBoth = true;
  const MoeParams& f;
  Control* ctl;
  uint32_t taken;
  Tile tile;               // current task
  int nb, layer;
  bool ready;
  __device__ __forceinline__ TaskFeed(const MoeParams& params, Control* control) : f(params), ctl(control), taken(0) {}
  __device__ __forceinline__ bool next(Waiter& waiter) {
    const uint32_t slot = taken % kQueue, bar = smem_u32(&ctl->q_full[slot]), parity = (taken / kQueue) & 1u;
    if (!(kOneLanePolls ? waiter.wait_warp(bar, parity) : waiter.wait_uniform(bar, parity))) return false;
    const QueueSlot& s = ctl->slots[slot];
    tile = s.tile;
    nb = s.nb;
    layer = s.layer;
    ready = s.ready != 0;
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(smem_u32(&ctl->q_empty[slot]));
    ++taken;
    return layer != 0;
  }
};

// body(layer as a type, parameters of that layer) for every task of a role
template <typename Walk, typename Body>
__device__ __forceinline__ void for_each_task(Walk& walk, Waiter& waiter, RoleState& st, Body&& body) {
  while (st.ok && walk.next(waiter)) {
    if constexpr (Walk::kBoth) {
      if (walk.layer == 1) body(std::integral_constant<int, 1>{}, walk.f.layer[0]);
      else body(std::integral_constant<int, 2>{}, walk.f.layer[1]);
    } else {
      body(std::integral_constant<int, Walk::kLayer>{}, walk.p);
    }
  }
}

// ------------------------------------------------------------------------------------------------ routing in the launch
// Calls of at most kStagedTokens tokens: the epilogue warps of the first CTA to ask, idle until its first accumulator 15 us
// later, order the routes and build the plan, which only epilogues and layer 2 need.  All other CTAs wait for that one, so it has
// to be one that runs: a CTA takes an SM to itself, and work on other streams may hold any of them back for as long as it
// likes.  A launch of its own took 8-20 us in front of GEMM1: little work, but every instruction line comes from DRAM (each
// call streams its weights through the L2), so what counts is that the code is short.  Pool blocks and tiles have 16 rows
// here, hence one tile per block.
constexpr int kRouteThreads = 128;
constexpr int kMaxHereRoutes = kStagedTokens * 31, kMaxHereExperts = 512;
struct alignas(16) RouteScratch {
  uint32_t count[kMaxHereExperts];
  uint32_t before[kMaxHereExperts];      // rows | blocks << 16 of the experts before it
  uint16_t ids[kMaxHereRoutes + 16];
  uint32_t warp_sum[4];
};
static_assert(6 * (Shape<1>::kABytes + kStagedTokens * kTileK + Shape<1>::kSfBytes) + sizeof(RouteScratch) <= Shape<1>::kRingBytes &&
                  Shape<1>::kRingBytes / (Shape<1>::kABytes + kStagedTokens * kTileK + Shape<1>::kSfBytes) == 6,
              "the scratch lives behind the six stages of a 16-row ring");
__device__ __forceinline__ void route_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kRouteThreads) : "memory"); }

// whether this CTA is the first of its launch to ask; all epilogue threads of every CTA, once
__device__ __forceinline__ bool sa_claim_route(const UmmaParams& p, Control* ctl, int t) {
  if (t == 0) {
    uint32_t* claims = &plan_view(const_cast<char*>(p.plan), p.e_local, p.num_ranks).hdr->claims;
    ctl->routes_here = atomicInc(claims, gridDim.x - 1) == 0 ? 1u : 0u;
  }
  route_barrier();
  return ctl->routes_here != 0;
}

__device__ __noinline__ void sa_route(const UmmaParams& p, RouteScratch& s, int t) {
  const int E = p.e_local, n = p.num_routes, lane = t & 31;
#pragma unroll 1
  for (int e = t; e < kMaxHereExperts; e += kRouteThreads) s.count[e] = 0u;
  route_barrier();
#pragma unroll 1
  for (int i = t; i < n; i += kRouteThreads) {
    const int64_t id = p.topk_idx[i];
    if (id >= E) report_bad_index(p.status);
    s.ids[i] = id >= 0 && id < E ? static_cast<uint16_t>(id) : 0xFFFF;
    if (id >= 0 && id < E) atomicAdd(&s.count[id], 1u);
  }
  route_barrier();
  uint4 c = reinterpret_cast<const uint4*>(s.count)[t];        // this thread's four experts
  c.x |= ((c.x + 15) >> 4) << 16;
  c.y |= ((c.y + 15) >> 4) << 16;
  c.z |= ((c.z + 15) >> 4) << 16;
  c.w |= ((c.w + 15) >> 4) << 16;
  const uint32_t sum = c.x + c.y + c.z + c.w;
  uint32_t incl = sum;
#pragma unroll 1
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  if (lane == 31) s.warp_sum[t >> 5] = incl;
  route_barrier();
  uint32_t at = incl - sum, total = 0;
#pragma unroll 1
  for (int w = 0; w < 4; ++w) {
    if (w < (t >> 5)) at += s.warp_sum[w];
    total += s.warp_sum[w];
  }
  reinterpret_cast<uint4*>(s.before)[t] = make_uint4(at, at + c.x, at + c.x + c.y, at + c.x + c.y + c.z);
  route_barrier();
  const PlanView pv = plan_view(const_cast<char*>(p.plan), E, 1);
#pragma unroll 1
  for (int e = t; e <= E; e += kRouteThreads) {
    const uint32_t off = e < E ? s.before[e] : total;
    const int row = static_cast<int>(off & 0xFFFF), block = static_cast<int>(off >> 16);
    p.send_offset[e] = row;
    pv.expert_block_off[e] = block;
    pv.expert_tile_off[e] = block;
    if (e == E) break;
    const int n_e = static_cast<int>(s.count[e]);
    p.send_count[e] = n_e;
    p.recv_count[e] = n_e;
    pv.expert_total[e] = n_e;
    pv.seg_pool_start[e] = block * kStagedTokens;
    pv.seg_recv_start[e] = row;
    if (p.stats != nullptr && n_e > 0) atomicAdd(&p.stats[e], n_e);      // cumulative per-expert receive statistics (dispatch.py:644-650)
    const int parts = (n_e + kStagedTokens - 1) / kStagedTokens;
#pragma unroll 1
    for (int j = 0; j < parts; ++j)
      pv.tiles[block + j] = Tile{e, (block + j) * kStagedTokens, min(kStagedTokens, n_e - j * kStagedTokens), block + j, j, parts, {0, 0}};
  }
  if (t == 0) {
    const int rows = static_cast<int>(total & 0xFFFF), tiles = static_cast<int>(total >> 16);
    int32_t* h = reinterpret_cast<int32_t*>(pv.hdr);       // the fields in order
    reinterpret_cast<int4*>(h)[0] = make_int4(tiles, p.shared_tiles.parts, tiles, rows);
    reinterpret_cast<int4*>(h)[1] = make_int4(kStagedTokens, p.shared_tiles.m, tiles, kStagedTokens);
    h[8] = kStagedTokens;
    pv.rank_off[0] = 0;
    pv.rank_off[1] = rows;
    if (p.shared_tiles.parts > 0) pv.tiles[tiles] = p.shared_tiles.at(0);
  }
#pragma unroll 1
  for (int i = t; i < n; i += kRouteThreads) {
    const uint32_t e = s.ids[i];
    int pos = -1;
    if (e != 0xFFFFu) {
      uint32_t rank = 0;
#pragma unroll 1
      for (int o = 0; o < i; ++o) rank += s.ids[o] == e ? 1u : 0u;
      pos = static_cast<int>((s.before[e] & 0xFFFF) + rank);
      const int row = static_cast<int>((s.before[e] >> 16) * kStagedTokens + rank);
      p.sorted_route[pos] = i;
      p.pool_w[row] = p.topk_weights[i];
      p.pool_dst[row] = pos;
    }
    p.route_pos[i] = pos;
  }
  __threadfence();
  route_barrier();
  if (t == 0) asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(&pv.hdr->routed), "r"(1) : "memory");
}

// The placed rows and scales of such a call, which nothing in it reads, by a warp of their own.
__device__ __noinline__ void sa_place(const UmmaParams& p) {
  const int lane = threadIdx.x & 31, vec = p.hidden / 16, words = p.hidden / kTileK;
  const PlanView pv = plan_view(const_cast<char*>(p.plan), p.e_local, 1);
  for (int i = blockIdx.x; i < p.num_routes; i += gridDim.x) {
    const int pos = p.route_pos[i];
    if (pos < 0) continue;
    const int e = static_cast<int>(p.topk_idx[i]), r = pos - p.send_offset[e], t = i / p.topk, block = pv.expert_block_off[e];
    const uint4* src = p.x + (int64_t)t * vec;
    uint4* dst = p.pool_x + (int64_t)(block * kStagedTokens + r) * vec;
#pragma unroll 1
    for (int v = lane; v < vec; v += 32) dst[v] = src[v];
    int32_t* sf = p.pool_sf + (int64_t)(block + r / kStagedTokens) * kChunkRows + chunk_pos(r % kStagedTokens);
#pragma unroll 1
    for (int w = lane; w < words; w += 32) sf[w * p.pool_sf_rows] = p.x_sf[(int64_t)t * words + w];
  }
}

// waits until the plan is complete, whole warp; false when the call is being abandoned
__device__ __forceinline__ bool sa_wait_plan(const UmmaParams& p, Waiter& waiter) {
  if (!p.route_here) {
    chain_wait();
    return true;
  }
  const int32_t* flag = &plan_view(const_cast<char*>(p.plan), p.e_local, p.num_ranks).hdr->routed;
  for (uint32_t spin = 0;; ++spin) {
    int32_t v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (__any_sync(0xffffffffu, v != 0)) {
      asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");   // by every lane
      return true;
    }
    if ((spin & 63u) == 63u && __any_sync(0xffffffffu, waiter.abandoned())) return false;
    __nanosleep(100);
  }
}

// ------------------------------------------------------------------------------------------------ both layers in one launch
// Counts a part of GEMM1 (see part_release), for its expert and in one counter for all, which spares a CTA the question once GEMM1 is
// over.  One fence releases both additions; with a sequentially consistent one and a release of its own on the first addition, each of
// which waits for the stores, one token took 39.45 us instead of 38.95, seven 134.2 instead of 133.1.
__device__ __forceinline__ void sa_publish(const PlanView& pv, int slot) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    part_release();
    part_count(pv.done + slot);
    part_count(&pv.hdr->layer1_done);
  }
}

// The task list of such a launch: shared expert and routed tiles of layer 1, then of layer 2.  CTAs claim tasks from a counter when
// the last stages of the one before are being requested, so that
//   * the memory system never waits for the slowest CTA: claimed by whoever is free, GEMM2's tasks fill GEMM1's last round, and
//     their weights are requested before the activations are complete.  Two launches with tasks dealt out beforehand: 4 tokens
//     of 384 experts 94 -> 84 us, 7 tokens 147 -> 137, 128 tokens of 32 experts 150 -> 132, 64 of 384 762 -> 744, 256 of 384
//     1166 -> 1138, 1021 of 384 skewed 483 -> 467;
//   * what a CTA waits for was claimed earlier, by a CTA that runs: a call needs no particular CTA to be resident, whatever other
//     streams do to the SMs.
// A warp of its own claims and looks up (the scheduler): the latency of the counter and of the tables in the producer's loop
// left stages empty, 10 % of GEMM2's time at HBM speed.
// The shared expert's tasks of layer 1 need nothing but the staged tokens and the host's count of them, the routed ones the plan.
//
// GEMM1 of at most 16 tokens needs no placed rows either: an UMMA takes 16 token columns at least, so every expert that some
// token is routed to multiplies all staged tokens, and the epilogue takes the columns of the tokens routed to it.  Which
// experts those are every CTA reads from the route table itself; only the epilogue waits for the plan.
// The 256 stored weight rows of a task.  Layer 1 reads W13 in its stored order [g0..7, u0..7, g8..15, ...] through a 5-D map (K, row
// in group of 8, group of 16 rows, gate/up, slice): one box of 8 x 16 x 2 lands the 128 gate rows and then the 128 up rows of
// 128 consecutive channels.  Layer 2 reads 256 consecutive rows; with slices of an odd number of 128-row blocks (`halves`) the
// two blocks are loaded one by one, the second may be in the other slice.
struct WeightRows {
  const CUtensorMap* map;
  int row, slice, row2, slice2;
  bool halves;
};
template <int kLayer>
__device__ __forceinline__ WeightRows sa_weight_rows(const UmmaParams& p, const Tile& tile, int nb) {
  const bool shared = tile.expert == kSharedExpert, sliced = !shared && p.routed_sliced != 0;
  const int e = shared ? 0 : tile.expert;
  const int rows_slice = sliced ? p.rows_per_expert / 2 : p.rows_per_expert;   // rows of one expert in one slice
  const int r0 = 2 * nb * kTileRows;                                           // first stored row of the task
  const bool halves = kLayer == 2 && sliced && p.routed_halves != 0;
  WeightRows w{shared ? &p.map_w_shared : &p.map_w_routed, e * rows_slice + r0 % rows_slice, sliced ? r0 / rows_slice : 0, 0, 0, halves};
  if (halves) {
    w.row2 = e * rows_slice + (r0 + kTileRows) % rows_slice;
    w.slice2 = (r0 + kTileRows) / rows_slice;
  }
  return w;
}

// layer 2: the counter of a task's expert and what it has to reach
__device__ __forceinline__ const int32_t* sa_done_of(const MoeParams& f, const PlanView& pv, const Tile& tile) {
  return pv.done + (tile.expert == kSharedExpert ? f.layer[0].e_local : tile.expert);
}
template <bool kStaged>
__device__ __forceinline__ int sa_need_of(const MoeParams& f, const Tile& tile) {
  return 4 * f.layer[0].n_blocks * (kStaged && tile.expert != kSharedExpert ? 1 : tile.parts);
}

template <bool kStaged>
struct TaskQueue {
  const MoeParams& f;
  Control* ctl;
  PlanView pv;
  SharedTiles shared;
  bool plan_known, over;
  int small_tiles, small_rows, hit_experts;
  uint32_t claimed;        // lane 0
  uint32_t handed_on;
  __device__ __forceinline__ TaskQueue(const MoeParams& params, Control* control)
      : f(params), ctl(control), pv(plan_view(const_cast<char*>(params.layer[0].plan), params.layer[0].e_local, params.layer[0].num_ranks)),
        shared(params.layer[0].shared_tiles), plan_known(false), over(false), small_tiles(0), small_rows(0), hit_experts(-1), claimed(0),
        handed_on(0) {}
  __device__ __forceinline__ void load_plan() {
    small_tiles = pv.hdr->num_small_tiles;
    small_rows = pv.hdr->small_rows;
    shared = sa_shared_tiles(f.layer[0]);
    plan_known = true;
  }
  __device__ __forceinline__ bool wait_plan(Waiter& waiter) {
    if (plan_known) return true;
    if (kStaged) {
      if (!sa_wait_plan(f.layer[0], waiter)) return false;
    } else {
      chain_wait();
    }
    load_plan();
    return true;
  }
  // which experts are hit, from the route table
  __device__ __forceinline__ void find_hits() {
    const int lane = threadIdx.x & 31;
    if (lane < 16) ctl->hit[lane] = 0u;
    __syncwarp();
    for (int i = lane; i < f.layer[0].num_routes; i += 32) {
      const int64_t id = f.layer[0].topk_idx[i];
      if (id >= 0 && id < f.layer[0].e_local) atomicOr(&ctl->hit[id >> 5], 1u << (id & 31));
    }
    __syncwarp();
    hit_experts = __reduce_add_sync(0xffffffffu, lane < 16 ? __popc(ctl->hit[lane]) : 0);
  }
  // i-th expert (ascending) with a bit in `hit`; whole warp
  __device__ __forceinline__ int hit_expert(int i) const {
    const int lane = threadIdx.x & 31;
    uint32_t word = lane < 16 ? ctl->hit[lane] : 0u;
    const int mine = __popc(word);
    int before = mine;
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, before, d);
      if (lane >= d) before += t;
    }
    before -= mine;
    const int owner = __ffs(__ballot_sync(0xffffffffu, i >= before && i < before + mine)) - 1;
    for (int drop = i - before; drop > 0 && lane == owner; --drop) word &= word - 1;
    return __shfl_sync(0xffffffffu, 32 * lane + __ffs(word) - 1, owner);
  }
  __device__ __forceinline__ void claim() {
    if ((threadIdx.x & 31) == 0) claimed = atomicAdd(&pv.hdr->next_task, 1u);
  }
  // what the claimed number stands for; false when the call is being abandoned
  __device__ __forceinline__ bool decode(Waiter& waiter, QueueSlot* out) {
    int i = static_cast<int>(__shfl_sync(0xffffffffu, claimed, 0));
    for (int layer = 1; layer <= 2; ++layer) {
      const int n_blocks = f.layer[layer - 1].n_blocks, shared_tasks = shared.parts * n_blocks;
      out->layer = layer;
      if (i < shared_tasks) {
        out->nb = i / shared.parts;
        out->tile = shared.at(i - out->nb * shared.parts);
        return true;
      }
      i -= shared_tasks;
      if (kStaged && layer == 1) {
        if (hit_experts < 0) find_hits();
        if (i < hit_experts * n_blocks) {
          const int u = i / n_blocks;
          out->nb = i - u * n_blocks;
          out->tile = Tile{hit_expert(u), 0, shared.m, 0, 0, 1, {0, 0}};
          return true;
        }
        i -= hit_experts * n_blocks;
      } else {
        if (!wait_plan(waiter)) return false;
        if (i < small_tiles * n_blocks) {
          locate_task(pv.tiles, i, n_blocks, &out->tile, &out->nb);
          return true;
        }
        i -= small_tiles * n_blocks;
      }
    }
    out->layer = 0;
    return true;
  }
  // whether all of layer 1 is complete
  __device__ __forceinline__ bool layer1_over() {
    if (!over && plan_known) {
      const int tiles = shared.parts + (kStaged ? hit_experts : small_tiles);
      over = rows_ready(&pv.hdr->layer1_done, 4 * f.layer[0].n_blocks * tiles);
    }
    return over;
  }
  // to the other roles of the CTA
  __device__ __forceinline__ bool hand_on(Waiter& waiter, QueueSlot& t) {
    t.ready = t.layer == 2 && (layer1_over() || rows_ready(sa_done_of(f, pv, t.tile), sa_need_of<kStaged>(f, t.tile))) ? 1 : 0;
    const uint32_t slot = handed_on % kQueue;
    if (!waiter.wait_uniform(smem_u32(&ctl->q_empty[slot]), ((handed_on / kQueue) & 1u) ^ 1u)) return false;
    if ((threadIdx.x & 31) == 0) {
      ctl->slots[slot] = t;
      mbar_arrive(smem_u32(&ctl->q_full[slot]));
    }
    __syncwarp();
    ++handed_on;
    return true;
  }
};

// ------------------------------------------------------------------------------------------------ producer
// One warp in step, one elected lane issues.  Everything that does not change inside a task is computed once per task; the
// K loop only bumps 32-bit coordinates and two pointers, because such a loop runs at instruction latency, not throughput.
// `done` (layer 2 behind layer 1 in the same launch): the token tile is complete when this counter has reached `need`; until then
// as many stages as there are get their weights.  `want`: a barrier that asks the scheduler for the next task.
template <int kLayer, typename L, bool kStaged>
__device__ __forceinline__ void sa_load_task(const UmmaParams& p, const Cta& c, const Tile& tile, int nb, Waiter& waiter, RoleState& st,
                                             const int32_t* done, int need, uint32_t want) {
  const int k_stages = p.k_dim / kTileK;
  const uint32_t full0 = smem_u32(&c.ctl->full[0]), empty0 = smem_u32(&c.ctl->empty[0]);
  const uint32_t sf_full0 = smem_u32(&c.ctl->sf_full[0]);
  const uint32_t a0 = smem_u32(c.a_base), b0 = smem_u32(c.b_base), sf0 = smem_u32(c.sf_base);
  const bool shared = tile.expert == kSharedExpert;
  const bool staged = kLayer == 1 && (shared || kStaged);     // the token tile is rows of the staged tokens
  const int box_sel = (max(tile.n_valid, 1) - 1) >> 4;         // token box: n_valid rounded up to 16 rows
  const uint32_t box_rows = 16u * (box_sel + 1);
  const CUtensorMap* tmap = shared || staged ? &p.map_tok_shared_box[box_sel] : &p.map_tok_routed_box[box_sel];
  const int e = shared ? 0 : tile.expert;
  const WeightRows w = sa_weight_rows<kLayer>(p, tile, nb);
  const int32_t* wsf = (shared ? p.wsf_shared : p.wsf_routed) + (int64_t)e * k_stages * p.rows_per_expert + 2 * nb * kTileRows;
  const int64_t tsf_rows = shared ? p.tsf_rows_shared : p.tsf_rows_routed;
  const int32_t* tsf = (shared ? p.tsf_shared : p.tsf_routed) + (int64_t)tile.sf_chunk * kChunkRows;
  const uint32_t w_tx = (shared ? 2 * kTileRows * kTileK : kTileRows * kTileK) + (kLayer == 1 ? 0 : 1024);   // packed FP4 counts its global bytes
  const uint32_t t_tx = box_rows * kTileK + (staged ? 0 : 512);     // scales of staged tokens come from the scale arranger
  auto load_weights = [&](uint32_t stage, int k0, const int32_t* sf) {
    const uint32_t bar = full0 + 8 * stage;
    if (kLayer == 1) {
      tma_load_5d(a0 + stage * L::kABytes, w.map, k0, 0, w.row / 16, 0, w.slice, bar);
    } else {
      tma_load_3d(a0 + stage * L::kABytes, w.map, k0, w.row, w.slice, bar);
      if (w.halves) tma_load_3d(a0 + stage * L::kABytes + kTileRows * kTileK, w.map, k0, w.row2, w.slice2, bar);
      bulk_load(sf0 + stage * L::kSfBytes, sf, 1024, bar);       // two chunks already in tensor-memory order
    }
  };
  int ahead = 0;                                                 // stages whose weights have been requested
  if (kLayer == 2 && done != nullptr) {
    if (!rows_ready(done, need)) {
      uint32_t stage = st.stage, phase = st.phase;
      const int most = min(static_cast<int>(c.num_stages), k_stages);
      for (; ahead < most; ++ahead) {
        if (!waiter.wait_uniform(empty0 + 8 * stage, phase ^ 1u)) { st.ok = false; return; }
        if (elect_one()) {
          mbar_expect_tx_only(full0 + 8 * stage, w_tx);
          load_weights(stage, ahead * kTileK, wsf + (int64_t)ahead * p.rows_per_expert);
        }
        __syncwarp();
        if (++stage == c.num_stages) { stage = 0; phase ^= 1u; }
      }
      for (uint32_t spin = 0; !rows_ready(done, need); ++spin) {
        if ((spin & 63u) == 63u && __any_sync(0xffffffffu, waiter.abandoned())) { st.ok = false; return; }
        __nanosleep(40);
      }
    }
  }
  const int want_at = max(k_stages - 8, 0);
  int k0 = 0;
  for (int kb = 0; kb < k_stages; ++kb, k0 += kTileK, wsf += p.rows_per_expert, tsf += tsf_rows) {
    if ((kLayer == 1 || kb >= ahead) && !waiter.wait_uniform(empty0 + 8 * st.stage, st.phase ^ 1u)) { st.ok = false; return; }
    const uint32_t bar = full0 + 8 * st.stage;
    if (elect_one()) {
      if (want != 0 && kb == want_at) mbar_arrive(want);
      if (kLayer == 1) {
        // scales of the 256 stored rows, rearranged by the scale arranger: their own barrier, first in the queue
        mbar_expect_tx(sf_full0 + 8 * st.stage, 1024);
        bulk_load(sf0 + st.stage * L::kSfBytes, wsf, 1024, sf_full0 + 8 * st.stage);
      }
      if (kLayer == 2 && kb < ahead) {
        mbar_expect_tx(bar, t_tx);
      } else {
        mbar_expect_tx(bar, w_tx + t_tx);
        load_weights(st.stage, k0, wsf);
      }
      tma_load_2d(b0 + st.stage * c.b_bytes, tmap, k0, tile.row0, bar);
      if (!staged) bulk_load(sf0 + st.stage * L::kSfBytes + 2 * 512, tsf, 512, bar);
    }
    __syncwarp();
    if (++st.stage == c.num_stages) { st.stage = 0; st.phase ^= 1u; }
  }
}

// One layer in the launch.
template <int kLayer, typename L>
__device__ __forceinline__ void sa_producer(const UmmaParams& p, const Cta& c, TaskWalk<kLayer> walk, Waiter& waiter, RoleState& st) {
  while (st.ok && walk.next(waiter)) sa_load_task<kLayer, L, false>(p, c, walk.tile, walk.nb, waiter, st, nullptr, 0, 0u);
}

// Both layers.  The producer asks for the next task eight stages before the end of the one before, 3 us at HBM speed, and not
// before it knows its own rows to be complete: a CTA that waits must not hold back another task.
template <typename L, bool kStaged>
__device__ __forceinline__ void sa_producer_both(const MoeParams& f, const Cta& c, TaskFeed<false> feed, Waiter& waiter, RoleState& st) {
  const PlanView pv = plan_view(const_cast<char*>(f.layer[0].plan), f.layer[0].e_local, f.layer[0].num_ranks);
  const uint32_t want = smem_u32(&c.ctl->q_want);
  while (st.ok && feed.next(waiter)) {
    if (feed.layer == 1) sa_load_task<1, L, kStaged>(f.layer[0], c, feed.tile, feed.nb, waiter, st, nullptr, 0, want);
    else sa_load_task<2, L, false>(f.layer[1], c, feed.tile, feed.nb, waiter, st, feed.ready ? nullptr : sa_done_of(f, pv, feed.tile),
                                   sa_need_of<kStaged>(f, feed.tile), want);
  }
  if constexpr (!kStaged) {
    if (!st.ok || c.ctl->next_rows == 0) return;
    // before another stage layout: every stage has been read, and the barriers have seen all that will arrive on them
    for (uint32_t i = 0; i < c.num_stages; ++i) {
      if (!waiter.wait_uniform(smem_u32(&c.ctl->empty[st.stage]), st.phase ^ 1u)) return;
      if (++st.stage == c.num_stages) { st.stage = 0; st.phase ^= 1u; }
    }
  }
}

// `rows`: the token slots.  A launch that started before the plan was complete, with the shared expert's tasks, may find larger tiles in it.
// The roles then leave as if there were no more tasks, and start over with slots of that size and with the task just claimed.
template <bool kStaged>
__device__ __forceinline__ void sa_scheduler(const Cta& c, TaskQueue<kStaged>& queue, int rows, Waiter& waiter) {
  queue.handed_on = 0;
  for (uint32_t n = 0;; ++n) {
    QueueSlot t;
    if (!queue.decode(waiter, &t)) return;
    if (!kStaged && t.layer != 0 && queue.small_rows > rows) {
      if ((threadIdx.x & 31) == 0) c.ctl->next_rows = queue.small_rows;
      t.layer = 0;
    }
    if (!queue.hand_on(waiter, t) || t.layer == 0) return;
    if (!waiter.wait_uniform(smem_u32(&c.ctl->q_want), n & 1u)) return;
    queue.claim();
  }
}

// ------------------------------------------------------------------------------------------------ MMA issuers
// Layer 1: one warp rewrites each stage's weight scales from stored order into tensor-memory order while the stage's tile
// copies are still in flight.  The stored W13 scales follow the stored row order (gate/up interleaved by 8, then the 4x32
// transpose inside each 128-row block); the accumulators want the scales of 128 gate (h = 0) and 128 up (h = 1) channels.
// On the MMA warps' path this work was a third of a stage's issue time (about 230 of 700 clk, and a stage is 580 clk of
// HBM time at the clock a power-capped B200 runs this kernel at).
// (Layer 2's scales are stored in tensor-memory order; in a launch of both layers no task of layer 1 follows one of layer 2.)
template <typename L, bool kStaged, typename Walk>
__device__ __forceinline__ void sa_arrange_scales(const Cta& c, Walk walk, Waiter& waiter, RoleState& st) {
  const int lane = threadIdx.x & 31;
  const uint32_t sf_full0 = smem_u32(&c.ctl->sf_full[0]), sf_ready0 = smem_u32(&c.ctl->sf_ready[0]);
  int src[8];                                    // source word of the 8 destination words this lane writes
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int h = t >> 2;
    const int q = lane + 32 * (t & 3);           // destination position inside the tile's 128-word block
    const int m = 32 * (q & 3) + (q >> 2);       // channel of the tile that position serves
    const int r = 16 * ((m & 63) >> 3) + 8 * h + (m & 7);   // stored row inside its 128-row block
    src[t] = 128 * (m >> 6) + 4 * (r & 31) + (r >> 5);
  }
  if (!kStaged) asm volatile("fence.acq_rel.gpu;" ::: "memory");      // nothing of the rows staged before is left in the L1
  for_each_task(walk, waiter, st, [&](auto layer, const UmmaParams& p) {
    if constexpr (decltype(layer)::value == 1) {
    const int k_stages = p.k_dim / kTileK;
    // The scales of staged tokens are gathered here, word kb of the staged scale rows (chunk position 4 (i % 32) + i / 32
    // for token i), two stages ahead: such tiles need no placement, only the staging.  Through the L1, which has a row's next 31 words then
    // (from the L2 each: 7 tokens 131 -> 136 us).
    const bool staged = walk.tile.expert == kSharedExpert || kStaged;
    const int32_t* x_sf = p.x_sf + (int64_t)(walk.tile.row0 + lane) * k_stages;
    uint32_t ahead[2][4] = {};
    auto gather = [&](uint32_t (&w)[4], int kb) {
#pragma unroll
      for (int a = 0; a < 4; ++a)
        w[a] = staged && kb < k_stages && lane + 32 * a < walk.tile.n_valid ? __ldca(x_sf + 32 * a * k_stages + kb) : 0u;
    };
    gather(ahead[0], 0);
    gather(ahead[1], 1);
    for (int kb = 0; kb < k_stages; ++kb) {
      // the stage's scales have landed, which also says that the MMAs which read the previous ones have retired
      if (!waiter.wait_uniform(sf_full0 + 8 * st.stage, st.phase)) { st.ok = false; break; }
      uint32_t* area = reinterpret_cast<uint32_t*>(c.sf_base + st.stage * L::kSfBytes);
      uint32_t v[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) v[t] = area[src[t]];
      __syncwarp();
#pragma unroll
      for (int t = 0; t < 8; ++t) area[lane + 32 * t] = v[t];
      if (staged) {
        *reinterpret_cast<uint4*>(area + 2 * 128 + 4 * lane) = make_uint4(ahead[0][0], ahead[0][1], ahead[0][2], ahead[0][3]);
#pragma unroll
        for (int a = 0; a < 4; ++a) ahead[0][a] = ahead[1][a];
        gather(ahead[1], kb + 2);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes -> visible to tcgen05.cp
      __syncwarp();
      if (elect_one()) mbar_arrive(sf_ready0 + 8 * st.stage);
      __syncwarp();
      if (++st.stage == c.num_stages) { st.stage = 0; st.phase ^= 1u; }
    }
    }
  });
}

// Two warps, one per weight tile / accumulator (h = 0, 1).  The whole warp walks the loop so that loop state stays
// warp-uniform; one elected lane issues.  Each warp copies the scales it needs into its own TMEM columns, so no
// ordering between the two warps' tensor-core instructions is needed.
template <typename L, typename Walk>
__device__ __forceinline__ void sa_mma(const Cta& c, Walk walk, Waiter& waiter, RoleState& st, int h) {
  const uint32_t full0 = smem_u32(&c.ctl->full[0]), sf_ready0 = smem_u32(&c.ctl->sf_ready[0]);
  const uint32_t empty0 = smem_u32(&c.ctl->empty[0]);
  const uint64_t sw128_hi = desc_hi_sw128();
  const uint64_t sf_hi = desc_hi_sf(128);
  const uint32_t a_lo0 = ((smem_u32(c.a_base) & 0x3FFFFu) >> 4) + h * (kTileRows * kTileK >> 4);
  const uint32_t b_lo0 = (smem_u32(c.b_base) & 0x3FFFFu) >> 4;
  const uint32_t sf_lo0 = (smem_u32(c.sf_base) & 0x3FFFFu) >> 4;
  const uint32_t sfa_col = c.tmem_base + L::kSfCol + 4 * h;
  const uint32_t sfb_col = c.tmem_base + L::kSfCol + 8 + 4 * h;
  for_each_task(walk, waiter, st, [&](auto layer, const UmmaParams& p) {
    constexpr int kLayer = decltype(layer)::value;
    const int k_stages = p.k_dim / kTileK;
    const Tile tile = walk.tile;
    const bool shared = tile.expert == kSharedExpert;
    const uint32_t acc_stage = st.it & 1u, acc_phase = (st.it >> 1) & 1u;
    if (!waiter.wait_uniform(smem_u32(&c.ctl->tmem_empty[acc_stage]), acc_phase ^ 1u)) { st.ok = false; return; }
    tc_fence_after();
    const uint32_t n = static_cast<uint32_t>((tile.n_valid + 15) & ~15);
    const uint32_t idesc0 = make_idesc(shared ? 0u : 5u, 0u, n, 0);
    const uint32_t d = c.tmem_base + acc_stage * L::kAccCols + h * L::kNCap;
    for (int kb = 0; kb < k_stages; ++kb) {
      if (kLayer == 1 && !waiter.wait_uniform(sf_ready0 + 8 * st.stage, st.phase)) { st.ok = false; break; }
      if (!waiter.wait_uniform(full0 + 8 * st.stage, st.phase)) { st.ok = false; break; }
      const uint32_t a_lo = a_lo0 + st.stage * (L::kABytes >> 4);
      const uint32_t b_lo = b_lo0 + st.stage * (c.b_bytes >> 4);
      const uint32_t sf_lo = sf_lo0 + st.stage * (L::kSfBytes >> 4);
      if (elect_one()) {
        tc_cp_sf(sfa_col, sf_hi | (sf_lo + 32 * h));
        tc_cp_sf(sfb_col, sf_hi | (sf_lo + 64));
#pragma unroll
        for (int k = 0; k < kTileK / 32; ++k)
          tc_mma(d, sw128_hi | (a_lo + 2 * k), sw128_hi | (b_lo + 2 * k),
                 idesc0 + k * ((1u << 4) | (1u << 29)),               // scale byte k of both operands
                 sfa_col, sfb_col, (kb | k) != 0 ? 1u : 0u);
        tc_commit(empty0 + 8 * st.stage);            // shared memory of this stage is free once these MMAs retire
      }
      __syncwarp();
      if (++st.stage == c.num_stages) { st.stage = 0; st.phase ^= 1u; }
    }
    if (st.ok && elect_one()) tc_commit(smem_u32(&c.ctl->tmem_full[acc_stage]));
    __syncwarp();
    ++st.it;
  });
}

// ------------------------------------------------------------------------------------------------ epilogue
// Four warps; a thread owns one weight row (accumulator lane), the columns are the tile's tokens.
// kFused (layer 2, EP > 1): every output row goes to the rank its token came from; compiled as kernels of its own so
// that the single-destination epilogue of the other cases keeps its shorter inner loop.
// Tiles of at most this many rows leave column by column in a rolled loop: the unrolled batches of 16 columns are 16 KB of
// instructions, which a call that has just streamed its weights through the L2 fetches from DRAM line by line (9 us at one
// token), and with a token or two per expert most of their columns are padding.
constexpr int kThinRows = 8;

// GEMM1 epilogue of one column: this warp's 32 channels of one token, in a rolled loop
__device__ __forceinline__ int sa_l1_column(const UmmaParams& p, uint32_t taddr, uint32_t up_offset, float wt, uint8_t* out) {
  const uint32_t g = tc_ld1(taddr), u = tc_ld1(taddr + up_offset);
  tc_ld_wait();
  const float a = p.fast_math != 0 ? swiglu_act_t<true>(__uint_as_float(g), __uint_as_float(u), wt, p.clamp)
                                   : swiglu_act_t<false>(__uint_as_float(g), __uint_as_float(u), wt, p.clamp);
  const int sf_exp = ue8m0_exp_of_amax(warp_max_nonneg(fabsf(a)));
  *out = float_to_e4m3(__fmul_rn(a, ue8m0_inv(sf_exp)));
  return sf_exp;
}

// GEMM1 epilogue of a routed task whose columns are the staged tokens: every pool row of the expert takes the column of its
// token.
template <typename L>
__device__ __forceinline__ bool sa_epilogue_staged(const UmmaParams& p, const Cta& c, const Tile& tile, int nb, Waiter& waiter, RoleState& st) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = warp & 3;
  const uint32_t acc_stage = st.it & 1u, acc_phase = (st.it >> 1) & 1u;
  const PlanView pv = plan_view(const_cast<char*>(p.plan), p.e_local, p.num_ranks);
  const int n = pv.expert_total[tile.expert];
  const Tile first = pv.tiles[pv.expert_tile_off[tile.expert]];
  auto token_of = [&](int r) { return r < n ? p.sorted_route[p.pool_dst[first.row0 + r]] / p.topk : 0; };
  int token = token_of(lane);
  float weight = lane < n ? p.pool_w[first.row0 + lane] : 0.f;
  if (!waiter.wait_warp(smem_u32(&c.ctl->tmem_full[acc_stage]), acc_phase)) return false;
  tc_fence_after();
  const uint32_t d0 = c.tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc_stage * L::kAccCols;
  uint8_t* out = p.act_routed + (int64_t)first.row0 * p.inter + nb * kTileRows + q * 32 + lane;
  // scale byte of (row r, channel group nb*4+q): word nb of the row's chunk (one per 16 rows), byte q
  uint8_t* sf_out = p.act_sf_routed + ((int64_t)nb * p.act_sf_rows_routed + (int64_t)first.sf_chunk * kChunkRows) * 4 + q;
#pragma unroll 1
  for (int r = 0; r < n; ++r, out += p.inter) {
    if (r > 0 && (r & 31) == 0) {                    // more than 32 rows: tokens that name the expert several times
      token = token_of(r + lane);
      weight = r + lane < n ? p.pool_w[first.row0 + r + lane] : 0.f;
    }
    const int j = __shfl_sync(0xffffffffu, token, r & 31);
    const int sf_exp = sa_l1_column(p, d0 + j, L::kNCap, __shfl_sync(0xffffffffu, weight, r & 31), out);
    if (lane == 0) sf_out[((r / kStagedTokens) * kChunkRows + chunk_pos(r % kStagedTokens)) * 4] = static_cast<uint8_t>(sf_exp);
  }
  tc_fence_before();
  mbar_arrive(smem_u32(&c.ctl->tmem_empty[acc_stage]));
  sa_publish(pv, tile.expert);
  return true;
}

template <typename L, bool kFused, bool kStaged, typename Walk>
__device__ __forceinline__ void sa_epilogue(const Cta& c, Walk walk, bool plan_known, Waiter& waiter, RoleState& st) {
  Control* ctl = c.ctl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = warp & 3;                     // TMEM lane quadrant this warp may read
  const uint32_t lane_sel = static_cast<uint32_t>(q * 32) << 16;
  for_each_task(walk, waiter, st, [&](auto layer, const UmmaParams& p) {
    constexpr int kLayer = decltype(layer)::value;
    const Tile tile = walk.tile;
    const int nb = walk.nb;
    const bool shared = tile.expert == kSharedExpert;
    if (!plan_known && !shared && !(kStaged && kLayer == 2)) {       // (the scheduler knew it before it handed on a task of layer 2)
      if (kStaged) {
        if (!sa_wait_plan(p, waiter)) { st.ok = false; return; }
      } else {
        chain_wait();
      }
      plan_known = true;
    }
    if (kStaged && kLayer == 1 && !shared) {
      if (!sa_epilogue_staged<L>(p, c, tile, nb, waiter, st)) { st.ok = false; return; }
      ++st.it;
      return;
    }
    const uint32_t acc_stage = st.it & 1u, acc_phase = (st.it >> 1) & 1u;
    // Per-token side data of the tile (top-k weight / destination row), one coalesced load per 32 tokens issued
    // before the accumulator is awaited; tokens read it by shuffle.
    float wv[4] = {1.0f, 1.0f, 1.0f, 1.0f};
    int dv[4] = {0, 0, 0, 0};
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      const int i = 32 * cc + lane;
      if (i < tile.n_valid) {
        if (kLayer == 1) { if (!shared) wv[cc] = __ldcg(p.pool_w + tile.row0 + i); }
        else if (!kFused) dv[cc] = shared ? tile.row0 + i : (kStaged ? p.pool_dst[tile.row0 + i] : __ldcg(p.pool_dst + tile.row0 + i));
        else if (shared) dv[cc] = static_cast<int>((32u << kOutSlotShift) | static_cast<uint32_t>(tile.row0 + i));
        else {
          const int r = __ldcg(p.pool_dst + tile.row0 + i);      // receive-order row
          int sr = 0;
          while (sr + 1 < p.num_ranks && r >= ctl->rank_off[sr + 1]) ++sr;
          dv[cc] = static_cast<int>((static_cast<uint32_t>(sr) << kOutSlotShift) |
                                    static_cast<uint32_t>(ctl->home_base[sr] + r - ctl->rank_off[sr]));
        }
      }
    }
    if (!waiter.wait_warp(smem_u32(&ctl->tmem_full[acc_stage]), acc_phase)) { st.ok = false; return; }
    tc_fence_after();
    const uint32_t d0 = c.tmem_base + lane_sel + acc_stage * L::kAccCols;
    const int n16 = (tile.n_valid + 15) & ~15;
    if (kLayer == 1) {
      const int row = nb * kTileRows + q * 32 + lane;       // channel
      uint8_t* act = shared ? p.act_shared : p.act_routed;
      uint8_t* act_sf = shared ? p.act_sf_shared : p.act_sf_routed;
      const int64_t sf_rows = shared ? p.act_sf_rows_shared : p.act_sf_rows_routed;
      // scale byte of (token i, channel group nb*4+q): word nb of the chunk row, byte q
      uint8_t* sf_out = act_sf + ((int64_t)nb * sf_rows + (int64_t)tile.sf_chunk * kChunkRows) * 4 + q;
      uint8_t* act_col = act + (int64_t)tile.row0 * p.inter + row;
      if (tile.n_valid <= kThinRows) {
#pragma unroll 1
        for (int i = 0; i < tile.n_valid; ++i, act_col += p.inter) {
          const int sf_exp = sa_l1_column(p, d0 + i, L::kNCap, __shfl_sync(0xffffffffu, wv[0], i), act_col);
          if (lane == 0) sf_out[chunk_pos(i) * 4] = static_cast<uint8_t>(sf_exp);
        }
      } else for (int i0 = 0; i0 < n16; i0 += 16) {
        uint32_t g[16], u[16];
        tc_ld16(d0 + i0, g);
        tc_ld16(d0 + L::kNCap + i0, u);
        tc_ld_wait();
        const int cc = i0 >> 5;
        const float wcur = cc == 0 ? wv[0] : (cc == 1 ? wv[1] : (cc == 2 ? wv[2] : wv[3]));
        int my_sf = 0;
        // branch-free over the 16 columns so that their dependency chains interleave (the fast-math choice is made
        // once per batch, not per element); padding columns compute garbage that is never stored
        auto batch = [&](auto fast) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float wt = __shfl_sync(0xffffffffu, wcur, (i0 & 16) + j);
            const float a = swiglu_act_t<decltype(fast)::value>(__uint_as_float(g[j]), __uint_as_float(u[j]), wt, p.clamp);
            const float amax = warp_max_nonneg(fabsf(a));
            const int sf_exp = ue8m0_exp_of_amax(amax);
            g[j] = float_to_e4m3(__fmul_rn(a, ue8m0_inv(sf_exp)));
            if (lane == j) my_sf = sf_exp;
          }
        };
        if (p.fast_math != 0) batch(std::true_type{});
        else batch(std::false_type{});
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (i0 + j < tile.n_valid) act_col[(int64_t)(i0 + j) * p.inter] = static_cast<uint8_t>(g[j]);
        if (lane < 16 && i0 + lane < tile.n_valid)
          sf_out[chunk_pos(i0 + lane) * 4] = static_cast<uint8_t>(my_sf);
      }
    } else if (!kFused && tile.n_valid <= kThinRows) {
      __nv_bfloat16* out = (shared ? p.shared_out : p.ret) + nb * 2 * kTileRows + q * 32 + lane;
#pragma unroll 1
      for (int i = 0; i < tile.n_valid; ++i) {
        const uint32_t v0 = tc_ld1(d0 + i), v1 = tc_ld1(d0 + L::kNCap + i);
        tc_ld_wait();
        __nv_bfloat16* o = out + (int64_t)__shfl_sync(0xffffffffu, dv[0], i) * p.hidden;
        o[0] = __float2bfloat16_rn(__uint_as_float(v0));
        o[kTileRows] = __float2bfloat16_rn(__uint_as_float(v1));
      }
    } else if (!kFused) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = nb * 2 * kTileRows + h * kTileRows + q * 32 + lane;     // output feature
        __nv_bfloat16* out = (shared ? p.shared_out : p.ret) + row;
        for (int i0 = 0; i0 < n16; i0 += 16) {
          uint32_t v[16];
          tc_ld16(d0 + h * L::kNCap + i0, v);
          tc_ld_wait();
          const int cc = i0 >> 5;
          const int dcur = cc == 0 ? dv[0] : (cc == 1 ? dv[1] : (cc == 2 ? dv[2] : dv[3]));
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int dst = __shfl_sync(0xffffffffu, dcur, (i0 & 16) + j);
            if (i0 + j < tile.n_valid) out[(int64_t)dst * p.hidden] = __float2bfloat16_rn(__uint_as_float(v[j]));
          }
        }
      }
    } else {
      // one destination per token: resolve the 16 row pointers of a batch once, use them for both weight blocks
      const int row0 = nb * 2 * kTileRows + q * 32 + lane;                      // output feature of weight block 0
      for (int i0 = 0; i0 < n16; i0 += 16) {
        uint32_t v0[16], v1[16];
        tc_ld16(d0 + i0, v0);
        tc_ld16(d0 + L::kNCap + i0, v1);
        const int cc = i0 >> 5;
        const int dcur = cc == 0 ? dv[0] : (cc == 1 ? dv[1] : (cc == 2 ? dv[2] : dv[3]));
        tc_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const uint32_t dst = static_cast<uint32_t>(__shfl_sync(0xffffffffu, dcur, (i0 & 16) + j));
          if (i0 + j < tile.n_valid) {
            __nv_bfloat16* out = ctl->out_base[dst >> kOutSlotShift] +
                                 (int64_t)(dst & ((1u << kOutSlotShift) - 1u)) * p.hidden + row0;
            out[0] = __float2bfloat16_rn(__uint_as_float(v0[j]));
            out[kTileRows] = __float2bfloat16_rn(__uint_as_float(v1[j]));
          }
        }
      }
    }
    tc_fence_before();
    mbar_arrive(smem_u32(&ctl->tmem_empty[acc_stage]));
    if (Walk::kBoth && kLayer == 1)
      sa_publish(plan_view(const_cast<char*>(p.plan), p.e_local, p.num_ranks), shared ? p.e_local : tile.expert);
    ++st.it;
  });
}

// ------------------------------------------------------------------------------------------------ set-up / teardown
__device__ __forceinline__ uint8_t* sa_align(uint8_t* smem_raw) {
  return smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
}

// the stages behind the control block, for tiles of at most `tile_rows` rows
template <typename L>
__device__ __forceinline__ Cta sa_carve(uint8_t* smem, int tile_rows, int max_stages) {
  Cta c;
  int stages = L::stages(tile_rows);
  if (max_stages > 0 && max_stages < stages) stages = max_stages;
  c.num_stages = static_cast<uint32_t>(stages);
  c.b_bytes = static_cast<uint32_t>(tile_rows * kTileK);
  c.ctl = reinterpret_cast<Control*>(smem);
  c.a_base = smem + 1024;
  c.b_base = c.a_base + stages * L::kABytes;
  c.sf_base = c.b_base + stages * c.b_bytes;
  c.tmem_base = 0;
  return c;
}

// rows of the largest tile of the call
__device__ __forceinline__ int sa_tile_rows(const UmmaParams& p) {
  return p.tile_rows > 0 ? p.tile_rows : max(16, min(kSmallTileRows, plan_view(const_cast<char*>(p.plan), p.e_local, p.num_ranks).hdr->small_rows));
}

// one thread; kAgain: the barriers have been in use, and nothing will arrive on them any more
template <typename L, bool kBoth, bool kAgain>
__device__ __forceinline__ void sa_barriers(Control* ctl) {
  auto init = [](uint64_t& bar, uint32_t count) {
    if (kAgain) mbar_inval(smem_u32(&bar));
    mbar_init(smem_u32(&bar), count);
  };
  for (int i = 0; i < L::kMaxStages; ++i) {
    init(ctl->full[i], 1);
    init(ctl->empty[i], 2);          // both MMA warps release a stage
    init(ctl->sf_full[i], 1);
    init(ctl->sf_ready[i], 1);
  }
  for (int i = 0; i < 2; ++i) {
    init(ctl->tmem_full[i], 2);      // both MMA warps finish an accumulator pair
    init(ctl->tmem_empty[i], 128);
  }
  if (kBoth)
    for (int i = 0; i < kQueue; ++i) {
      init(ctl->q_full[i], 1);
      init(ctl->q_empty[i], 8);      // producer, MMA, epilogue and scale warps
    }
  if (kBoth) init(ctl->q_want, 1);
  ctl->next_rows = 0;
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// barriers and tensor memory: touches only this CTA's own shared / tensor memory
template <typename L, bool kBoth>
__device__ __forceinline__ void sa_setup(Control* ctl) {
  if (threadIdx.x == 0) {
    ctl->abort_flag = 0;
    sa_barriers<L, kBoth, false>(ctl);
  }
  if ((threadIdx.x >> 5) == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
}

__device__ __forceinline__ void sa_teardown(Control* ctl, uint32_t tmem_base) {
  __syncwarp();
  if (ctl->abort_flag != 0) {
    // abandoned call: give copies that are still in flight time to land in this CTA's shared memory before it exits
    const uint64_t t0 = global_timer();
    while (global_timer() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if ((threadIdx.x >> 5) == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// One layer per launch.
template <int kLayer, bool kFused>
__global__ void __launch_bounds__(kThreads, 1) umma_kernel(const __grid_constant__ UmmaParams p) {
  static_assert(!kFused || kLayer == 2, "only GEMM2 writes rows back");
  using L = Shape<kLayer>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = sa_align(smem_raw);
  Control* ctl = reinterpret_cast<Control*>(smem);
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);   // warp-uniform for the compiler too
  chain_release();
  sa_setup<L, false>(ctl);
  // Everything above touches only this CTA's own shared and tensor memory, so it may run while the kernel before this
  // one in the stream is still running.
  if (warp == 0 && elect_one()) {
    prefetch_map(&p.map_w_routed);
    prefetch_map(&p.map_w_shared);
  }
  chain_wait();
  if (kFused) {
    if (threadIdx.x == 0) ctl->out_base[32] = p.shared_out;
    const int t = threadIdx.x - 32;
    if (t >= 0 && t < p.num_ranks) {
      ctl->out_base[t] = p.ep_ret_recv[t];
      int b = 0;
      for (int d = 0; d < p.ep_me; ++d) b += p.ep_totals[t * 32 + d];
      ctl->home_base[t] = b;
    }
    if (threadIdx.x == 64) {
      int run = 0;
      for (int sr = 0; sr < p.num_ranks; ++sr) { ctl->rank_off[sr] = run; run += p.ep_totals[sr * 32 + p.ep_me]; }
      ctl->rank_off[p.num_ranks] = run;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  Cta c = sa_carve<L>(smem, sa_tile_rows(p), p.max_stages);
  c.tmem_base = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
  const TaskWalk<kLayer> walk(p, true);
  Waiter waiter{&ctl->abort_flag, p.status, global_timer() + static_cast<uint64_t>(p.timeout_ns), kLayer, warp};
  RoleState st;
  if (warp == 0) {
    sa_producer<kLayer, L>(p, c, walk, waiter, st);
  } else if (warp == 1 || warp == 6) {
    sa_mma<L>(c, walk, waiter, st, warp == 1 ? 0 : 1);
  } else if (warp == 7) {
    if constexpr (kLayer == 1) sa_arrange_scales<L, false>(c, walk, waiter, st);
  } else {
    sa_epilogue<L, kFused, false>(c, walk, true, waiter, st);
  }
  sa_teardown(ctl, c.tmem_base);
}

// Both layers of a single-GPU call, for the experts that do not run on CTA pairs.  kStaged: calls of at most kStagedTokens tokens.
template <bool kStaged>
__global__ void __launch_bounds__(both_threads(kStaged), 1) moe_kernel(const __grid_constant__ MoeParams f) {
  using L = Shape<1>;
  const UmmaParams& p = f.layer[0];
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = sa_align(smem_raw);
  Control* ctl = reinterpret_cast<Control*>(smem);
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const PlanView pv = plan_view(const_cast<char*>(p.plan), p.e_local, p.num_ranks);
  chain_release();
  const bool behind_pairs = !kStaged && p.behind_pairs != 0;
  if (behind_pairs && !chain_opened(pv.pairs_open)) chain_wait();
  if (behind_pairs && p.shared_tiles.parts == 0 && pv.hdr->num_small_tiles == 0) {      // every expert ran on the pairs in front
    chain_wait();
    return;
  }
  // The first claim may come this early: the counters were zero before the last call's combine let anything start.
  TaskQueue<kStaged> queue(f, ctl);
  if (warp == 8) queue.claim();
  sa_setup<L, true>(ctl);
  // Everything above touches only this CTA's own shared and tensor memory, and a plan that is complete.  The launch of a call
  // without pair tiles goes on with the shared expert: it is let start by the route ordering's blocks once they have seen the
  // staging complete.  One that orders the routes itself follows the staging, whose predecessors may be anything: not even
  // weights are read ahead of the wait.
  if (warp == 0 && elect_one()) {
    prefetch_map(&p.map_w_routed);
    prefetch_map(&p.map_w_shared);
  }
  const bool route_here = kStaged && p.route_here, plan_ready = !p.early && !route_here;
  if ((!p.early || route_here) && !behind_pairs) chain_wait();
  if (plan_ready) queue.load_plan();
  int rows = sa_tile_rows(p);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
  Waiter waiter{&ctl->abort_flag, p.status, global_timer() + static_cast<uint64_t>(p.timeout_ns), kStatusBothLayers, warp};
  for (;;) {
    Cta c = sa_carve<L>(smem, rows, p.max_stages);
    c.tmem_base = tmem_base;
    RoleState st;
    if (warp == 0) {
      sa_producer_both<L, kStaged>(f, c, TaskFeed<false>(f, ctl), waiter, st);
    } else if (warp == 1 || warp == 6) {
      sa_mma<L>(c, TaskFeed<false>(f, ctl), waiter, st, warp == 1 ? 0 : 1);
    } else if (warp == 7) {
      sa_arrange_scales<L, kStaged>(c, TaskFeed<false>(f, ctl), waiter, st);
    } else if (warp == 8) {
      sa_scheduler<kStaged>(c, queue, rows, waiter);
    } else if (warp == 9) {
      if (route_here && sa_wait_plan(p, waiter)) sa_place(p);
    } else {
      const int t = static_cast<int>(threadIdx.x) - 64;
      if (route_here && sa_claim_route(p, ctl, t))
        sa_route(p, *reinterpret_cast<RouteScratch*>(c.sf_base + c.num_stages * L::kSfBytes), t);
      sa_epilogue<L, false, kStaged>(c, TaskFeed<true>(f, ctl), plan_ready, waiter, st);
    }
    if (kStaged) break;
    // Another stage layout, once: behind this barrier no role waits, copies or multiplies, and the accumulators have been read.
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const int next = ctl->abort_flag != 0 ? 0 : ctl->next_rows;
    if (next == 0) break;
    rows = next;
    __syncthreads();                                   // everyone has read it
    if (threadIdx.x == 0) sa_barriers<L, true, true>(ctl);
    __syncthreads();
  }
  chain_wait();       // a CTA that has not waited yet must not end before what precedes the launch
  sa_teardown(ctl, tmem_base);
}

// ---------------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
constexpr int kMaxDevices = 64;
int g_num_sms[kMaxDevices] = {};   // per device, 0 = mmoe_prepare() has not run there
int g_tune_stages = 0;             // 0: every stage that fits
int g_orientation = 0;             // 0: chosen per expert, 1: weights-as-A, 2 and 3: tokens-as-A on CTA pairs

int current_device() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
  return dev;
}

// W13 (stored rows [g0..7, u0..7, g8..15, ...]): 5-D map [slices, gate/up, groups of 16 rows, row in group of 8, K];
// a box of 8 x 16 x 2 is the 128 gate rows followed by the 128 up rows of 128 channels
int make_w13_map(CUtensorMap* map, bool fp4, const void* base, uint64_t k_elems, uint64_t rows_total, int64_t slice_stride) {
  const uint64_t row_bytes = fp4 ? k_elems / 2 : k_elems;
  const uint64_t slices = slice_stride > 0 ? 2 : 1;
  const uint64_t rows = rows_total / slices;
  const cuuint64_t dims[5] = {k_elems, 8, rows / 16, 2, slices};
  const cuuint64_t strides[4] = {row_bytes, 16 * row_bytes, 8 * row_bytes,
                                 slice_stride > 0 ? static_cast<uint64_t>(slice_stride) : rows * row_bytes};
  const cuuint32_t box[5] = {kTileK, 8, 16, 2, 1};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const CUresult r = g_encode(map, fp4 ? CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B : CU_TENSOR_MAP_DATA_TYPE_UINT8, 5,
                              const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

template <typename Kernel>
cudaError_t prepare_one(Kernel* kernel, int smem_bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
}

template <int kLayer, bool kFused>
cudaError_t launch_layer(UmmaParams& p, cudaStream_t s) {
  p.max_stages = g_tune_stages;
  return launch_chained(umma_kernel<kLayer, kFused>, dim3(tc_num_sms()), dim3(kThreads), Shape<kLayer>::kSmemBytes, s, p);
}

template <bool kStaged>
cudaError_t launch_both(MoeParams& p, cudaStream_t s) {
  p.layer[0].max_stages = g_tune_stages;
  return launch_chained(moe_kernel<kStaged>, dim3(tc_num_sms()), dim3(both_threads(kStaged)), Shape<1>::kSmemBytes, s, p);
}

// ---------------------------------------------------------------------------------------------------------------
// Launch parameters that depend only on (workspace, weights, geometry) -- above all the encoded tensor maps, 32 for the
// weights-as-A kernels and 28 for the pairs -- are built once and kept: a serving engine calls its layers with the same buffers
// thousands of times.  What changes per call (tile selection, options, peers) is patched into a copy.  The reference keeps the
// same kind of record per validated call (backend/frontend.py:650-754).
//
// A model's layers share one workspace: the parameters of a second layer begin as a copy of the first one's and only the 4 (8)
// maps of its weights are encoded.  Each kernel family is built when a call first launches it.  256 layers fit (2.6 MB).
// ---------------------------------------------------------------------------------------------------------------
struct PlanKey {
  const void* ws;
  const void* w[8];
  int64_t s13, s2;
  MmoeGeometry geo;
  int has_shared;
  int device;
  bool operator==(const PlanKey& o) const { return memcmp(this, &o, sizeof(PlanKey)) == 0; }
  bool same_workspace(const PlanKey& o) const {
    return ws == o.ws && has_shared == o.has_shared && device == o.device && memcmp(&geo, &o.geo, sizeof geo) == 0;
  }
};
constexpr int kPlanCacheSize = 256;
using SaPlan = MoeParams;
struct TmPlan { TmParams layer[2]; };
PlanCache<PlanKey, SaPlan, kPlanCacheSize> g_sa_plans;
PlanCache<PlanKey, TmPlan, kPlanCacheSize> g_tm_plans;

PlanKey make_key(const Ctx& c, const MmoeWeights& w, bool has_shared) {
  PlanKey k;
  memset(&k, 0, sizeof k);           // padding bytes take part in the comparison
  k.ws = c.ws;
  const void* ptrs[8] = {w.w13, w.w13_sf, w.w2, w.w2_sf, w.shared_w13, w.shared_w13_sf, w.shared_w2, w.shared_w2_sf};
  for (int i = 0; i < 8; ++i) k.w[i] = ptrs[i];
  k.s13 = w.w13_slice_stride;
  k.s2 = w.w2_slice_stride;
  k.geo = c.geo;
  k.has_shared = has_shared ? 1 : 0;
  k.device = current_device();
  return k;
}

// Pair kernels: what depends on the workspace alone ...
bool set_workspace(const Ctx& c, bool has_shared, TmPlan* plan) {
  const int h = c.geo.hidden, inter = c.geo.intermediate, el = c.e_local;
  const int64_t shared_sf_rows = shared_chunk_rows(c.geo.num_max_tokens);
  TmParams& p1 = plan->layer[0];
  TmParams& p2 = plan->layer[1];
  p1.plan = c.ws + c.lay.plan;
  p1.act_routed = c.at<uint8_t>(c.lay.act_x);
  p1.act_shared = c.at<uint8_t>(c.lay.shared_act_x);
  p1.act_sf_routed = c.at<int32_t>(c.lay.act_sf);
  p1.act_sf_shared = c.at<int32_t>(c.lay.shared_act_sf);
  p1.act_sf_rows_routed = c.lay.pool_sf_rows;
  p1.act_sf_rows_shared = c.lay.shared_sf_rows;
  p1.pool_w = c.at<float>(c.lay.pool_w);
  p1.status = c.at<int32_t>(c.lay.status);
  p1.e_local = el;
  p1.num_ranks = c.geo.num_ranks;
  p1.k_dim = h;
  p1.rows_per_expert = 2 * inter;
  p1.hidden = h;
  p1.inter = inter;
  p2 = p1;
  p2.ret = c.at<__nv_bfloat16>(c.lay.ret);
  p2.shared_out = c.at<__nv_bfloat16>(c.lay.shared_out);
  p2.pool_dst = c.at<int32_t>(c.lay.pool_dst);
  p2.k_dim = inter;
  p2.rows_per_expert = h;
  int bad = make_scale_map(&p1.map_tsf_routed, c.ws + c.lay.pool_sf, c.lay.pool_sf_rows, h / kTileK, kChunkRows);
  bad |= make_scale_map(&p2.map_tsf_routed, c.ws + c.lay.act_sf, c.lay.pool_sf_rows, inter / kTileK, kChunkRows);
  for (int b = 0; b < 4; ++b) {
    bad |= make_token_map(&p1.map_tok_routed[b], c.ws + c.lay.pool_x, h, c.lay.pool_rows, 32 * (b + 1));
    bad |= make_token_map(&p2.map_tok_routed[b], c.ws + c.lay.act_x, inter, c.lay.pool_rows, 32 * (b + 1));
  }
  if (has_shared) {
    bad |= make_scale_map(&p1.map_tsf_shared, c.ws + c.lay.shared_tile_sf, shared_sf_rows, h / kTileK, kChunkRows);
    bad |= make_scale_map(&p2.map_tsf_shared, c.ws + c.lay.shared_act_sf, c.lay.shared_sf_rows, inter / kTileK, kChunkRows);
    for (int b = 0; b < 4; ++b) {
      bad |= make_token_map(&p1.map_tok_shared[b], c.ws + c.lay.x, h, c.geo.num_max_tokens, 32 * (b + 1));
      bad |= make_token_map(&p2.map_tok_shared[b], c.ws + c.lay.shared_act_x, inter, c.geo.num_max_tokens + 128, 32 * (b + 1));
    }
  }
  return bad == 0;
}
// ... and what depends on the weights
bool set_weights(const Ctx& c, const MmoeWeights& w, bool has_shared, TmPlan* plan) {
  const int h = c.geo.hidden, inter = c.geo.intermediate, el = c.e_local;
  TmParams& p1 = plan->layer[0];
  TmParams& p2 = plan->layer[1];
  p1.routed_sliced = w.w13_slice_stride > 0 ? 1 : 0;
  p2.routed_sliced = w.w2_slice_stride > 0 ? 1 : 0;
  int bad = make_weight_map(&p1.map_w_routed, true, w.w13, h, (uint64_t)el * 2 * inter, w.w13_slice_stride, kTileRows);
  bad |= make_scale_map(&p1.map_wsf_routed, w.w13_sf, 2 * (uint64_t)inter, (uint64_t)el * (h / kTileK), 256);
  bad |= make_weight_map(&p2.map_w_routed, true, w.w2, inter, (uint64_t)el * h, w.w2_slice_stride, kTileRows);
  bad |= make_scale_map(&p2.map_wsf_routed, w.w2_sf, h, (uint64_t)el * (inter / kTileK), 256);
  if (has_shared) {
    bad |= make_weight_map(&p1.map_w_shared, false, w.shared_w13, h, 2 * (uint64_t)inter, 0, kTileRows);
    bad |= make_scale_map(&p1.map_wsf_shared, w.shared_w13_sf, 2 * (uint64_t)inter, h / kTileK, 256);
    bad |= make_weight_map(&p2.map_w_shared, false, w.shared_w2, inter, (uint64_t)h, 0, kTileRows);
    bad |= make_scale_map(&p2.map_wsf_shared, w.shared_w2_sf, h, inter / kTileK, 256);
  }
  return bad == 0;
}

// The same two steps for the weights-as-A kernels.
bool set_workspace(const Ctx& c, bool has_shared, SaPlan* plan) {
  const int h = c.geo.hidden, inter = c.geo.intermediate, el = c.e_local;
  UmmaParams& p1 = plan->layer[0];
  UmmaParams& p2 = plan->layer[1];
  p1.plan = c.ws + c.lay.plan;
  p1.tsf_routed = c.at<int32_t>(c.lay.pool_sf);
  p1.x_sf = c.at<int32_t>(c.lay.x_sf);
  p1.topk_idx = c.at<int64_t>(c.lay.topk_idx);
  p1.sorted_route = c.at<int32_t>(c.lay.sorted_route);
  p1.pool_dst = c.at<int32_t>(c.lay.pool_dst);
  p1.topk = c.geo.num_topk;
  p1.topk_weights = c.at<float>(c.lay.topk_weights);
  p1.route_pos = c.at<int32_t>(c.lay.route_pos);
  p1.send_count = c.at<int32_t>(c.lay.send_count);
  p1.send_offset = c.at<int32_t>(c.lay.send_offset);
  p1.recv_count = c.at<int32_t>(c.lay.recv_count);
  p1.x = c.at<uint4>(c.lay.x);
  p1.pool_x = c.at<uint4>(c.lay.pool_x);
  p1.pool_sf = c.at<int32_t>(c.lay.pool_sf);
  p1.pool_sf_rows = c.lay.pool_sf_rows;
  p1.tsf_rows_routed = c.lay.pool_sf_rows;
  p1.act_routed = c.at<uint8_t>(c.lay.act_x);
  p1.act_shared = c.at<uint8_t>(c.lay.shared_act_x);
  p1.act_sf_routed = c.at<uint8_t>(c.lay.act_sf);
  p1.act_sf_shared = c.at<uint8_t>(c.lay.shared_act_sf);
  p1.act_sf_rows_routed = c.lay.pool_sf_rows;
  p1.act_sf_rows_shared = c.lay.shared_sf_rows;
  p1.pool_w = c.at<float>(c.lay.pool_w);
  p1.status = c.at<int32_t>(c.lay.status);
  p1.e_local = el;
  p1.num_ranks = c.geo.num_ranks;
  p1.k_dim = h;
  p1.rows_per_expert = 2 * inter;
  p1.n_blocks = inter / kTileRows;
  p1.hidden = h;
  p1.inter = inter;
  p2 = p1;
  p2.tsf_routed = c.at<int32_t>(c.lay.act_sf);
  p2.tsf_shared = c.at<int32_t>(c.lay.shared_act_sf);
  p2.tsf_rows_shared = c.lay.shared_sf_rows;
  p2.ret = c.at<__nv_bfloat16>(c.lay.ret);
  p2.shared_out = c.at<__nv_bfloat16>(c.lay.shared_out);
  p2.k_dim = inter;
  p2.rows_per_expert = h;
  p2.n_blocks = h / (2 * kTileRows);
  int bad = 0;
  for (int b = 0; b < kNumBoxes; ++b) {
    bad |= make_token_map(&p1.map_tok_routed_box[b], c.ws + c.lay.pool_x, h, c.lay.pool_rows, 16 * (b + 1));
    bad |= make_token_map(&p1.map_tok_shared_box[b], c.ws + c.lay.x, h, c.geo.num_max_tokens, 16 * (b + 1));
    bad |= make_token_map(&p2.map_tok_routed_box[b], c.ws + c.lay.act_x, inter, c.lay.pool_rows, 16 * (b + 1));
    if (has_shared) bad |= make_token_map(&p2.map_tok_shared_box[b], c.ws + c.lay.shared_act_x, inter, c.geo.num_max_tokens, 16 * (b + 1));
    else p2.map_tok_shared_box[b] = p2.map_tok_routed_box[b];
  }
  return bad == 0;
}
bool set_weights(const Ctx& c, const MmoeWeights& w, bool has_shared, SaPlan* plan) {
  const int h = c.geo.hidden, inter = c.geo.intermediate, el = c.e_local;
  UmmaParams& p1 = plan->layer[0];
  UmmaParams& p2 = plan->layer[1];
  p1.wsf_routed = static_cast<const int32_t*>(w.w13_sf);
  p1.wsf_shared = static_cast<const int32_t*>(w.shared_w13_sf);
  p2.wsf_routed = static_cast<const int32_t*>(w.w2_sf);
  p2.wsf_shared = static_cast<const int32_t*>(w.shared_w2_sf);
  p1.routed_sliced = w.w13_slice_stride > 0 ? 1 : 0;
  p2.routed_sliced = w.w2_slice_stride > 0 ? 1 : 0;
  p2.routed_halves = w.w2_slice_stride > 0 && (h / 2) % (2 * kTileRows) != 0 ? 1 : 0;
  int bad = make_w13_map(&p1.map_w_routed, true, w.w13, h, (uint64_t)el * 2 * inter, w.w13_slice_stride);
  bad |= make_weight_map(&p2.map_w_routed, true, w.w2, inter, (uint64_t)el * h, w.w2_slice_stride, (p2.routed_halves != 0 ? 1 : 2) * kTileRows);
  if (has_shared) {
    bad |= make_w13_map(&p1.map_w_shared, false, w.shared_w13, h, 2 * (uint64_t)inter, 0);
    bad |= make_weight_map(&p2.map_w_shared, false, w.shared_w2, inter, (uint64_t)h, 0, 2 * kTileRows);
  } else {
    p1.map_w_shared = p1.map_w_routed;
    p2.map_w_shared = p2.map_w_routed;
  }
  return bad == 0;
}

// the kept parameters of (workspace, weights, geometry), built on first use; null when the driver refuses a map or the host is
// out of memory
template <typename Plan, typename Cache>
std::shared_ptr<const Plan> kept_plan(Cache& cache, const PlanKey& key, const Ctx& c, const MmoeWeights& w, bool has_shared) {
  try {
    return cache.get(key, [&](const Plan* sibling) -> std::shared_ptr<const Plan> {
      const std::shared_ptr<Plan> plan = sibling != nullptr ? std::make_shared<Plan>(*sibling) : std::make_shared<Plan>();
      if (sibling == nullptr && !set_workspace(c, has_shared, plan.get())) return nullptr;
      return set_weights(c, w, has_shared, plan.get()) ? plan : nullptr;
    });
  } catch (...) {
    return nullptr;
  }
}

}  // namespace

int tc_num_sms() {
  const int dev = current_device();
  return dev < 0 ? 0 : g_num_sms[dev];
}
bool tc_ready() { return g_encode != nullptr && tc_num_sms() > 0; }

void set_tuning(int max_stages, int orientation) {
  g_tune_stages = max_stages;
  g_orientation = orientation;
}
int tuned_orientation() { return g_orientation; }

int make_token_map(CUtensorMap* map, const void* base, uint64_t k_elems, uint64_t rows, uint32_t box_rows) {
  const cuuint64_t dims[2] = {k_elems, rows};
  const cuuint64_t strides[1] = {k_elems};
  const cuuint32_t box[2] = {kTileK, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

int make_weight_map(CUtensorMap* map, bool fp4, const void* base, uint64_t k_elems, uint64_t rows_total,
                    int64_t slice_stride, uint32_t box_rows) {
  const uint64_t row_bytes = fp4 ? k_elems / 2 : k_elems;
  const uint64_t slices = slice_stride > 0 ? 2 : 1;
  const uint64_t rows = rows_total / slices;
  const cuuint64_t dims[3] = {k_elems, rows, slices};
  const cuuint64_t strides[2] = {row_bytes, slice_stride > 0 ? static_cast<uint64_t>(slice_stride) : rows * row_bytes};
  const cuuint32_t box[3] = {kTileK, box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = g_encode(map, fp4 ? CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B : CU_TENSOR_MAP_DATA_TYPE_UINT8, 3,
                              const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

int make_scale_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t columns, uint32_t box_rows) {
  const cuuint64_t dims[2] = {rows, columns};
  const cuuint64_t strides[1] = {rows * 4};
  const cuuint32_t box[2] = {box_rows, 1};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

// Once per device (the dynamic shared-memory limits are per device) and outside stream capture.
int prepare_umma(const MmoeGeometry& geo) {
  (void)geo;
  if (g_encode == nullptr) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess || fn == nullptr)
      return MMOE_ERR_CUDA;
    g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  const int dev = current_device();
  if (dev < 0) return MMOE_ERR_CUDA;
  if (g_num_sms[dev] > 0) return MMOE_OK;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return MMOE_ERR_CUDA;
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = prepare_one(umma_kernel<1, false>, Shape<1>::kSmemBytes);
  if (e == cudaSuccess) e = prepare_one(umma_kernel<2, false>, Shape<2>::kSmemBytes);
  if (e == cudaSuccess) e = prepare_one(umma_kernel<2, true>, Shape<2>::kSmemBytes);
  if (e == cudaSuccess) e = prepare_one(moe_kernel<false>, Shape<1>::kSmemBytes);
  if (e == cudaSuccess) e = prepare_one(moe_kernel<true>, Shape<1>::kSmemBytes);
  if (e == cudaSuccess) e = tm_prepare();
  if (e != cudaSuccess) return MMOE_ERR_CUDA;
  g_num_sms[dev] = sms;
  return MMOE_OK;
}

cudaError_t launch_experts_umma(const Ctx& c, const MmoeWeights& w, const MmoeOptions& o, int m, int block_m,
                                cudaStream_t s) {
  if (!tc_ready()) return cudaErrorNotReady;
  const bool has_shared = c.geo.num_shared_experts > 0 && w.shared_w13 != nullptr && m > 0;
  const int64_t timeout_ns = (o.timeout_ms > 0 ? (int64_t)o.timeout_ms : 2000) * 1000000ll;
  const bool fused = c.fused();
  const int mask = o.layer_mask == 0 ? 3 : o.layer_mask;
  cudaError_t e = cudaSuccess;

  // what changes from call to call is patched into a copy of the kept parameters
  auto patch = [&](auto& p, bool layer2) {
    p.timeout_ns = timeout_ns;
    p.clamp = o.activation_clamp;
    p.fast_math = o.fast_math;
    p.with_routed = c.tile_select != 2 ? 1 : 0;
    if (layer2 && fused) {
      p.ep_me = c.geo.rank;
      p.ep_totals = reinterpret_cast<const int32_t*>(c.ws + c.lay.ep_sync + ep_totals_offset());
      for (int r = 0; r < c.geo.num_ranks; ++r)
        p.ep_ret_recv[r] = reinterpret_cast<__nv_bfloat16*>(static_cast<char*>(const_cast<void*>(c.peer_ws[r])) + c.lay.ret_recv);
    }
  };
  // Experts with many rows run on CTA pairs, the others on the weights-as-A kernels: which ones is in the plan.  The shared
  // expert is one or the other by the call's token count.
  const int shared_above = c.shared_above_for(m);
  const bool with_shared = has_shared && c.tile_select != 1;
  const Cut cut = shared_cut(with_shared ? m : 0, shared_above, c.shared_cap_for(m, block_m));
  const SharedTiles shared{cut.parts, cut.step, m}, none{0, 16, 0};
  const bool shared_pairs = m > shared_above;
  const GemmForms forms = gemm_forms(c, m, with_shared);
  const bool pairs = forms.pairs, small = forms.small;
  const bool staged = staged_tokens(c, m, block_m);      // only in a launch of both layers
  const PlanKey key = make_key(c, w, has_shared);
  std::shared_ptr<const TmPlan> tm_plan;
  std::shared_ptr<const SaPlan> sa_plan;
  if (pairs && (tm_plan = kept_plan<TmPlan>(g_tm_plans, key, c, w, has_shared)) == nullptr) return cudaErrorInvalidValue;
  if (small && (sa_plan = kept_plan<SaPlan>(g_sa_plans, key, c, w, has_shared)) == nullptr) return cudaErrorInvalidValue;
  // The whole of one GPU's call: the pairs' two launches, then one for all other experts.  It needs nothing of the pairs'
  // launches, so its CTAs start as theirs run out of tasks.
  const bool both = c.both_layers && small;
  auto small_params = [&](UmmaParams& p, int layer) {
    patch(p, layer == 2);
    p.shared_tiles = shared_pairs ? none : shared;
    p.tile_rows = c.tile_select == 2 ? cut.step : 0;
    p.shared_in_plan = pairs && c.geo.num_ranks == 1 && c.tile_select != 2 ? 1 : 0;
    p.behind_pairs = pairs && both ? 1 : 0;
  };
  const PlanView pv = plan_view(c.ws + c.lay.plan, c.e_local, c.geo.num_ranks);
  const bool claims = c.both_layers && pairs;
  for (int layer = 1; layer <= 2; ++layer) {
    if ((mask & layer) == 0) continue;
    if (e == cudaSuccess && pairs) {
      TmParams p = tm_plan->layer[layer - 1];
      patch(p, layer == 2);
      p.shared_tiles = shared_pairs ? shared : none;
      p.tasks = claims ? pv.pair_tasks + (layer - 1) : nullptr;
      p.done = claims ? pv.done : nullptr;
      e = tm_launch(layer, layer == 2 && fused, p, s);
    }
    if (e == cudaSuccess && small && !both) {
      UmmaParams p = sa_plan->layer[layer - 1];
      small_params(p, layer);
      e = layer == 1 ? launch_layer<1, false>(p, s) : (fused ? launch_layer<2, true>(p, s) : launch_layer<2, false>(p, s));
    }
  }
  if (e == cudaSuccess && both) {
    MoeParams p = *sa_plan;
    for (int layer = 1; layer <= 2; ++layer) small_params(p.layer[layer - 1], layer);
    UmmaParams& p1 = p.layer[0];
    p1.early = pairs ? 0 : 1;
    if (!pairs) p1.tile_rows = small_only_cap(m, block_m, c.e_local);
    p1.num_routes = m * c.geo.num_topk;
    p1.route_here = p.layer[1].route_here = c.route_in_gemm ? 1 : 0;
    p1.stats = c.stats;
    e = staged ? launch_both<true>(p, s) : launch_both<false>(p, s);
  }
  // a pair launch may have run, and no combine follows, which would zero its counters
  if (e != cudaSuccess && claims) cudaMemsetAsync(pv.done, 0, (c.e_local + 4) * sizeof *pv.done, s);
  return e;
}

}  // namespace mmoe
