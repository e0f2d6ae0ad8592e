// Grouped block-scaled GEMMs of the MegaMoE layer, tokens-as-A form on CTA pairs: the experts with many tokens, and the
// shared expert of any call past the decode sizes.
//
//   task  = (two token tiles of <= 128 rows of one expert, 256 consecutive STORED weight rows of that expert)
//   UMMA  = tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale, M = 256 (128 token rows per CTA, E4M3), N = 256 (weight
//           rows, E2M1 routed / E4M3 shared; each CTA stages 128 of them), K = 32, FP32 accumulator of 128 lanes x 256
//           TMEM columns per CTA
//
// What bounds it, measured with the kernel's own instruction stream (4 UMMAs, 3 scale copies, 1 commit and 1 barrier probe
// per 128-K stage, operands landing by TMA): the tensor pipe needs 2 N clk per stage.  One CTA at N = 192 needs 384 and
// takes 434-504, because an instruction costs its issuing warp about 100 clk whatever its size; a CTA pair at N = 256 needs
// 512 and takes 512, issued by one warp for two SMs.  A pair also stages half of the weight rows per CTA (34 KB for
// 128 x 256 x 128 MACs per SM instead of 42 KB for 128 x 192 x 128), so six stages look 3000 clk ahead.  From there the
// 1000 W limit takes over: 3.5-3.8 PFLOP/s at 1.5 GHz.
//
// Tensor memory: two accumulators of 256 columns do not leave room for the scales, so they overlap by 32 columns ([0, 256)
// and [224, 480)); the last 32 columns hold two sets of scale columns, used by alternate stages.  The epilogue reads the
// column group that holds the overlap first and releases it at once; the next task's UMMAs start then, not when the
// accumulator is drained.
//
// A thread of the epilogue owns a TOKEN (TMEM lane) and sees the task's weight rows as consecutive columns:
//   * the stored W13 row order [g0..7, u0..7, g8..15, ...] (backend/weights.py:83-97 of the reference) puts the gate and
//     the up value of a channel 8 columns apart in the same thread -- no de-interleaving tensor map, no shuffles, and the
//     stored scale words (4x32 transposed per 128 stored rows) are already what tcgen05.cp wants: nothing is permuted;
//   * the amax of 32 output channels is a reduction inside one thread;
//   * outputs leave in rows: 32 E4M3 bytes per scale group as two 16-byte stores (layer 1); layer 2 passes a block of
//     32 rows x 64 columns through a swizzled staging area so that 8 lanes write 128 contiguous bytes of one row -- also
//     when the row goes straight into the source rank's buffer over NVLink (kFused).
//
//   warp 0     producer (both CTAs): per stage one TMA box of token rows, one of weight rows (packed FP4 expands to byte
//              containers on the way into shared memory) and the two scale chunks; every copy signals the LEADER's barrier
//              (.cta_group::2), and none uses cluster multicast
//   warp 1     issuer (leader): scale copies into TMEM, UMMAs, one commit that frees the stage in both CTAs
//   warps 2-9  epilogue (both CTAs; layer 2: warps 2-5)
//   last warp  where the pairs claim their tasks: scheduler (leader), forwarder of the queue (peer)
//
// Copies and tensor-core instructions are issued by one elected lane of a warp that walks its loop in step (all lanes wait,
// elect.sync around the issue): operands then stay in uniform registers.  From a lane that alone runs the loop a stage took
// 563-703 clk.
//
// The same roles exist in the reference's kernel (backend/kernel/tma_warps.py, mma_warp.py, epilogue.py).  Persistent
// pairs take the tasks tile-major, so that the pairs working at the same time share token tiles and the tiles
// of one expert share its weights in L2.  Every wait is bounded (see Waiter).
#include <cuda_fp8.h>

#include "mmoe_pair_queue.h"
#include "mmoe_tc.cuh"

namespace mmoe {

namespace {

// Epilogue warps.  Layer 1 has two per scheduler, each with half of the columns: one alone runs at the latency of its own
// instructions, and with the IEEE sigmoid (fast_math off) that is longer than the 22 thousand clk of a task's UMMAs (2800
// tokens, 48 experts: 1304 us with one, 1024 with two).  Layer 2 only converts and stores, and has no shared memory left for more staging blocks.
__host__ __device__ constexpr int tm_epilogue_warps(int layer) { return layer == 1 ? 8 : 4; }
constexpr int tm_threads(int layer) { return 64 + 32 * tm_epilogue_warps(layer) + 32; }
constexpr int kTmN = 256;                          // weight rows of a task (UMMA N)
constexpr int kTmRows = 128;                       // token rows of a tile (UMMA M per CTA)
constexpr int kTmABytes = kTmRows * kTileK;        // 16 KB
constexpr int kTmBBytes = kTmN / 2 * kTileK;       // 16 KB of byte containers: this CTA's half of the weight rows
constexpr int kTmSfBytes = 512 + 2 * 512;          // token scale chunk, two weight scale chunks
constexpr int kTmStageBytes = kTmABytes + kTmBBytes + kTmSfBytes;
constexpr int kTmStages = 6;
constexpr int kTmStagingBytes = 4 * 32 * 128;      // layer 2: one 32-row x 128-byte output block per epilogue warp
constexpr uint32_t kTmAccStride = 224;             // the two accumulators: columns [0, 256) and [224, 480)
constexpr uint32_t kTmSfCol = 480;                 // scale columns: two sets of 16 (4 token rows' + 8 weight rows' + 4 unused)
constexpr int tm_smem_bytes(int layer) { return 1024 + kTmStages * kTmStageBytes + (layer == 2 ? kTmStagingBytes : 0) + 1024; }
static_assert(tm_smem_bytes(2) <= 227 * 1024, "shared memory budget");

struct TmControl {        // lives at the start of shared memory (same layout in both CTAs of a pair)
  uint64_t full[8];       // leader only: every copy of the stage, in both CTAs, has landed
  uint64_t empty[8];      // issuer -> producers of both CTAs: the stage may be overwritten
  uint64_t tmem_full[2];  // issuer -> epilogue of both CTAs
  uint64_t overlap_free;  // leader only: epilogue warps of both CTAs -> issuer: the overlapped columns have been read
  uint64_t q_full[kPairQueue];    // scheduler -> the roles of this CTA: a task ...
  uint64_t q_empty[kPairQueue];   // ... which all roles of this CTA have read; in the leader also those of the peer
  uint64_t q_want;                // leader only: producer -> scheduler: the next one, please
  volatile int32_t q_task[kPairQueue];
  uint32_t tmem_base;
  volatile int32_t abort_flag;
  // layer 2 with the write-back fused in: slot s < 32 is `ret_recv` of source rank s
  __nv_bfloat16* out_base[32];
  int32_t rank_off[33];   // first receive-order row of each source rank
  int32_t home_base[32];  // send position on that rank of the first row it sent here
};
static_assert(sizeof(TmControl) <= 1024, "control block");

// ---------------------------------------------------------------------------------------------------------------
// cluster / CTA-pair helpers
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Arrival on the barrier that hands columns of tensor memory back, in either CTA of the pair: ordered by the tcgen05 fences on
// either side, and no memory access rides on it (the queue of tasks has arrivals of its own).  So the default release, of CTA scope, is enough: one of cluster scope first waits for
// this warp's outstanding stores to global memory, which stood between every two tasks of the issuer.  Cluster scope -> CTA scope, one card: 3840
// tokens of 48 experts 930 -> 908 us repeated for seconds (at the power limit), 819 -> 800 in bursts of 30 calls; 2560 of 16 376 -> 369 and
// 333 -> 326, 3001 of 96 skewed 884 -> 870 and 778 -> 765, 1021 of 384 skewed 456 -> 451 and 410 -> 405.
__device__ __forceinline__ void mbar_arrive_pair(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair when everything issued so far has completed
__device__ __forceinline__ void pair_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(static_cast<uint16_t>(3)) : "memory");
}
__device__ __forceinline__ void pair_cp_sf(uint32_t tmem_addr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem_addr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}
// tile loads into this CTA's shared memory whose completion is counted on a barrier of either CTA of the pair
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void pair_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}

// What the queue of claimed tasks is made of (mmoe_pair_queue.h); every function by the whole warp.
template <bool kOneLanePolls>
struct PairPort {
  TmControl* ctl;
  Waiter& waiter;
  __device__ __forceinline__ uint32_t bar(PairBarrier which, uint32_t slot) const {
    return smem_u32(which == kPairFull ? &ctl->q_full[slot] : &ctl->q_empty[slot]);
  }
  __device__ __forceinline__ bool wait_own(PairBarrier which, uint32_t slot, uint32_t parity) {
    if (!(kOneLanePolls ? waiter.wait_warp(bar(which, slot), parity) : waiter.wait_uniform(bar(which, slot), parity))) return false;
    __syncwarp();
    return true;
  }
  // ... and what the other CTA did before completing the phase is visible to every lane.  The phase is over and the next one needs this role.
  __device__ __forceinline__ bool wait_pair(PairBarrier which, uint32_t slot, uint32_t parity) {
    if (!wait_own(which, slot, parity)) return false;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%0], %1;\n\t}"
                 ::"r"(bar(which, slot)), "r"(parity) : "memory");
    return true;
  }
  __device__ __forceinline__ int read(uint32_t slot) const { return ctl->q_task[slot]; }
  __device__ __forceinline__ void arrive_own(PairBarrier which, uint32_t slot) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar(which, slot));
  }
  __device__ __forceinline__ void arrive_leader(PairBarrier which, uint32_t slot) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
      asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(map_to_cta(bar(which, slot), 0)) : "memory");
  }
  // lane r: to CTA r, the slot's barrier completed with it
  __device__ __forceinline__ void send(uint32_t slot, int task) {
    const uint32_t lane = threadIdx.x & 31;
    if (lane < 2) {
      const uint32_t dst = map_to_cta(smem_u32(const_cast<int32_t*>(&ctl->q_task[slot])), lane), full = map_to_cta(bar(kPairFull, slot), lane);
      asm volatile("mbarrier.arrive.expect_tx.release.cluster.shared::cluster.b64 _, [%0], 4;" ::"r"(full) : "memory");
      asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(task), "r"(full) : "memory");
    }
    __syncwarp();
  }
};

// The task list as a role of a pair walks it: first the shared expert's tasks, which need nothing but the staged tokens
// and are on the host's count of tokens, then -- once everything before this launch in the stream has completed -- the pair
// tiles of the plan.  In GEMM1 of the single-GPU call the placement of the routed rows, and the launch itself, hide behind
// the shared expert this way.
// Either dealt out beforehand, or (both layers of a single-GPU call) claimed from a counter by the leader's scheduler: SMs come free
// one by one, over 25 us behind the placement and 50 behind GEMM1, and a pair that starts late takes fewer tasks.  GEMM2 then starts
// where GEMM1 has ended and waits expert by expert for its counted parts, not for its last CTA.  Dealt out with GEMM2 behind all of GEMM1 ->
// claimed so -> GEMM2 behind counted parts as well, the same card and conditions: 3840 tokens of 48 experts 917 -> 914 -> 908 us repeated, 804 -> 803
// -> 800 in bursts; 2560 of 16 371 -> 372 -> 369 and 327 -> 328 -> 326; 1021 skewed 455 -> 456 -> 451 and 409 -> 410 -> 405; 3001 skewed 868 -> 867 -> 870 and 766 ->
// 767 -> 764.  So claiming alone gives nothing, both together up to 1 %; other sizes lie within 0.4 % on either side.
struct PairWalk {
  const TmParams& p;
  TmControl* ctl;
  uint32_t cta;
  int n_blocks, task, stride;
  uint32_t taken;
  bool waited;
  int routed_tiles;
  const Tile* tiles;
  Tile tile;              // this CTA's half of the current task
  int peer_valid, nb;     // rows of the other half; weight block
  __device__ __forceinline__ PairWalk(const TmParams& params, TmControl* control, uint32_t cta_rank, bool plan_ready)
      : p(params), ctl(control), cta(cta_rank), n_blocks(params.rows_per_expert / kTmN), task(blockIdx.x / 2), stride(gridDim.x / 2),
        taken(0), waited(false), routed_tiles(0), tiles(nullptr) {
    if (plan_ready) load_plan();
  }
  __device__ __forceinline__ void load_plan() {
    const PlanView pv = plan_view(const_cast<char*>(p.plan), p.e_local, p.num_ranks);
    tiles = pv.tiles + pv.hdr->num_small_tiles;
    routed_tiles = p.with_routed ? pv.hdr->num_routed_tiles - pv.hdr->num_small_tiles : 0;
    waited = true;
  }
  // true: tile, peer_valid and nb are those of task t; false behind the last one
  __device__ __forceinline__ bool locate(int t) {
    const int pair = t / n_blocks, first = p.shared_tiles.parts / 2;
    nb = t - pair * n_blocks;
    if (pair < first) {
      tile = p.shared_tiles.at(2 * pair + static_cast<int>(cta));
      peer_valid = p.shared_tiles.at(2 * pair + static_cast<int>(cta ^ 1u)).n_valid;
      return true;
    }
    if (!waited) {
      chain_wait();
      load_plan();
    }
    const int i = 2 * (pair - first);
    if (i >= routed_tiles) return false;
    tile = tiles[i + cta];
    peer_valid = tiles[i + (cta ^ 1u)].n_valid;
    return true;
  }
  // true: ... of this role's next task; false when there is none or the call is being abandoned
  template <bool kOneLanePolls>
  __device__ __forceinline__ bool next(Waiter& waiter) {
    int t = task;
    task += stride;
    if (p.tasks != nullptr) {
      PairPort<kOneLanePolls> port{ctl, waiter};
      if (!pair_take(port, taken++, &t)) return false;
    }
    return locate(t);
  }
};

// token box of a tile: the smallest of 32 / 64 / 96 / 128 rows that covers it
__device__ __forceinline__ int tm_box(int n_valid) { return n_valid <= 32 ? 0 : (n_valid - 1) >> 5; }

// Layer-1 epilogue of one scale group: 64 accumulator columns = 32 channels (columns 16b + j hold the gate, 16b + 8 + j
// the up value of channel 8b + j) -> SwiGLU, x top-k weight, amax, UE8M0 exponent, 32 E4M3 bytes.  The fast-math choice
// is a template parameter: a per-element branch would serialise the 32 independent dependency chains.
template <bool kFast>
__device__ __forceinline__ int tm_l1_group(const uint32_t (&v)[64], float wt, float clamp, uint32_t (&w)[8]) {
  float a[32];
  uint32_t amax_bits = 0;
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float x = swiglu_act_t<kFast>(__uint_as_float(v[16 * b + j]), __uint_as_float(v[16 * b + 8 + j]), wt, clamp);
      a[8 * b + j] = x;
      amax_bits = max(amax_bits, __float_as_uint(fabsf(x)));
    }
  const int sf_exp = ue8m0_exp_of_amax(__uint_as_float(amax_bits));
  const float inv = ue8m0_inv(sf_exp);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(__fmul_rn(a[4 * c], inv), __fmul_rn(a[4 * c + 1], inv)),
                                                 __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(__fmul_rn(a[4 * c + 2], inv), __fmul_rn(a[4 * c + 3], inv)),
                                                 __NV_SATFINITE, __NV_E4M3);
    w[c] = lo | (hi << 16);
  }
  return sf_exp;
}

template <int kLayer, bool kFused>
__global__ void __launch_bounds__(tm_threads(kLayer), 1) tm_kernel(const __grid_constant__ TmParams p) {
  static_assert(!kFused || kLayer == 2, "only GEMM2 writes rows back");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);   // the same offset in both CTAs of a pair
  TmControl* ctl = reinterpret_cast<TmControl*>(smem);
  uint8_t* a_base = smem + 1024;
  uint8_t* b_base = a_base + kTmStages * kTmABytes;
  uint8_t* sf_base = b_base + kTmStages * kTmBBytes;
  uint8_t* staging = sf_base + kTmStages * kTmSfBytes;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();                         // 0 = leader

  // GEMM2 behind GEMM1 of the same call: GEMM1 opens the chain after its own wait, so all that comes before GEMM1 is complete, and
  // GEMM1 itself counts its finished parts.
  const PlanView pv = plan_view(const_cast<char*>(p.plan), p.e_local, p.num_ranks);
  const bool behind_layer1 = kLayer == 2 && p.done != nullptr, opens = kLayer == 1 && p.done != nullptr;
  auto wait_front = [&] {
    if (!behind_layer1 || !chain_opened(pv.pairs_open)) chain_wait();
  };
  if (p.shared_tiles.parts == 0) {        // routed tiles only, of which the call may have none
    wait_front();
    if (p.with_routed == 0 || pv.hdr->num_routed_tiles == pv.hdr->num_small_tiles) {
      if (opens && threadIdx.x == 0) open_chain(pv.pairs_open);
      chain_wait();
      return;
    }
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < kTmStages; ++i) {
      mbar_init(smem_u32(&ctl->full[i]), 1);
      mbar_init(smem_u32(&ctl->empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&ctl->tmem_full[i]), 1);
    mbar_init(smem_u32(&ctl->overlap_free), 2 * tm_epilogue_warps(kLayer));   // one arrival per epilogue warp of the pair
    for (uint32_t i = 0; i < kPairQueue; ++i) {
      mbar_init(smem_u32(&ctl->q_full[i]), pair_full_count());
      mbar_init(smem_u32(&ctl->q_empty[i]), pair_empty_count(cta == 0, tm_epilogue_warps(kLayer) + (cta == 0 ? 2 : 1)));   // ... producer and issuer
    }
    mbar_init(smem_u32(&ctl->q_want), 1);
    ctl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {       // the same warp of both CTAs of a pair allocates
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  // Everything above touches only this CTA's own shared and tensor memory.  GEMM2 that does not count GEMM1's parts waits
  // here for everything before it; GEMM1 in a programmatic chain starts when the blocks of the placement have all started,
  // i.e. after the launches before it (staging, counting) have completed, and waits when it comes to the routed tiles.
  // Only then does it let the next launch start.
  if (kLayer == 2 && p.shared_tiles.parts != 0) wait_front();
  if (kFused) {
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
  cluster_sync_all();                       // the peer's barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
  PairWalk walk(p, ctl, cta, kLayer == 2);
  const int k_stages = p.k_dim / kTileK;

  Waiter waiter{&ctl->abort_flag, p.status, global_timer() + static_cast<uint64_t>(p.timeout_ns), kStatusPairs + kLayer, warp};
  const uint32_t full0 = smem_u32(&ctl->full[0]), empty0 = smem_u32(&ctl->empty[0]);

  // Every role walks the same task list; its loop runs at instruction latency, so everything that does not change inside a
  // task is computed once per task.
  if (warp == 0) {
    // --------------------------------------------------------------------------------------------- producer
    uint32_t stage = 0, phase = 0;
    const uint32_t a0 = smem_u32(a_base), b0 = smem_u32(b_base), sf0 = smem_u32(sf_base);
    const uint32_t leader_full0 = map_to_cta(full0, 0);
    const int half = p.rows_per_expert / 2;
    const uint32_t want = p.tasks != nullptr && cta == 0 ? smem_u32(&ctl->q_want) : 0u;
    const int want_at = max(k_stages - 8, 0);            // a claim in time, and not earlier: that would hoard tasks
    bool ok = true, released = false;
    auto release = [&] {                                 // once everything in front of the launch is complete
      if (released || !walk.waited) return;
      __syncwarp();
      if (opens && cta == 0 && lane == 0) open_chain(pv.pairs_open);
      __syncwarp();
      chain_release();
      released = true;
    };
    while (ok && walk.next<false>(waiter)) {
      release();
      const Tile tile = walk.tile;
      const int nb = walk.nb;
      const bool shared = tile.expert == kSharedExpert;
      const int e = shared ? 0 : tile.expert;
      const int r0 = nb * kTmN + static_cast<int>(cta) * (kTmN / 2);     // this CTA's 128 stored weight rows: inside one slice
      const bool sliced = !shared && p.routed_sliced != 0;
      const int slice = sliced && r0 >= half ? 1 : 0;
      const int row = sliced ? e * half + r0 - slice * half : e * p.rows_per_expert + r0;
      const CUtensorMap* wmap = shared ? &p.map_w_shared : &p.map_w_routed;
      const CUtensorMap* wsfmap = shared ? &p.map_wsf_shared : &p.map_wsf_routed;
      const CUtensorMap* tsfmap = shared ? &p.map_tsf_shared : &p.map_tsf_routed;
      const int box = tm_box(tile.n_valid);
      const CUtensorMap* tmap = shared ? &p.map_tok_shared[box] : &p.map_tok_routed[box];
      // what both CTAs' copies add up to, counted on the leader's barrier; packed FP4 counts its global bytes
      const uint32_t tx = static_cast<uint32_t>((box + tm_box(walk.peer_valid) + 2) * 32 * kTileK) +
                          (shared ? kTmN * kTileK : kTmN * kTileK / 2) + 2 * kTmSfBytes;
      const int wsf_col = nb * kTmN, tsf_col = tile.sf_chunk * kChunkRows;
      int wsf_row = e * k_stages;
      int k0 = 0;
      if (behind_layer1) {
        const int32_t* done = p.done + (shared ? p.e_local : e);
        const int need = tile.parts * tm_epilogue_warps(1) * (2 * p.inter / kTmN);
        for (uint32_t spin = 0; ok && !rows_ready(done, need); ++spin) {
          if ((spin & 63u) == 63u && __any_sync(0xffffffffu, waiter.abandoned())) ok = false;
          __nanosleep(40);
        }
        if (!ok) break;
      }
      for (int kb = 0; kb < k_stages; ++kb, k0 += kTileK, ++wsf_row) {
        if (!waiter.wait_uniform(empty0 + 8 * stage, phase ^ 1u)) { ok = false; break; }
        const uint32_t bar = leader_full0 + 8 * stage;
        if (elect_one()) {
          if (want != 0 && kb == want_at) mbar_arrive(want);
          if (cta == 0) mbar_expect_tx(full0 + 8 * stage, tx);
          pair_load_3d(b0 + stage * kTmBBytes, wmap, k0, row, slice, bar);
          pair_load_2d(a0 + stage * kTmABytes, tmap, k0, tile.row0, bar);
          pair_load_2d(sf0 + stage * kTmSfBytes + 512, wsfmap, wsf_col, wsf_row, bar);   // scales of all 256 rows in both CTAs
          pair_load_2d(sf0 + stage * kTmSfBytes, tsfmap, tsf_col, kb, bar);
        }
        __syncwarp();
        if (++stage == kTmStages) { stage = 0; phase ^= 1u; }
      }
    }
    release();
  } else if (warp == 1) {
    // --------------------------------------------------------------------------------------------- issuer
    if (cta == 0) {
      uint32_t stage = 0, phase = 0, it = 0, sf_set = 0;
      bool ok = true;
      const uint64_t sw128_hi = desc_hi_sw128(), sf_hi = desc_hi_sf(128);
      const uint32_t a_lo0 = (smem_u32(a_base) & 0x3FFFFu) >> 4;
      const uint32_t b_lo0 = (smem_u32(b_base) & 0x3FFFFu) >> 4;
      const uint32_t sf_lo0 = (smem_u32(sf_base) & 0x3FFFFu) >> 4;
      for (; ok && walk.next<false>(waiter); ++it) {
        const bool shared = walk.tile.expert == kSharedExpert;
        // M = 256 over the pair; idesc field [24,29) = M >> 4
        const uint32_t idesc0 = make_idesc(0u, shared ? 0u : 5u, static_cast<uint32_t>(kTmN), 0) + ((128u >> 4) << 24);
        const uint32_t d = tmem_base + (it & 1u) * kTmAccStride;
        // Every epilogue warp has read its first columns of the previous task, the overlapped ones among them.  They take
        // tasks in order, so this task's own columns, last used two tasks ago, are free as well.
        if (it > 0 && !waiter.wait_uniform(smem_u32(&ctl->overlap_free), (it - 1u) & 1u)) { ok = false; break; }
        tc_fence_after();
        for (int kb = 0; kb < k_stages; ++kb) {
          if (!waiter.wait_uniform(full0 + 8 * stage, phase)) { ok = false; break; }
          const uint32_t a_lo = a_lo0 + stage * (kTmABytes >> 4);
          const uint32_t b_lo = b_lo0 + stage * (kTmBBytes >> 4);
          const uint32_t sf_lo = sf_lo0 + stage * (kTmSfBytes >> 4);
          const uint32_t sfa = tmem_base + kTmSfCol + 16 * sf_set, sfb = sfa + 4;
          if (elect_one()) {
            // every CTA of the pair copies from its own shared memory into its own tensor memory; copies and UMMAs of one
            // thread execute in order, so two alternating sets of scale columns suffice
            pair_cp_sf(sfa, sf_hi | sf_lo);
            pair_cp_sf(sfb, sf_hi | (sf_lo + 32));
            pair_cp_sf(sfb + 4, sf_hi | (sf_lo + 64));
#pragma unroll
            for (int k = 0; k < kTileK / 32; ++k)
              pair_mma(d, sw128_hi | (a_lo + 2 * k), sw128_hi | (b_lo + 2 * k),
                       idesc0 + k * ((1u << 4) | (1u << 29)),              // scale byte k of both operands
                       sfa, sfb, (kb | k) != 0 ? 1u : 0u);
            pair_commit(empty0 + 8 * stage);        // the stage is free in both CTAs once these UMMAs retire
          }
          __syncwarp();
          sf_set ^= 1u;
          if (++stage == kTmStages) { stage = 0; phase ^= 1u; }
        }
        if (ok && elect_one()) pair_commit(smem_u32(&ctl->tmem_full[it & 1u]));
        __syncwarp();
      }
    }
  } else if (warp == 2 + tm_epilogue_warps(kLayer)) {
    // --------------------------------------------------------------------------------------------- scheduler, forwarder
    PairPort<false> port{ctl, waiter};
    if (p.tasks == nullptr) {
    } else if (cta == 0) {
      for (uint32_t n = 0;; ++n) {
        int t = 0;
        if (lane == 0) t = atomicAdd(p.tasks, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (!pair_put(port, n, t) || !walk.locate(t)) break;
        if (!waiter.wait_uniform(smem_u32(&ctl->q_want), n & 1u)) break;
      }
    } else {
      int t;
      for (uint32_t n = 0; pair_peek(port, n, &t) && walk.locate(t) && pair_forward(port, n);) ++n;
    }
  } else {
    // --------------------------------------------------------------------------------------------- epilogue
    const int q = warp & 3;                       // TMEM lane quadrant this warp may read
    const int i = q * 32 + lane;                  // token row of the tile this thread owns
    const uint32_t lane_sel = static_cast<uint32_t>(q * 32) << 16;
    const uint32_t overlap_free_leader = map_to_cta(smem_u32(&ctl->overlap_free), 0);
    uint32_t it = 0;
    bool ok = true;
    // layer 1: this warp's part of a task is stored
    auto publish = [&](const Tile& tile) {
      if (kLayer == 2 || p.done == nullptr) return;
      __syncwarp();
      if (lane == 0) {
        part_release();
        part_count(p.done + (tile.expert == kSharedExpert ? p.e_local : tile.expert));
      }
    };
    for (; ok && walk.next<true>(waiter); ++it) {
      const Tile tile = walk.tile;
      const int nb = walk.nb;
      const bool shared = tile.expert == kSharedExpert;
      const uint32_t acc = it & 1u;
      const bool live = i < tile.n_valid;
      const int64_t row = (int64_t)tile.row0 + i;
      // per-token side data, fetched before the accumulator is awaited
      float wt = 1.0f;
      __nv_bfloat16* out = nullptr;
      if (kLayer == 1) {
        if (!shared && live) wt = __ldcg(p.pool_w + row);
      } else if (live) {
        if (shared) {
          out = p.shared_out + row * p.hidden;
        } else if (!kFused) {
          out = p.ret + (int64_t)__ldcg(p.pool_dst + row) * p.hidden;
        } else {
          const int r = __ldcg(p.pool_dst + row);         // receive-order row -> source rank and its send position
          int sr = 0;
          while (sr + 1 < p.num_ranks && r >= ctl->rank_off[sr + 1]) ++sr;
          out = ctl->out_base[sr] + (int64_t)(ctl->home_base[sr] + r - ctl->rank_off[sr]) * p.hidden;
        }
        out += nb * kTmN;
      }
      const int sub = lane >> 3, chunk = lane & 7;
      // layer 2: destination of the four rows this lane helps to write in each of the eight steps (row 4j + sub)
      __nv_bfloat16* dst_row[8];
      if (kLayer == 2) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const unsigned long long ptr = __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(out), 4 * j + sub);
          dst_row[j] = reinterpret_cast<__nv_bfloat16*>(ptr);       // null for rows past the tile's last token
        }
      }
      if (!waiter.wait_warp(smem_u32(&ctl->tmem_full[acc]), (it >> 1) & 1u)) { ok = false; break; }
      tc_fence_after();
      // None of this warp's rows is a token: nothing to do (350 rows per expert, fast_math off: 1035 -> 913 us).
      if (q * 32 >= tile.n_valid) {
        tc_fence_before();
        if (lane == 0) mbar_arrive_pair(overlap_free_leader);
        publish(tile);
        continue;
      }
      const uint32_t d0 = tmem_base + lane_sel + acc * kTmAccStride;
      // the 64-column group with the 32 overlapped columns comes first: columns 224-255 of accumulator 0, 0-31 of 1; in layer 1
      // warps 2-5 take groups 0 and 1, warps 6-9 groups 2 and 3
      const int first = acc == 0 ? 3 : 0, side = (warp - 2) >> 2;
      uint32_t sf_word = 0;
#pragma unroll 1
      for (int step = 0; step < 16 / tm_epilogue_warps(kLayer); ++step) {
        const int g = kLayer == 1 ? 2 * side + ((first + step) & 1) : (first + step) & 3;
        uint32_t v[64];
        tc_ld32(d0 + 64 * g, v);
        tc_ld32(d0 + 64 * g + 32, v + 32);
        tc_ld_wait();
        if (step == 0) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_pair(overlap_free_leader);
        }
        if (kLayer == 1) {
          uint32_t w[8];
          const int sf_exp = p.fast_math != 0 ? tm_l1_group<true>(v, wt, p.clamp, w) : tm_l1_group<false>(v, wt, p.clamp, w);
          sf_word |= static_cast<uint32_t>(sf_exp) << (8 * (g & 1));
          if (live) {
            uint4* dst = reinterpret_cast<uint4*>((shared ? p.act_shared : p.act_routed) + row * p.inter + nb * (kTmN / 2) + 32 * g);
            dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
            dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
          }
        } else {
          // Rows leave as 128-byte segments: the warp's 32 x 64 block of BF16 values goes through a swizzled staging block
          // in shared memory (16-byte chunk c of row r at chunk c ^ (r & 7): conflict-free both ways), then 8 lanes write
          // one row's 128 contiguous bytes -- four full lines per instruction instead of 32 scattered 16-byte pieces,
          // which is what matters when the destination is another rank's buffer across NVLink.
          uint8_t* stg = staging + (warp - 2) * 4096;
          __syncwarp();                                   // the previous block has been read out
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint32_t w[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const __nv_bfloat162 pr = __floats2bfloat162_rn(__uint_as_float(v[8 * c + 2 * t]), __uint_as_float(v[8 * c + 2 * t + 1]));
              w[t] = *reinterpret_cast<const uint32_t*>(&pr);
            }
            *reinterpret_cast<uint4*>(stg + lane * 128 + ((c ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int r = 4 * j + sub;
            const uint4 val = *reinterpret_cast<const uint4*>(stg + r * 128 + ((chunk ^ (r & 7)) << 4));
            if (dst_row[j] != nullptr) *reinterpret_cast<uint4*>(dst_row[j] + 64 * g + chunk * 8) = val;
          }
        }
      }
      if (kLayer == 1 && live) {
        // the task's 128 channels are one scale word of layer 2's K dimension, half of it from each of the row's two threads
        int32_t* act_sf = shared ? p.act_sf_shared : p.act_sf_routed;
        const int64_t sf_rows = shared ? p.act_sf_rows_shared : p.act_sf_rows_routed;
        reinterpret_cast<uint16_t*>(act_sf + nb * sf_rows + (int64_t)tile.sf_chunk * kChunkRows + chunk_pos(i))[side] = static_cast<uint16_t>(sf_word);
      }
      publish(tile);
    }
  }

  // ---------------------------------------------------------------------------------------------------- teardown
  chain_wait();                             // a unit without routed tasks must not end before what precedes the launch
  __syncwarp();
  if (ctl->abort_flag != 0) {
    // abandoned call: give copies that are still in flight time to land in this CTA's shared memory before it exits
    const uint64_t t0 = global_timer();
    while (global_timer() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                       // no CTA leaves while its peer may still arrive on its barriers
  tc_fence_after();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
}

template <int kLayer, bool kFused>
cudaError_t tm_prepare_one() {
  return cudaFuncSetAttribute(tm_kernel<kLayer, kFused>, cudaFuncAttributeMaxDynamicSharedMemorySize, tm_smem_bytes(kLayer));
}

}  // namespace

cudaError_t tm_prepare() {
  cudaError_t e = tm_prepare_one<1, false>();
  if (e == cudaSuccess) e = tm_prepare_one<2, false>();
  if (e == cudaSuccess) e = tm_prepare_one<2, true>();
  return e;
}

cudaError_t tm_launch(int layer, bool fused, const TmParams& p, cudaStream_t s) {
  const int grid = tc_num_sms() & ~1;
  if (grid <= 0) return cudaErrorNotReady;
  const dim3 g(grid), b(tm_threads(layer));
  if (layer == 1) return launch_clustered(tm_kernel<1, false>, g, b, tm_smem_bytes(1), 2, s, p);
  return fused ? launch_clustered(tm_kernel<2, true>, g, b, tm_smem_bytes(2), 2, s, p)
               : launch_clustered(tm_kernel<2, false>, g, b, tm_smem_bytes(2), 2, s, p);
}

}  // namespace mmoe
