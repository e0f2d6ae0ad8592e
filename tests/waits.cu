// The waits of a launch of both GEMMs, one at a time, for a flag that nothing sets.  Test helper: compiled with the kernels' source.
#include "../vllm_plugin_b200/csrc/mmoe_umma.cu"

namespace mmoe {
bool chained() { return false; }
int ep_totals_offset() { return 0; }
cudaError_t tm_prepare() { return cudaSuccess; }
cudaError_t tm_launch(int, bool, const TmParams&, cudaStream_t) { return cudaSuccess; }

namespace {
// out[0]: 1 when the wait gave up, 2 when it ended some other way
__global__ void __launch_bounds__(32) wait_kernel(int which, const __grid_constant__ MoeParams f, int32_t* out) {
  __shared__ Control ctl;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&ctl.q_full[0]), 1);
    mbar_init(smem_u32(&ctl.q_empty[0]), 1);
    ctl.abort_flag = 0;
    ctl.slots[0].layer = 1;
  }
  __syncwarp();
  const UmmaParams& p = f.layer[0];
  Waiter waiter{&ctl.abort_flag, p.status, global_timer() + static_cast<uint64_t>(p.timeout_ns), 4, 10 + which};
  bool ended;
  if (which == 0) {
    ended = sa_wait_plan(p, waiter);
  } else if (which == 1) {
    ended = TaskFeed<false>(f, &ctl).next(waiter);
  } else if (which == 2) {
    ended = TaskFeed<true>(f, &ctl).next(waiter);
  } else {
    TaskQueue<true> queue(f, &ctl);
    queue.handed_on = kQueue;                       // the slot has been used once and nothing has released it
    QueueSlot t{Tile{0, 0, 1, 0, 0, 1, {0, 0}}, 0, 1, 0};
    ended = queue.hand_on(waiter, t);
  }
  if (threadIdx.x == 0) out[0] = ended ? 2 : 1;
}
}  // namespace
}  // namespace mmoe

extern "C" int run_wait(int which, void* plan, int e_local, void* status, int64_t timeout_ns, void* out, void* stream) {
  auto f = std::make_unique<mmoe::MoeParams>();
  memset(static_cast<void*>(f.get()), 0, sizeof *f);
  mmoe::UmmaParams& p = f->layer[0];
  p.plan = static_cast<const char*>(plan);
  p.status = static_cast<int32_t*>(status);
  p.e_local = e_local;
  p.num_ranks = 1;
  p.route_here = 1;
  p.timeout_ns = timeout_ns;
  return static_cast<int>(mmoe::launch_plain(mmoe::wait_kernel, dim3(1), dim3(32), 0, static_cast<cudaStream_t>(stream), which, *f,
                                             static_cast<int32_t*>(out)));
}
