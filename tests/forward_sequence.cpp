// Prints the steps that mmoe_forward (csrc/mmoe_abi.cu) takes, with launches that fail where a CPU test wants them to.  Host code
// only: every launcher is a stand-in, and nothing touches a device.
#include "../vllm_plugin_b200/csrc/mmoe_abi.cu"

static std::string g_steps, g_failing;

static cudaError_t step(const char* name) {
  g_steps += std::string(" ") + name;
  return g_failing == name ? cudaErrorLaunchOutOfResources : cudaSuccess;
}

namespace mmoe {
ChainScope::ChainScope(bool) : saved_(false) {}
ChainScope::~ChainScope() {}
bool chained() { return false; }
bool tc_ready() { return true; }
void set_tuning(int, int) {}
int tuned_orientation() { return 0; }
int prepare_umma(const MmoeGeometry&) { return MMOE_OK; }
int ep_sync_bytes() { return 0; }
int ep_totals_offset() { return 0; }
int route_order_static_max_tokens() { return 0; }
int route_order_static_max_experts() { return 0; }
cudaError_t launch_stage(const Ctx&, const void*, const void*, int, const float*, const uint8_t*, int, int, cudaStream_t) { return step("stage"); }
cudaError_t launch_route_stage(const Ctx&, const void*, const void*, int, const float*, const float*, int, const int32_t*, const int32_t*, int,
                               const uint8_t*, int, int, cudaStream_t) { return step("stage"); }
cudaError_t launch_stage_nvfp4(const void*, void*, void*, float, int64_t, int, cudaStream_t) { return step("stage"); }
cudaError_t launch_count_sort(const Ctx&, int, cudaStream_t) { return step("sort"); }
cudaError_t launch_pack(const Ctx&, int, cudaStream_t) { return step("pack"); }
cudaError_t launch_route_small(const Ctx&, int, int, int32_t*, cudaStream_t) { return step("route"); }
cudaError_t launch_route_large(const Ctx&, int, int, int32_t*, cudaStream_t) { return step("route"); }
cudaError_t launch_plan_place(const Ctx&, int, int, int32_t*, cudaStream_t) { return step("place"); }
cudaError_t launch_shared_plan(const Ctx&, int, cudaStream_t) { return step("shared"); }
cudaError_t launch_combine(const Ctx&, void*, const void*, int, cudaStream_t) { return step("combine"); }
cudaError_t zero_counters(const Ctx&, cudaStream_t) { return step("zero"); }
cudaError_t launch_experts_simt(const Ctx&, const MmoeWeights&, const MmoeOptions&, int, int, cudaStream_t) { return step("experts"); }
cudaError_t launch_experts_umma(const Ctx&, const MmoeWeights&, const MmoeOptions&, int, int, cudaStream_t) { return step("experts"); }
cudaError_t route_order_static(const int64_t*, int, int, int, int32_t*, int32_t*, int32_t*, int32_t*, cudaStream_t) { return step("order"); }
cudaError_t launch_interleave_rows(const void*, void*, int, int, int, cudaStream_t) { return step("rows"); }
cudaError_t launch_scale_layout(const int32_t*, int32_t*, int, int, int, int, int, cudaStream_t) { return step("scales"); }
cudaError_t launch_split_halves(const void*, void*, int, int64_t, int64_t, cudaStream_t) { return step("split"); }
cudaError_t launch_ep_signal_return(const Ctx&, const void* const*, int64_t, cudaStream_t) { return step("signal"); }
cudaError_t launch_ep_dispatch(const Ctx&, const void* const*, int, int64_t, cudaStream_t) { return step("dispatch"); }
cudaError_t launch_ep_return(const Ctx&, const void* const*, int64_t, cudaStream_t) { return step("return"); }
}  // namespace mmoe

// forward_sequence <tokens> <layer mask> <engine> <step that fails, or "none">: status of the call, then its steps
int main(int, char** argv) {
  const int m = atoi(argv[1]);
  g_failing = argv[4];
  const MmoeGeometry geo{1, 0, 384, 6, 5120, 2304, 1, 3840};
  char* at = reinterpret_cast<char*>(1 << 20);                       // device addresses, which no stand-in looks at
  const MmoeWeights weights{at, at, at, at, at, at, at, at, 0, 0};
  const MmoeOptions opt{10.f, 1, atoi(argv[3]), 2000, atoi(argv[2]), nullptr};
  const int rc = mmoe_forward(&geo, at, &weights, &opt, at, m, mmoe_block_m(1, 384, m, 6), nullptr, nullptr);
  printf("%d%s\n", rc, g_steps.c_str());
  return 0;
}
