// A kernel that lets its successor start at once and writes its output a while later, as a programmatic chain allows: the
// successor has to wait before it reads.  Test helper.
#include <cuda_runtime.h>
#include <stdint.h>

namespace {
__device__ uint64_t now() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__global__ void late_writer(uint4* dst, const uint4* src, int64_t vecs, int64_t delay_ns) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint64_t t0 = now();
  for (int i = 0; i < 100000 && now() - t0 < static_cast<uint64_t>(delay_ns); ++i) __nanosleep(500);
  for (int64_t i = threadIdx.x; i < vecs; i += blockDim.x) dst[i] = src[i];
}
}  // namespace

extern "C" int late_write(void* dst, const void* src, int64_t bytes, int64_t delay_ns, void* stream) {
  late_writer<<<1, 1024, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<uint4*>(dst), static_cast<const uint4*>(src), bytes / 16, delay_ns);
  return static_cast<int>(cudaGetLastError());
}
