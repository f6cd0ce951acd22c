// Kernels of a caller that launches programmatically in front of this library (tests/test_launch_order_gpu.py).
#include <cuda_runtime.h>

namespace {
// Lets its successor start, and writes only after a while (about a millisecond).
__global__ void late_writer(const unsigned short* from, unsigned short* to, int count) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  long long const t0 = clock64();
  while (clock64() - t0 < 2000000LL) {}
  for (int i = threadIdx.x; i < count; i += blockDim.x) to[i] = from[i];
}
// Has nothing to do with the rows.  Waits: keeps the rule that the header states.
template <bool Waits> __global__ void bystander(int* counter) {
  if (threadIdx.x == 0) atomicAdd(counter, 1);
  if (Waits) asm volatile("griddepcontrol.wait;" ::: "memory");
}
}  // namespace

extern "C" int caller_launch(const unsigned short* from, unsigned short* to, int count, int* counter, int waits, void* stream) {
  late_writer<<<1, 256, 0, static_cast<cudaStream_t>(stream)>>>(from, to, count);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = 1;
  cfg.blockDim = 32;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t const st = waits ? cudaLaunchKernelEx(&cfg, bystander<true>, counter) : cudaLaunchKernelEx(&cfg, bystander<false>, counter);
  return int(st != cudaSuccess ? st : cudaGetLastError());
}
