// The two SwiGLU quotients of the library against the divisions they stand for, over every float.  The pack's quotient of -0 is
// +0, the only difference: neither sign changes a code, a scale or a sum.
#include <cstdio>

#include "../../qw38_b200/csrc/decode_entry.cu"
#include "../../qw38_b200/csrc/q8_quantize.cu"

namespace q4k {
bool launch_overlap() { return false; }
namespace {

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (isnan(a) && isnan(b)); }

__global__ void compare(unsigned long long* differ) {
  uint32_t const threads = gridDim.x * blockDim.x;
  unsigned long long pack = 0, store = 0;
  for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32); i += threads) {
    float const g = __uint_as_float(uint32_t(i));
    float const x = silu(g), want = __fdiv_rn(g, __fadd_rn(1.f, expf(-g)));
    pack += isfinite(g) ? !same(x, want) && (x != 0.f || want != 0.f || __float_as_uint(g) != 0x80000000u) : isfinite(x);
    float const e = expf(-fabsf(g));
    store += !same(sigmoid_fp32(g), __fdiv_rn(g >= 0.f ? 1.f : e, __fadd_rn(1.f, e)));
  }
  if (pack) atomicAdd(differ, pack);
  if (store) atomicAdd(differ + 1, store);
}

}  // namespace
}  // namespace q4k

int main() {
  unsigned long long* differ = nullptr;
  unsigned long long host[2] = {~0ull, ~0ull};
  cudaMalloc(&differ, sizeof host);
  cudaMemset(differ, 0, sizeof host);
  q4k::compare<<<148 * 8, 256>>>(differ);
  cudaMemcpy(host, differ, sizeof host, cudaMemcpyDeviceToHost);
  std::printf("differ: pack %llu, store %llu, %s\n", host[0], host[1], cudaGetErrorString(cudaGetLastError()));
  return host[0] || host[1];
}
