// Epilogue kernels of the decode entry points (q4k_decode_mmv, _paired, _ranges): the four
// DecodeEpilogue forms of the reference (cuda/decode_mmv.hpp:45-51) applied to fp32 projection
// rows.  StoreFp32 and ResidualAddFp32 need no kernel of their own: the projection writes the
// destination directly (the residual is its last fp32 add, cuda/q4k_q8.cu:100).
#include <cuda_bf16.h>

#include "common.cuh"
#include "launch.h"
#include "swiglu.cuh"

namespace q4k {
namespace {

__global__ void store_bf16_kernel(const float* in, uint16_t* __restrict__ out, uint64_t count) {
  pdl_wait();
  pdl_launch_dependents();  // after the wait: the next launch never runs beside anything older than this one
  uint64_t const i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < count) out[i] = f32_to_bf16_rne(in[i]);
}

// y = bf16(SiLU(gate) * up)  (SwigluStoreBf16, cuda/decode_mmv.cu:238-242).  Bound: HBM beyond a few hundred tokens, 10
// bytes per value; Wide (all pointers 16-byte aligned, count a multiple of eight): eight values per thread, four loads in
// flight.  2048 x 17408: 53 us, 112 before (one value per thread, a division that left its short form, rounding in software).
template <bool Wide>
__global__ void swiglu_store_bf16_kernel(const float* gate, const float* up,
                                         uint16_t* __restrict__ out, uint64_t count) {
  pdl_wait();
  pdl_launch_dependents();  // after the wait: the next launch never runs beside anything older than this one
  uint64_t const i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if constexpr (Wide) {
    if (i >= count / 8) return;
    float4 const g0 = reinterpret_cast<const float4*>(gate)[2 * i], g1 = reinterpret_cast<const float4*>(gate)[2 * i + 1];
    float4 const u0 = reinterpret_cast<const float4*>(up)[2 * i], u1 = reinterpret_cast<const float4*>(up)[2 * i + 1];
    float const g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w}, u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float const a = g[2 * j] * sigmoid_fp32(g[2 * j]) * u[2 * j], b = g[2 * j + 1] * sigmoid_fp32(g[2 * j + 1]) * u[2 * j + 1];
      __nv_bfloat162 const v = __floats2bfloat162_rn(a, b);
      w[j] = *reinterpret_cast<const uint32_t*>(&v);
      if (isnan(a) || isnan(b)) w[j] = uint32_t(f32_to_bf16_rne(a)) | uint32_t(f32_to_bf16_rne(b)) << 16;  // NaNs keep their bits
    }
    reinterpret_cast<uint4*>(out)[i] = make_uint4(w[0], w[1], w[2], w[3]);
  } else if (i < count) {
    float const g = gate[i];
    out[i] = f32_to_bf16_rne(g * sigmoid_fp32(g) * up[i]);
  }
}

}  // namespace

cudaError_t launch_store_bf16(const float* in, uint16_t* out, uint64_t count, cudaStream_t stream) {
  if (count == 0) return cudaSuccess;
  return launch_kernel(store_bf16_kernel, unsigned((count + 255) / 256), 256, 0, stream, true, in, out, count);
}

cudaError_t launch_swiglu_store_bf16(const float* gate, const float* up, uint16_t* out, uint64_t count, cudaStream_t stream) {
  if (count == 0) return cudaSuccess;
  bool const wide = count % 8 == 0 && ((reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(up) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  uint64_t const threads = wide ? count / 8 : count;
  return launch_kernel(wide ? swiglu_store_bf16_kernel<true> : swiglu_store_bf16_kernel<false>, unsigned((threads + 255) / 256), 256, 0, stream,
                       true, gate, up, out, count);
}

}  // namespace q4k
