// Activation producers: bf16/fp32 rows -> Q8 (int8 codes, fp32 scale, int32 sum per 32),
// the fused RMS-norm and SwiGLU producers, and the 36-byte record export.
//
// The arithmetic of a group is in q8_pack.cuh; columns >= k count as 0.  An invalid group raises the failure flag.
//
// Mapping: four lanes own one K32 group, eight values per lane, so a warp covers
// 256 consecutive columns with 16-byte loads and 8-byte stores.
#include <cuda_bf16.h>

#include "common.cuh"
#include "launch.h"
#include "q8_pack.cuh"
#include "rms.cuh"
#include "swiglu.cuh"

namespace q4k {
namespace {

constexpr int kThreads = kRmsThreads, kBlocksPerSm = 6;

// Quantise the eight values of this lane; lanes (4j..4j+3) share a group.
__device__ __forceinline__ void pack8(const float (&x)[8], int8_t* codes, float* scales,
                                      int32_t* sums, uint64_t group, uint32_t sub, int* failure) {
  Packed8 const r = quantize8(x);
  uint32_t* dst = reinterpret_cast<uint32_t*>(codes + group * 32 + sub * 8);
  dst[0] = r.w0;
  dst[1] = r.w1;
  if (sub == 0) {
    scales[group] = r.a;
    sums[group] = r.sum;
    if (!r.valid) atomicExch(failure, 1);
  }
}

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<uint16_t>(uint16_t v) { return bf16_bits_to_f32(v); }
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }

// Vec: rows start 16-byte aligned and k % 8 == 0, so a lane's eight values are
// one (bf16) or two (fp32) aligned 16-byte loads.
template <typename T, bool Vec>
__device__ __forceinline__ void load8(const T* src, uint32_t col0, uint32_t k, float (&x)[8]) {
  if (Vec && col0 + 8 <= k) {
    if constexpr (sizeof(T) == 2) {
      uint4 v = *reinterpret_cast<const uint4*>(src + col0);
      uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[2 * i] = __uint_as_float(w[i] << 16);
        x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
      }
    } else {
      float4 lo = *reinterpret_cast<const float4*>(src + col0);
      float4 hi = *reinterpret_cast<const float4*>(src + col0 + 4);
      x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w;
      x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = col0 + i < k ? to_f32<T>(src[col0 + i]) : 0.f;
  }
}

// A warp takes 256 columns of a row at a time; the next ones are requested before the present ones are quantised.
template <typename T, bool Vec>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) pack_kernel(const T* in, int8_t* __restrict__ codes,
                                                                       float* __restrict__ scales, int32_t* __restrict__ sums, uint32_t m,
                                                                       uint32_t k, uint32_t pk, int* failure) {
  uint32_t const lane = threadIdx.x & 31, sub = lane & 3, grp = lane >> 2;
  uint32_t const chunks_row = pk / 256, tasks = m * chunks_row;  // below 2^32 for every accepted shape
  uint32_t const warps = gridDim.x * (kThreads / 32);
  uint32_t task = blockIdx.x * (kThreads / 32) + threadIdx.x / 32;
  if (task < tasks && lane * 8 % (128 / sizeof(T)) == 0) {
    uint32_t const col = task % chunks_row * 256 + lane * 8;
    if (col < k) prefetch_line(in + uint64_t(task / chunks_row) * k + col);
  }
  pdl_wait();               // the input may come from the kernel before this one
  pdl_launch_dependents();  // the projection that follows may start prefetching its weights (after the wait: the
                            // next launch never runs beside anything older than this one)
  float x[8], next[8];
  auto load = [&](uint32_t t, float (&to)[8]) { load8<T, Vec>(in + uint64_t(t / chunks_row) * k, t % chunks_row * 256 + lane * 8, k, to); };
  if (task < tasks) load(task, x);
  for (; task < tasks; task += warps) {
    bool const more = task + warps < tasks;
    if (more) load(task + warps, next);
    pack8(x, codes, scales, sums, uint64_t(task) * 8 + grp, sub, failure);
    if (more) {
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = next[i];
    }
  }
}

// v = bf16_rne(silu(g) * u); non-finite g or u poisons the value
// (reference: swiglu_pack_kernel, cuda/q4k_q8.cu:52-61).  ffn % 256 == 0.
__global__ void __launch_bounds__(kThreads) swiglu_pack_kernel(const float* gate, const float* up,
                                                                int8_t* __restrict__ codes, float* __restrict__ scales,
                                                                int32_t* __restrict__ sums, uint64_t chunks,
                                                                int* failure) {
  pdl_wait();
  pdl_launch_dependents();
  uint32_t const lane = threadIdx.x & 31, sub = lane & 3, grp = lane >> 2;
  uint64_t const warps = uint64_t(gridDim.x) * (kThreads / 32);
  for (uint64_t task = uint64_t(blockIdx.x) * (kThreads / 32) + threadIdx.x / 32; task < chunks;
       task += warps) {
    uint64_t const i0 = task * 256 + grp * 32 + sub * 8;
    float4 g0 = *reinterpret_cast<const float4*>(gate + i0), g1 = *reinterpret_cast<const float4*>(gate + i0 + 4);
    float4 u0 = *reinterpret_cast<const float4*>(up + i0), u1 = *reinterpret_cast<const float4*>(up + i0 + 4);
    float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
    float u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
    float x[8];
    swiglu8(g, u, x);  // what is not finite makes the group invalid
    pack8(x, codes, scales, sums, task * 8 + grp, sub, failure);
  }
}

// RMS norm, then the Q8 pack of the rounded row.  One block per token; dynamic shared memory = the scaled row as floats (Held), or the
// rounded one.
template <bool Held>
__global__ void __launch_bounds__(Held ? kRmsHeldColumns / 8 : kThreads) hidden_rms_q8_kernel(const float* residual, const uint16_t* gamma,
                                                                                             float eps, uint32_t hidden, bool vec,
                                                                                             int8_t* codes, float* scales,
                                                                                             int32_t* sums, int* failure) {
  extern __shared__ __align__(16) uint8_t row[];
  const float* const x = residual + uint64_t(blockIdx.x) * hidden;
  rms_prefetch(x, gamma, hidden);
  pdl_wait();
  pdl_launch_dependents();
  uint32_t const lane = threadIdx.x & 31, sub = lane & 3, grp = lane >> 2;
  uint64_t const group0 = uint64_t(blockIdx.x) * (hidden / 32) + grp;
  float v[8];
  if constexpr (Held) {
    rms_row_held(x, gamma, eps, hidden, vec, reinterpret_cast<float*>(row), v);
    if (threadIdx.x * 8 < hidden) pack8(v, codes, scales, sums, group0 + threadIdx.x / 32 * 8, sub, failure);
  } else {
    uint16_t* const rounded = reinterpret_cast<uint16_t*>(row);
    rms_row(x, gamma, eps, hidden, rounded);
    for (uint32_t chunk = threadIdx.x / 32; chunk < hidden / 256; chunk += kThreads / 32) {
      uint32_t const col0 = chunk * 256 + grp * 32 + sub * 8;
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = bf16_bits_to_f32(rounded[col0 + i]);
      pack8(v, codes, scales, sums, group0 + chunk * 8, sub, failure);
    }
  }
}

// One thread per K32 group: {fp16 d = a, fp16 s = a * sum, 32 codes}.
__global__ void export_q8_1_kernel(const int8_t* __restrict__ codes, const float* __restrict__ scales,
                                   const int32_t* __restrict__ sums, uint64_t groups,
                                   uint32_t* __restrict__ records) {
  uint64_t g = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (g >= groups) return;
  float a = scales[g];
  uint32_t d = __half_as_ushort(__float2half_rn(a));
  uint32_t s = __half_as_ushort(__float2half_rn(a * float(sums[g])));
  uint32_t* dst = records + g * 9;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(codes + g * 32);
  dst[0] = d | (s << 16);
#pragma unroll
  for (int i = 0; i < 8; ++i) dst[1 + i] = src[i];
}

int grid_for(uint64_t tasks) {
  uint64_t blocks = (tasks + kThreads / 32 - 1) / (kThreads / 32);
  if (blocks > uint64_t(148 * kBlocksPerSm)) blocks = 148 * kBlocksPerSm;
  return int(blocks ? blocks : 1);
}

}  // namespace

cudaError_t launch_pack_q8(const void* input, bool fp32, Q8Out out, uint32_t k, int* failure,
                           cudaStream_t stream) {
  uint64_t const tasks = uint64_t(out.m) * (out.padded_k / 256);
  int const grid = grid_for(tasks);
  bool const vec = (k % 8 == 0) && (reinterpret_cast<uintptr_t>(input) % 16 == 0);
  if (fp32) {
    auto* in = static_cast<const float*>(input);
    if (vec) return launch_kernel(pack_kernel<float, true>, grid, kThreads, 0, stream, true, in, out.codes, out.scales, out.sums, out.m, k, out.padded_k, failure);
    else return launch_kernel(pack_kernel<float, false>, grid, kThreads, 0, stream, true, in, out.codes, out.scales, out.sums, out.m, k, out.padded_k, failure);
  } else {
    auto* in = static_cast<const uint16_t*>(input);
    if (vec) return launch_kernel(pack_kernel<uint16_t, true>, grid, kThreads, 0, stream, true, in, out.codes, out.scales, out.sums, out.m, k, out.padded_k, failure);
    else return launch_kernel(pack_kernel<uint16_t, false>, grid, kThreads, 0, stream, true, in, out.codes, out.scales, out.sums, out.m, k, out.padded_k, failure);
  }
  return cudaGetLastError();
}

cudaError_t launch_swiglu_pack_q8(const float* gate, const float* up, Q8Out out, int* failure,
                                  cudaStream_t stream) {
  uint64_t const chunks = uint64_t(out.m) * (out.padded_k / 256);
  return launch_kernel(swiglu_pack_kernel, grid_for(chunks), kThreads, 0, stream, true, gate, up, out.codes, out.scales, out.sums,
                       chunks, failure);
}

cudaError_t launch_hidden_rms_q8(const float* residual, const uint16_t* gamma, float eps,
                                 uint32_t hidden, Q8Out out, int* failure, cudaStream_t stream) {
  bool const held = hidden <= kRmsHeldColumns;
  size_t const smem = size_t(hidden) * (held ? 4 : 2);
  auto kernel = held ? hidden_rms_q8_kernel<true> : hidden_rms_q8_kernel<false>;
  if (smem > 48 * 1024) {
    cudaError_t st = allow_smem(reinterpret_cast<const void*>(kernel), int(smem));
    if (st != cudaSuccess) return st;
  }
  return launch_kernel(kernel, out.m, held ? rms_held_threads(hidden) : kThreads, smem, stream, true, residual, gamma, eps, hidden,
                       rms_vector_rows(residual, gamma), out.codes, out.scales, out.sums, failure);
}

cudaError_t launch_export_q8_1(const int8_t* codes, const float* scales, const int32_t* sums,
                               uint64_t groups, uint8_t* records, cudaStream_t stream) {
  uint64_t const blocks = (groups + 255) / 256;
  export_q8_1_kernel<<<unsigned(blocks), 256, 0, stream>>>(codes, scales, sums, groups, reinterpret_cast<uint32_t*>(records));
  return cudaGetLastError();
}

}  // namespace q4k
