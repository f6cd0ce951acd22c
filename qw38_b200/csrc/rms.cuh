// Max-scaled RMS norm of one row by one block (reference: hidden_rms_kernel<3>, cuda/activation.cu:134-190).
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

#include "common.cuh"
#include "q8_pack.cuh"

namespace q4k {

constexpr int kRmsThreads = 256;

__device__ __forceinline__ float block_reduce(float v, float* scratch, bool is_max) {
  for (int off = 16; off; off >>= 1) {
    float o = __shfl_xor_sync(0xffffffffu, v, off);
    v = is_max ? fmaxf(v, o) : v + o;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = scratch[0];
  for (int i = 1; i < kRmsThreads / 32; ++i) r = is_max ? fmaxf(r, scratch[i]) : r + scratch[i];
  return r;
}

// (1 + gamma) * x / rms(x) rounded to bf16; hidden % 256 == 0.  The squares of columns t, t + 256, ... are summed in that order for
// t = 0 .. 255, then over t: both forms give the same bits.
//
// Bound: latency (a decode step has a handful of rows).  Up to kRmsHeldColumns a thread holds eight consecutive columns from the load to
// the pack (a block of hidden / 8 threads, 256 at least): one load of row and gain, two block reductions, and only the scaled row goes
// through shared memory, where the first 256 threads find the columns whose squares they sum.  Against 256 threads with 24 columns each
// (three passes over registers and the pack out of shared memory in three rounds), MLP chains 5120 / 17408,
// us: one token 45.0 -> 42.0, four 48.8 -> 46.1, thirteen 58.3 -> 56.5;
// with quotients through a reciprocal 56.0.  From the wait to the end 3.4 to 4.6 us, of which 1 to 2 fetch the code, which a layer's weights
// drive out of L2.
constexpr uint32_t kRmsHeldColumns = 8192;
__host__ __device__ constexpr uint32_t rms_held_threads(uint32_t hidden) { return hidden / 8 > kRmsThreads ? hidden / 8 : kRmsThreads; }

inline bool rms_vector_rows(const float* residual, const uint16_t* gamma) {
  return (reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(gamma)) % 16 == 0;  // rows are multiples of 1024 bytes
}

// Asks L2 for a thread's share; before the wait for what writes the row.
__device__ __forceinline__ void rms_prefetch(const float* x, const uint16_t* gamma, uint32_t hidden) {
  uint32_t const col = threadIdx.x * 8;
  if (col < hidden && threadIdx.x % 4 == 0) prefetch_line(x + col);
  if (col < hidden && threadIdx.x % 8 == 0) prefetch_line(gamma + col);
}

// Thread t's columns 8t .. 8t + 7 as bf16 values in v (zeros beyond the row); scaled: shared memory, hidden floats.  vec: row and gain are
// 16-byte aligned.
__device__ __forceinline__ void rms_row_held(const float* x, const uint16_t* gamma, float eps, uint32_t hidden, bool vec, float* scaled,
                                             float (&v)[8]) {
  __shared__ uint32_t tops[32];
  __shared__ float4 sums[2];
  uint32_t const t = threadIdx.x, lane = t & 31, warp = t >> 5, col = t * 8;
  bool const live = col < hidden;  // whole warps
  uint32_t gain[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = 0.f;
  if (live) {
    if (vec) {
      float4 const lo = *reinterpret_cast<const float4*>(x + col), hi = *reinterpret_cast<const float4*>(x + col + 4);
      uint4 const g = *reinterpret_cast<const uint4*>(gamma + col);
      v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
      gain[0] = g.x; gain[1] = g.y; gain[2] = g.z; gain[3] = g.w;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = x[col + i];
#pragma unroll
      for (int i = 0; i < 4; ++i) gain[i] = uint32_t(gamma[col + 2 * i]) | uint32_t(gamma[col + 2 * i + 1]) << 16;
    }
  }
  float top = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) top = fmaxf(top, fabsf(v[i]));  // never a NaN, so its bits compare as it does
  uint32_t const warp_top = __reduce_max_sync(0xffffffffu, __float_as_uint(top));
  if (lane == 0) tops[warp] = warp_top;
  __syncthreads();
  float const scale = __uint_as_float(__reduce_max_sync(0xffffffffu, lane < blockDim.x / 32 ? tops[lane] : 0u));
  float const safe = scale == 0.f ? 1.f : scale;
  // The quotients through one reciprocal, bitwise the divisions (q8_pack.cuh) where neither a quotient nor its residual is subnormal.
  float least = 1.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) least = fminf(least, v[i] == 0.f ? 1.f : fabsf(v[i]));
  if (__all_sync(0xffffffffu, least >= 0x1p-90f && safe >= 0x1p-60f && safe <= 0x1p30f)) {
    float const r = __frcp_rn(safe);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      float2 const s = rounded_quotients(make_float2(v[i], v[i + 1]), make_float2(safe, safe), make_float2(r, r));
      v[i] = s.x;
      v[i + 1] = s.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = v[i] / safe;
  }
  if (live) {
    *reinterpret_cast<float4*>(scaled + col) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(scaled + col + 4) = make_float4(v[4], v[5], v[6], v[7]);
  }
  __syncthreads();
  if (t < kRmsThreads) {
    float sumsq = 0.f;
#pragma unroll 4
    for (uint32_t i = t; i < hidden; i += kRmsThreads) sumsq += scaled[i] * scaled[i];
#pragma unroll
    for (int off = 16; off; off >>= 1) sumsq += __shfl_xor_sync(0xffffffffu, sumsq, off);
    if (lane == 0) reinterpret_cast<float*>(sums)[warp] = sumsq;
  }
  float const se = sqrtf(eps) / safe;
  __syncthreads();
  float4 const s0 = sums[0], s1 = sums[1];
  float const sumsq = s0.x + s0.y + s0.z + s0.w + s1.x + s1.y + s1.z + s1.w;
  float const inv = 1.0f / sqrtf(sumsq / float(hidden) + se * se);
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    float const g0 = __uint_as_float(gain[i / 2] << 16), g1 = __uint_as_float(gain[i / 2] & 0xffff0000u);
    __nv_bfloat162 const both = __floats2bfloat162_rn((1.0f + g0) * (v[i] * inv), (1.0f + g1) * (v[i + 1] * inv));
    uint32_t const w = *reinterpret_cast<const uint32_t*>(&both);
    v[i] = __uint_as_float(w << 16);
    v[i + 1] = __uint_as_float(w & 0xffff0000u);
  }
}

// Wider rows, into shared memory: 256 threads in passes over memory.
__device__ __forceinline__ void rms_row(const float* x, const uint16_t* gamma, float eps, uint32_t hidden, uint16_t* rounded) {
  __shared__ float scratch[kRmsThreads / 32];
  float scale = 0.f;
#pragma unroll 8
  for (uint32_t i = threadIdx.x; i < hidden; i += kRmsThreads) scale = fmaxf(scale, fabsf(x[i]));
  scale = block_reduce(scale, scratch, true);
  float const safe = scale == 0.f ? 1.f : scale;
  float sumsq = 0.f;
#pragma unroll 8
  for (uint32_t i = threadIdx.x; i < hidden; i += kRmsThreads) {
    float s = x[i] / safe;
    sumsq += s * s;
  }
  sumsq = block_reduce(sumsq, scratch, false);
  float const se = sqrtf(eps) / safe;
  float const inv = 1.0f / sqrtf(sumsq / float(hidden) + se * se);
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < hidden; i += kRmsThreads) {
    float g = bf16_bits_to_f32(gamma[i]);
    float v = (1.0f + g) * ((x[i] / safe) * inv);
    rounded[i] = f32_to_bf16_rne(v);
  }
  __syncthreads();
}

}  // namespace q4k
