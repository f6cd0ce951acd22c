// Max-scaled RMS norm of one row by one block (reference: hidden_rms_kernel<3>, cuda/activation.cu:134-190).
#pragma once
#include <stdint.h>

#include "common.cuh"

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

// (1 + gamma) * x / rms(x) rounded to bf16 into shared memory; hidden % 256 == 0.  Thread t owns columns t, t + 256, ... and sums
// them in that order.
//
// Bound: latency (a decode step has a handful of rows).  With Held > 0 (hidden <= 256 * Held) a thread requests its whole
// share of the row and of the gain at once and keeps it in registers for the three passes; the loop form, which serves
// wider rows, waits for memory in every iteration of every pass: 15 us at 5120 columns against 4 us.
template <int Held>
__device__ __forceinline__ void rms_row(const float* x, const uint16_t* gamma, float eps, uint32_t hidden, uint16_t* rounded) {
  __shared__ float scratch[kRmsThreads / 32];
  float held[Held > 0 ? Held : 1], gain[Held > 0 ? Held : 1];
  float scale = 0.f;
  if constexpr (Held > 0) {
#pragma unroll
    for (int j = 0; j < Held; ++j) {
      uint32_t const i = threadIdx.x + j * kRmsThreads;
      held[j] = i < hidden ? x[i] : 0.f;
      gain[j] = i < hidden ? bf16_bits_to_f32(gamma[i]) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < Held; ++j) scale = fmaxf(scale, fabsf(held[j]));
  } else {
#pragma unroll 8
    for (uint32_t i = threadIdx.x; i < hidden; i += kRmsThreads) scale = fmaxf(scale, fabsf(x[i]));
  }
  scale = block_reduce(scale, scratch, true);
  float const safe = scale == 0.f ? 1.f : scale;
  float sumsq = 0.f;
  if constexpr (Held > 0) {
#pragma unroll
    for (int j = 0; j < Held; ++j) {
      held[j] = held[j] / safe;
      if (threadIdx.x + j * kRmsThreads < hidden) sumsq += held[j] * held[j];
    }
  } else {
#pragma unroll 8
    for (uint32_t i = threadIdx.x; i < hidden; i += kRmsThreads) {
      float s = x[i] / safe;
      sumsq += s * s;
    }
  }
  sumsq = block_reduce(sumsq, scratch, false);
  float const se = sqrtf(eps) / safe;
  float const inv = 1.0f / sqrtf(sumsq / float(hidden) + se * se);
  if constexpr (Held > 0) {
#pragma unroll
    for (int j = 0; j < Held; ++j) {
      uint32_t const i = threadIdx.x + j * kRmsThreads;
      if (i < hidden) rounded[i] = f32_to_bf16_rne((1.0f + gain[j]) * (held[j] * inv));
    }
  } else {
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < hidden; i += kRmsThreads) {
      float g = bf16_bits_to_f32(gamma[i]);
      float v = (1.0f + g) * ((x[i] / safe) * inv);
      rounded[i] = f32_to_bf16_rne(v);
    }
  }
  __syncthreads();
}

}  // namespace q4k
