// The two SiLU forms of the library, their quotients through one reciprocal and a residual correction.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

#include "q8_pack.cuh"

namespace q4k {

// g / (1 + exp(-g)), rounded as the division would be (-0 gives +0, which changes no code).  A divisor above 2^64 is scaled
// (exactly: the quotient of a finite g stays a normal number) and an infinite one replaced, so that no residual of the quotient
// underflows.  Not finite for a g that is not.  (The MLP chain's form: swiglu_pack_kernel, cuda/q4k_q8.cu:52-61.)
__device__ __forceinline__ float silu(float g) {
  float const d = 1.f + expf(-g);
  bool const far = d > 0x1p64f, lost = isinf(d);
  float const by = lost ? 1.f : (far ? d * 0x1p-64f : d);
  return rounded_quotient(g, by, __frcp_rn(by)) * (lost ? 0.f : (far ? 0x1p-64f : 1.f));
}

// x = bf16_rne(silu(g) * u) as floats; what is not finite stays so.
__device__ __forceinline__ void swiglu8(const float (&g)[8], const float (&u)[8], float (&x)[8]) {
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    __nv_bfloat162 const v = __floats2bfloat162_rn(silu(g[i]) * u[i], silu(g[i + 1]) * u[i + 1]);
    uint32_t const w = *reinterpret_cast<const uint32_t*>(&v);
    x[i] = __uint_as_float(w << 16);
    x[i + 1] = __uint_as_float(w & 0xffff0000u);
  }
}

// sigmoid / SiLU exactly as the reference's decode epilogue states them
// (cuda/decode_mmv.cu:78-89): the exponential is always taken of a non-positive number.
__device__ __forceinline__ float sigmoid_fp32(float u) {
  // below 2^-24 the divisor is 1; the others are between 1 and 2, their quotient rounded as the division would be
  float const e = expf(-fabsf(u)), d = 1.0f + e, n = u >= 0.0f ? 1.0f : e;
  return d == 1.0f ? n : rounded_quotient(n, d, __frcp_rn(d));
}

}  // namespace q4k
