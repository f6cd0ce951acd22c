// Quantisation of one K32 group by four neighbouring lanes, eight values each (reference: q8_pack_warp,
// cuda/q8_device.cuh:5-25):
//   peak = max |x|, a = peak == 0 ? 1 : peak / 127 (IEEE division), z = clamp(rint(x / a), -127, 127), sum = sum z.
// A group with a non-finite value (or a scale that is not positive and finite) is not valid: zero codes, NaN scale, sum 0.
#pragma once
#include <stdint.h>

namespace q4k {

struct Packed8 {
  uint32_t w0, w1;  // this lane's eight codes
  float a;          // scale and sum of the group, in all four lanes
  int sum;
  bool valid;
};

// x / a rounded to nearest, for r = 1 / a rounded to nearest: two residual corrections (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990, theorem on correctly rounded quotients: a faithful
// quotient corrected once by the rounded reciprocal is the rounded quotient; the first correction makes it faithful).
// The residual must not underflow where the result matters: the caller bounds a.
__device__ __forceinline__ float rounded_quotient(float x, float a, float r) {
  float const q0 = __fmul_rn(x, r);
  float const q1 = __fmaf_rn(__fmaf_rn(-q0, a, x), r, q0);
  return __fmaf_rn(__fmaf_rn(-q1, a, x), r, q1);
}

// Executed by full warps.  Scales between 2^-80 and 2^100 (one vote per warp) take the eight quotients through one
// reciprocal, the rounding through the bias 1.5 * 2^23 (|x / a| < 127.5, so nothing needs a clamp) and the codes out of the
// low bytes; the eight divisions of the other path are 100 instructions and leave their short form where x is tiny against
// a or zero, as behind a SwiGLU.  Pack of 2048 x 17408 bf16 rows: 106 us before, 44 with this.
__device__ __forceinline__ Packed8 quantize8(const float (&x)[8]) {
  bool finite = true;
  float peak = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    bool f = isfinite(x[i]);
    finite = finite && f;
    peak = fmaxf(peak, f ? fabsf(x[i]) : 0.f);
  }
  peak = fmaxf(peak, __shfl_xor_sync(0xffffffffu, peak, 1));
  peak = fmaxf(peak, __shfl_xor_sync(0xffffffffu, peak, 2));
  int fin = finite ? 1 : 0;
  fin &= __shfl_xor_sync(0xffffffffu, fin, 1);
  fin &= __shfl_xor_sync(0xffffffffu, fin, 2);
  float const a = peak == 0.f ? 1.f : __fdiv_rn(peak, 127.f);
  Packed8 r;
  r.valid = fin && isfinite(a) && a > 0.f;
  if (__all_sync(0xffffffffu, a >= 0x1p-80f && a <= 0x1p100f)) {
    float const inv = __frcp_rn(a);
    uint32_t t[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = __float_as_uint(__fadd_rn(rounded_quotient(x[i], a, inv), 12582912.f));
    r.w0 = __byte_perm(__byte_perm(t[0], t[1], 0x0040), __byte_perm(t[2], t[3], 0x0040), 0x5410);
    r.w1 = __byte_perm(__byte_perm(t[4], t[5], 0x0040), __byte_perm(t[6], t[7], 0x0040), 0x5410);
    if (!r.valid) r.w0 = r.w1 = 0u;  // a value that is not finite
    int sum = __dp4a(int(r.w0), 0x01010101, __dp4a(int(r.w1), 0x01010101, 0));
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    r.a = r.valid ? a : __int_as_float(0x7fc00000);
    r.sum = sum;
    return r;
  }
  int z[8];
  int sum = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    z[i] = r.valid ? max(-127, min(127, __float2int_rn(__fdiv_rn(x[i], a)))) : 0;
    sum += z[i];
  }
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);
  sum += __shfl_xor_sync(0xffffffffu, sum, 2);
  r.w0 = (uint32_t(z[0]) & 255u) | ((uint32_t(z[1]) & 255u) << 8) | ((uint32_t(z[2]) & 255u) << 16) | ((uint32_t(z[3]) & 255u) << 24);
  r.w1 = (uint32_t(z[4]) & 255u) | ((uint32_t(z[5]) & 255u) << 8) | ((uint32_t(z[6]) & 255u) << 16) | ((uint32_t(z[7]) & 255u) << 24);
  r.a = r.valid ? a : __int_as_float(0x7fc00000);
  r.sum = sum;
  return r;
}

}  // namespace q4k
