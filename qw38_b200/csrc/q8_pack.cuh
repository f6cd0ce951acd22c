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

// Executed by full warps.
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
