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

__device__ __forceinline__ float2 rounded_quotients(float2 x, float2 a, float2 r) {  // two of them, in packed instructions
  float2 const na = make_float2(-a.x, -a.y);
  float2 const q0 = __fmul2_rn(x, r);
  float2 const q1 = __ffma2_rn(__ffma2_rn(q0, na, x), r, q0);
  return __ffma2_rn(__ffma2_rn(q1, na, x), r, q1);
}

// Executed by full warps.  Where all peaks are zero or between 2^-73 and 2^106 (one vote per warp) the scale and the eight
// quotients come from reciprocals, the rounding through the bias 1.5 * 2^23 (|x / a| < 127.5, so nothing needs a clamp) and the
// codes out of the low bytes; the eight divisions of the other path are 100 instructions and leave their short form where x is
// tiny against a or zero, as behind a SwiGLU.  The largest magnitude is that of the bits, so a value that is not finite shows in it.
// Bound: issue.  Pack of bf16 rows (us, rested part): 8192 x 5120 40.6, 2048 x 17408 34.3; with scalar quotients and a finiteness test
// per value 53.6 and 45.4, with divisions 106 for the latter.
__device__ __forceinline__ Packed8 quantize8(const float (&x)[8]) {
  uint32_t top = 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i) top = max(top, __float_as_uint(x[i]) & 0x7fffffffu);
  top = max(top, __shfl_xor_sync(0xffffffffu, top, 1));
  top = max(top, __shfl_xor_sync(0xffffffffu, top, 2));
  float const peak = __uint_as_float(top);
  Packed8 r;
  if (__all_sync(0xffffffffu, top == 0u || (peak >= 0x1p-73f && peak <= 0x1p106f))) {
    constexpr float kInv127 = 1.f / 127.f;
    float const a = top == 0u ? 1.f : rounded_quotient(peak, 127.f, kInv127), inv = __frcp_rn(a);
    float2 const a2 = make_float2(a, a), inv2 = make_float2(inv, inv), bias = make_float2(12582912.f, 12582912.f);
    uint32_t t[8];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      float2 const q = __fadd2_rn(rounded_quotients(make_float2(x[i], x[i + 1]), a2, inv2), bias);
      t[i] = __float_as_uint(q.x);
      t[i + 1] = __float_as_uint(q.y);
    }
    r.w0 = __byte_perm(__byte_perm(t[0], t[1], 0x0040), __byte_perm(t[2], t[3], 0x0040), 0x5410);
    r.w1 = __byte_perm(__byte_perm(t[4], t[5], 0x0040), __byte_perm(t[6], t[7], 0x0040), 0x5410);
    int sum = __dp4a(int(r.w0), 0x01010101, __dp4a(int(r.w1), 0x01010101, 0));
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    r.valid = true;
    r.a = a;
    r.sum = sum;
    return r;
  }
  float const a = top == 0u ? 1.f : __fdiv_rn(peak, 127.f);
  r.valid = top < 0x7f800000u && a > 0.f;  // not where a peak of the smallest numbers divides to zero
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

struct Packed4x2 {
  int z[4][2];  // codes of this lane's four values of either group
  float a[2];   // scale and sum of the groups, in all eight lanes
  int sum[2];
  bool valid[2];
};

// The same for two groups (two tokens) held by the eight lanes with one lane & 3, four values of each per lane (x[i][e]: group e).
// Executed by full warps.
__device__ __forceinline__ Packed4x2 quantize4x2(const float (&x)[4][2]) {
  constexpr uint32_t kBias = 0x4B400000u;  // 1.5 * 2^23
  uint32_t top[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    top[e] = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) top[e] = max(top[e], __float_as_uint(x[i][e]) & 0x7fffffffu);
  }
#pragma unroll
  for (int off = 4; off < 32; off <<= 1)
#pragma unroll
    for (int e = 0; e < 2; ++e) top[e] = max(top[e], __shfl_xor_sync(0xffffffffu, top[e], off));
  float const p0 = __uint_as_float(top[0]), p1 = __uint_as_float(top[1]);
  Packed4x2 r;
  bool const easy = (top[0] == 0u || (p0 >= 0x1p-73f && p0 <= 0x1p106f)) && (top[1] == 0u || (p1 >= 0x1p-73f && p1 <= 0x1p106f));
  if (__all_sync(0xffffffffu, easy)) {
    constexpr float kInv127 = 1.f / 127.f;
    float2 const a2 = make_float2(top[0] == 0u ? 1.f : rounded_quotient(p0, 127.f, kInv127), top[1] == 0u ? 1.f : rounded_quotient(p1, 127.f, kInv127));
    float2 const inv2 = make_float2(__frcp_rn(a2.x), __frcp_rn(a2.y)), bias = make_float2(12582912.f, 12582912.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 const q = __fadd2_rn(rounded_quotients(make_float2(x[i][0], x[i][1]), a2, inv2), bias);
      r.z[i][0] = int(__float_as_uint(q.x) - kBias);
      r.z[i][1] = int(__float_as_uint(q.y) - kBias);
    }
    r.a[0] = a2.x;
    r.a[1] = a2.y;
    r.valid[0] = r.valid[1] = true;
  } else {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float const a = top[e] == 0u ? 1.f : __fdiv_rn(__uint_as_float(top[e]), 127.f);
      r.valid[e] = top[e] < 0x7f800000u && a > 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) r.z[i][e] = r.valid[e] ? max(-127, min(127, __float2int_rn(__fdiv_rn(x[i][e], a)))) : 0;
      r.a[e] = r.valid[e] ? a : __int_as_float(0x7fc00000);
    }
  }
  // both sums are below 2^15 in magnitude: one word carries them
  int both = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) both += r.z[i][0] + r.z[i][1] * 65536;
#pragma unroll
  for (int off = 4; off < 32; off <<= 1) both += __shfl_xor_sync(0xffffffffu, both, off);
  r.sum[0] = int(int16_t(uint16_t(uint32_t(both) & 0xffffu)));
  r.sum[1] = (both - r.sum[0]) >> 16;
  return r;
}

}  // namespace q4k
