// Vectors of eight bf16, and the arithmetic of the softmax cross-entropy on them.
#pragma once
#include <cuda_bf16.h>
#include <float.h>
#include <stdint.h>

namespace b200 {

using bf16 = __nv_bfloat16;
using bf162 = __nv_bfloat162;

struct alignas(16) Bf16x8 {
  bf162 v[4];
};
__device__ __forceinline__ void unpack8(const Bf16x8& p, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __low2float(p.v[i]);
    f[2 * i + 1] = __high2float(p.v[i]);
  }
}
__device__ __forceinline__ Bf16x8 pack8(const float (&f)[8]) {
  Bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}

// ------------------------------------------------------------------ cross-entropy
// Exponentials are powers of two of f * log2(e) - c, one fused multiply-add: c is the maximum times log2(e), rounded, the
// same for every term, and the loss adds what the rounding left out. Taking the maximum off first is one instruction more, and registers that the
// row kernel does not have: 69 us for 4096 x 16040, 57 this way. Maxima start below all bf16 but -inf, so that masked elements of that value
// count as nothing.
constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Powers below 2^-126 are zero: several instructions less. What they are added to is at least one of the sums' own powers, 2^0.
__device__ __forceinline__ float exp2_flushed(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// From here on a finite maximum's product with log2(e) may overflow (masks are often the lowest bf16). Neighbouring values lie 1e36
// apart there: e^(f - m) is 1 or 0.
__device__ __forceinline__ bool huge_max(float m) { return fabsf(m) >= 2e38f && m < INFINITY; }
__device__ __forceinline__ float exp_base(float m) { return __fmul_rn(m, LOG2E); }
// A value relative to a huge maximum, as an argument for the base 0
__device__ __forceinline__ bf16 from_huge(bf16 x, float m) {
  const float f = __bfloat162float(x);
  return __float2bfloat16(f == m ? 0.f : f < m ? -INFINITY : f);
}
// What a sum relative to the maximum `part` counts relative to m
__device__ __forceinline__ float exp_share(float part, float m) {
  const float scale = huge_max(m) ? 1.f : LOG2E;
  return exp2_approx(__fmul_rn(part, scale) - __fmul_rn(m, scale));
}
// The largest of eight values, NaN left aside.
__device__ __forceinline__ float max8(const Bf16x8& x) {
  const bf162 m = __hmax2(__hmax2(x.v[0], x.v[1]), __hmax2(x.v[2], x.v[3]));
  return fmaxf(__low2float(m), __high2float(m));
}
__device__ __forceinline__ float exp_sum8(const Bf16x8& x, float c) {
  float f[8], s = 0.f;
  unpack8(x, f);
#pragma unroll
  for (int j = 0; j < 8; ++j) s += exp2_flushed(fmaf(f[j], LOG2E, -c));
  return s;
}
// s: the sum relative to exp_base(m), or to m itself where that is huge
__device__ __forceinline__ float ce_loss(float m, float s, float target_logit) {
  return logf(s) + (m - target_logit) + (huge_max(m) ? 0.f : fmaf(m, -LOG2E, exp_base(m)) * LN2);
}
// Whether a power below 2^-126 times inv can be a bf16 (of which the smallest is 2^-133) other than zero
__device__ __forceinline__ bool small_powers_count(float inv) { return !(fabsf(inv) <= 0x1p-8f); }
// `own`: the target's place among the eight elements, if it is one of them; SMALL: small_powers_count
template <bool SMALL>
__device__ __forceinline__ Bf16x8 ce_gradient8(const Bf16x8& x, float c, float inv, int own, float grad_scale) {
  float f[8];
  unpack8(x, f);
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = (SMALL ? exp2_approx(fmaf(f[j], LOG2E, -c)) : exp2_flushed(fmaf(f[j], LOG2E, -c))) * inv;
  if (own >= 0 && own < 8) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (own == j) f[j] -= grad_scale;
  }
  return pack8(f);
}

// The same where the maximum is huge or small powers count, out of the loops that every other row runs. Vectors are passed in registers.
__device__ __noinline__ float exp_sum8_huge(uint4 v, float m) {
  const Bf16x8 x = *reinterpret_cast<const Bf16x8*>(&v);
  float f[8], s = 0.f;
  unpack8(x, f);
#pragma unroll
  for (int j = 0; j < 8; ++j) s += __expf(f[j] - m);
  return s;
}
__device__ __noinline__ uint4 ce_gradient8_special(uint4 v, float m, float inv, int own, float grad_scale) {
  const Bf16x8 x = *reinterpret_cast<const Bf16x8*>(&v);
  Bf16x8 o;
  if (huge_max(m)) {
    float f[8];
    unpack8(x, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = __expf(f[j] - m) * inv - (own == j ? grad_scale : 0.f);
    o = pack8(f);
  } else {
    o = ce_gradient8<true>(x, exp_base(m), inv, own, grad_scale);
  }
  return *reinterpret_cast<const uint4*>(&o);
}

}  // namespace b200
