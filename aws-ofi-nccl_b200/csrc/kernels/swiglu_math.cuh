// silu and the logistic function as the SwiGLU kernels and the epilogues of the MLP's products use them.
//
// IEEE division is a sequence with a branch for rare operands, and elements on either side of such a branch do not
// overlap: a warp that is alone on its scheduler, as in an epilogue, took 125 clocks for each. The quotients are
// written out instead, for denominators that need no such branch: the reciprocal unit's value and one residual
// correction of the quotient (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor",
// 1990). His proof that this rounds correctly asks for a correctly rounded reciprocal, which the unit's is not: of 1.6
// billion random quotients above 2^-99 three differed from IEEE division, by one ulp. Below, the residual
// loses bits to underflow, and the quotient is within an ulp of IEEE division's (1 % differ between 2^-126 and 2^-100, 29 % of the subnormal ones). What
// errs is the exponential. Against 64
// bits, over bf16's gates within 20, silu is off by 0.16 ulp on average and the logistic function by 0.13, with IEEE
// division by 0.17 and 0.15; over normally distributed gates of 32 bits silu_ordinary by 0.82 like the division.
#pragma once

namespace b200 {

// n / d for 1 <= d < 2^126 and finite n, within an ulp of IEEE division
__device__ __forceinline__ float quotient(float n, float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = n * r;
  return fmaf(r, fmaf(-d, q, n), q);
}

// With t = exp(-|g|) the denominator lies in [1, 2] whatever the gate.
__device__ __forceinline__ float silu(float g) {
  const float t = __expf(-fabsf(g));
  const float q = quotient(g < 0.f ? g * t : g, 1.f + t);
  return g == INFINITY ? g : q;
}
__device__ __forceinline__ float logistic(float g) {
  const float t = __expf(-fabsf(g));
  return quotient(g < 0.f ? t : 1.f, 1.f + t);
}

// For gates of 32 bits, where the rounding of g * t would show: 1 + exp(-g) itself, while it is in range.
constexpr float ORDINARY_GATE = 80.f;
__device__ __forceinline__ float silu_ordinary(float g) { return quotient(g, 1.f + __expf(-g)); }
// Any gate, without a branch: below the range e^g times the gate. All gates that way, 1024 tokens x 2816 x 1024 take 16.7 us, 16.2 with
// the form above for the ordinary ones; as a call that divides as IEEE does, rare gates made 8192 x 8192 x 1024 with gates of deviation 64
// take 957 us, 194 so.
__device__ __forceinline__ float silu_any(float g) {
  const bool low = g <= -ORDINARY_GATE;
  const float t = __expf(low ? g : -g);
  const float q = quotient(low ? g * t : g, 1.f + t);
  return g == INFINITY ? g : q;
}

}  // namespace b200
