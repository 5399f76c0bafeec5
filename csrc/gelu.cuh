// GELU (erf form) and its derivative, for the elementwise passes and the GEMM epilogue.
#pragma once
#include "common.cuh"

namespace tsp {

// Phi(-|x|) = (1 - erf(|x| / sqrt 2)) / 2 through the rational form of Abramowitz & Stegun 7.1.26 (|error| <= 0.75e-7):
// one reciprocal, one exponential and six FMAs instead of the two-branch library routine.  E = exp(-x^2 / 2) is returned
// for the backward.  gelu(x) = max(x, 0) - |x| Phi(-|x|) then needs no sign handling and does not cancel for negative x.
// For 16-bit activations the hardware's approximate reciprocal and exponential do (2^-22 relative); fp32 activations take the
// correctly rounded reciprocal and exp2f.  Over every bf16 argument, alone and behind five biases, value and derivative of
// the two forms round to the same bf16 numbers but where either is the wrong neighbour, equally often (83 of 26180 values
// with |gelu| > 2^-100, 63 of 33407 derivatives; 0.5 (1 + erf x) was wrong in 117 and 97, by up to 250 units in the last
// place).  [12608, 3072] forward 35.8 us and backward 45.3, with the exact ones 54.2 and 61.7.
template <bool FAST>
__device__ __forceinline__ float upper_tail(float x, float& e_out) {
  const float z = fabsf(x) * 0.70710678118654752f;
  float t, e;
  if constexpr (FAST) {
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(0.3275911f, z, 1.f)));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * z * -1.4426950408889634f));
  } else {
    t = __frcp_rn(fmaf(0.3275911f, z, 1.f));
    e = exp2f(-1.4426950408889634f * z * z);
  }
  float p = fmaf(0.5f * 1.061405429f, t, 0.5f * -1.453152027f);
  p = fmaf(p, t, 0.5f * 1.421413741f);
  p = fmaf(p, t, 0.5f * -0.284496736f);
  p = fmaf(p, t, 0.5f * 0.254829592f);
  e_out = e;
  return p * t * e;
}
template <typename T>
__device__ __forceinline__ float gelu_f(float x) {
  float e;
  const float ax = fmaxf(-x, fminf(x, 3.402823466e38f));      // |x|, finite for +inf (whose tail is an exact zero)
  return fmaf(-ax, upper_tail<sizeof(T) == 2>(x, e), fmaxf(x, 0.f));
}
template <typename T>
__device__ __forceinline__ float gelu_grad_f(float x) {
  float e;                                        // e = exp(-x^2 / 2): the Gaussian density needs it too
  const float q = upper_tail<sizeof(T) == 2>(x, e);
  return fmaf(x * 0.3989422804014327f, e, x >= 0.f ? 1.f - q : q);
}

}  // namespace tsp
