// GELU (erf form) and its derivative, for the elementwise passes and the GEMM epilogue.
#pragma once
#include "common.cuh"

namespace tsp {

// Phi(-|x|) = (1 - erf(|x| / sqrt 2)) / 2 through the rational form of Abramowitz & Stegun 7.1.26 (|error| <= 0.75e-7):
// one reciprocal, one exponential and six FMAs instead of the two-branch library routine.  E = exp(-x^2 / 2) is returned
// for the backward.  gelu(x) = max(x, 0) - |x| Phi(-|x|) then needs no sign handling and does not cancel for negative x.
// fp32 activations take the correctly rounded reciprocal and exp2f.
__device__ __forceinline__ float upper_tail(float x, float& e_out) {
  const float z = fabsf(x) * 0.70710678118654752f;
  const float t = __frcp_rn(fmaf(0.3275911f, z, 1.f)), e = exp2f(-1.4426950408889634f * z * z);
  float p = fmaf(0.5f * 1.061405429f, t, 0.5f * -1.453152027f);
  p = fmaf(p, t, 0.5f * 1.421413741f);
  p = fmaf(p, t, 0.5f * -0.284496736f);
  p = fmaf(p, t, 0.5f * 0.254829592f);
  e_out = e;
  return p * t * e;
}
__device__ __forceinline__ float gelu_f(float x) {
  float e;
  const float ax = fmaxf(-x, fminf(x, 3.402823466e38f));      // |x|, finite for +inf (whose tail is an exact zero)
  return fmaf(-ax, upper_tail(x, e), fmaxf(x, 0.f));
}
__device__ __forceinline__ float gelu_grad_f(float x) {
  float e;                                        // e = exp(-x^2 / 2): the Gaussian density needs it too
  const float q = upper_tail(x, e);
  return fmaf(x * 0.3989422804014327f, e, x >= 0.f ? 1.f - q : q);
}

// The same for two values of 16-bit activations, two to an instruction where there is one for two.  The hardware's approximate
// reciprocal and exponential do here (2^-22 relative): of 26180 bf16 arguments with |gelu| > 2^-100 83 have the wrong neighbour for
// a result, of 33407 derivatives 63 (0.5 (1 + erf x) was wrong in 117 and 97, by up to 250 units in the last place).  The passes move
// at close to the memory's rate, the GEMM epilogue waits for its own instructions.  B200, [12608, 3072]: forward 36.9 us, one
// value to an instruction 38.9, with the exact reciprocal and exponential 54.2; backward 48.7, 50.3 and 61.7; a product of K = 768 with
// this epilogue 74.8 and 78.8 (16384 rows, one output: 83.0 and 87.0).
__device__ __forceinline__ Pair upper_tail(Pair x, Pair& e_out) {
  auto both = [](float c) { return Pair(c, c); };
  const Pair z = x * both(0.70710678118654752f), power = z * z * both(-1.4426950408889634f);
  float z0, z1, s0, s1, t0, t1, e0, e1;
  z.split(z0, z1);
  power.split(s0, s1);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t0) : "f"(fmaf(0.3275911f, fabsf(z0), 1.f)));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t1) : "f"(fmaf(0.3275911f, fabsf(z1), 1.f)));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(s0));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(s1));
  const Pair t(t0, t1);
  Pair p = fma2(both(0.5f * 1.061405429f), t, both(0.5f * -1.453152027f));
  p = fma2(p, t, both(0.5f * 1.421413741f));
  p = fma2(p, t, both(0.5f * -0.284496736f));
  p = fma2(p, t, both(0.5f * 0.254829592f));
  e_out = Pair(e0, e1);
  return p * t * e_out;
}
__device__ __forceinline__ Pair gelu2(Pair x) {
  Pair e;
  const Pair q = upper_tail(x, e);
  float a, b;
  x.split(a, b);
  const Pair minus(fminf(a, fmaxf(-a, -3.402823466e38f)), fminf(b, fmaxf(-b, -3.402823466e38f)));   // -|x|, as gelu_f has it
  return fma2(minus, q, Pair(fmaxf(a, 0.f), fmaxf(b, 0.f)));
}
__device__ __forceinline__ Pair gelu_grad2(Pair x) {
  Pair e;
  const Pair q = upper_tail(x, e), r = Pair(1.f, 1.f) - q;
  float a, b, q0, q1, r0, r1;
  x.split(a, b);
  q.split(q0, q1);
  r.split(r0, r1);
  return fma2(x * Pair(0.3989422804014327f, 0.3989422804014327f), e, Pair(a >= 0.f ? r0 : q0, b >= 0.f ? r1 : q1));
}
// v[e] = gelu(v[e] + b[e]) and g[e] *= gelu'(v[e] + b[e])
template <typename T, int N>
__device__ __forceinline__ void gelu_all(float (&v)[N], const float (&b)[N]) {
#pragma unroll
  for (int e = 0; e < N; e += 2) {
    if constexpr (sizeof(T) == 2) {
      gelu2(Pair(v[e], v[e + 1]) + Pair(b[e], b[e + 1])).split(v[e], v[e + 1]);
    } else {
      v[e] = gelu_f(v[e] + b[e]);
      v[e + 1] = gelu_f(v[e + 1] + b[e + 1]);
    }
  }
}
template <typename T, int N>
__device__ __forceinline__ void times_gelu_grad(float (&g)[N], const float (&v)[N], const float (&b)[N]) {
#pragma unroll
  for (int e = 0; e < N; e += 2) {
    if constexpr (sizeof(T) == 2) {
      (Pair(g[e], g[e + 1]) * gelu_grad2(Pair(v[e], v[e + 1]) + Pair(b[e], b[e + 1]))).split(g[e], g[e + 1]);
    } else {
      g[e] *= gelu_grad_f(v[e] + b[e]);
      g[e + 1] *= gelu_grad_f(v[e + 1] + b[e + 1]);
    }
  }
}

}  // namespace tsp
