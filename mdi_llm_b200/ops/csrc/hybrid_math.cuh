// Division, roots, softplus and tanh without the special cases' branches, so that several of them run side by side (a branch a value makes the
// next value wait): gated_chunk_prep_kernel over 2048 tokens, 16 heads of 128 x 128, 85 us, and 91 with 1 / x, 1 / sqrtf and log1pf; the
// read-out 47 and 49.  Each holds for the arguments named beside it, with the error named there against the exact value, in units in the
// last place of the result; hyb_flat_math evaluates them one by one.
#pragma once
#include "hybrid_common.cuh"

namespace hyb {

__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 1 / x for x of 1 to infinity: the hardware's approximation and one step of Newton's iteration on 1 / y - x.  0.51, above 1e37 1; a
// result below 2^-126 is zero.
__device__ __forceinline__ float inverse(float x) {
  float y = rcp_approx(x);
  return x > 1e37f ? y : fmaf(fmaf(-x, y, 1.f), y, y);
}
// 1 / sqrt(x) for x of 2^-126 to infinity: rsqrtf and one step of Newton's iteration on 1 / y^2 - x.  1, above 1e37 2.
__device__ __forceinline__ float inverse_root(float x) {
  float y = rsqrtf(x);
  return x > 1e37f ? y : fmaf(0.5f * y, fmaf(-x * y, y, 1.f), y);
}
// x / by for x of zero, 2^-100 to infinity (either sign) and by of 2^-20 to 2^20, inv = 1 / by: the product with the inverse and what its
// exact residual adds (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990).  0.51.  A quotient that
// is not finite stays, its residual would be no number.
__device__ __forceinline__ float divided(float x, float by, float inv) {
  float y = x * inv, z = fmaf(fmaf(-y, by, x), inv, y);
  return finite(y) ? z : y;
}
// log(1 + exp(x)) for any x: max(x, 0) + log(1 + t) of t = exp(-|x|), where log(u) of the rounded sum u = 1 + t gets back what the sum lost, over u
// (Kahan's logarithm of 1 + t, to first order).  3.
__device__ __forceinline__ float softplus_flat(float x) {
  float t = expf(-fabsf(x)), u = 1.f + t;
  return fmaxf(x, 0.f) + fmaf(t - (u - 1.f), rcp_approx(u), logf(u));
}
// 1 / (1 + exp(-x)) for any x.  3; a result below 2^-126 is zero.
__device__ __forceinline__ float sigmoid_flat(float x) { return inverse(1.f + expf(-x)); }
// tanh(x) for |x| <= 0.75: x + x^3 P(x^2), P the polynomial of degree 5 with the least largest relative error of the whole on that range (by
// Remez exchange on tanh in 80 bits; 2.4e-9 with the coefficients rounded to fp32).  0.75.
__device__ __forceinline__ float small_tanh(float x) {
  const float u = x * x;
  float p = 1.7441476e-3f;
  p = fmaf(p, u, -7.6692365e-3f);
  p = fmaf(p, u, 2.1459442e-2f);
  p = fmaf(p, u, -5.3894807e-2f);
  p = fmaf(p, u, 1.3332720e-1f);
  p = fmaf(p, u, -3.3333316e-1f);
  return fmaf(x * u, p, x);
}

}  // namespace hyb
