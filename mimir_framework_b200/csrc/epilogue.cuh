// epilogue.cuh — activations applied to a contraction's accumulators before they leave the kernel.
#pragma once

#include "mimir_b200.h"

namespace mb {
namespace {

// GELU in the reference's tanh form (LayerOps.hpp:556-568), x * 0.5 * (1 + tanh(u)) with u = c * (x + 0.044715 x^3) and
// c = sqrt(2.0f / 3.14159265359f) evaluated in fp32.  0.5 * (1 + tanh(u)) is the logistic function of 2u, so the value is
// x / (1 + exp(-2u)): one ex2 and one reciprocal on the special-function unit instead of tanhf's ~30 instructions (the
// epilogue of a K = 768 layer has only ~12 000 cycles per 128 x 256 tile for 32 768 of these), and without the
// cancellation of 1 + tanh(u) for negative arguments.  Error: the two instructions' 2^-22 each and, for negative x, what rounding the
// exponent costs, |2u| 2^-24: 1e-6 of the result at x = -5, where the result is 5e-8 of x.
__device__ __forceinline__ float gelu_ref(float x) {
  const float c = 0.7978845608f;
  const float u = c * (x + 0.044715f * x * x * x);
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(u * -2.885390082f));  // exp(-2u) = 2^(-2u log2 e)
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
  return __fmul_rn(x, r);  // (not contracted with a residual that follows)
}
// 1 / (1 + exp(-x)), the factor of SiLU, with two special-function instructions (expf and a division: a third more time on a GroupNorm).
// exp(-x) = 2^t with t = -x log2 e.  What rounding t loses goes back in as a first-order factor: the constant in two parts (W. J. Cody and
// W. Waite, Software Manual for the Elementary Functions, 1980), the product's rounding error by fused multiply-add, 2^d = 1 + d ln 2 for
// |d| < 1.2e-5 (the next term is 4e-11).  With 2^-22 for each of the two instructions x times the result is within 2^-21 of its value for
// -87.3 <= x, infinity included: above 64 it is x itself (2^t is 0 next to 1; the bound keeps `lost` finite).  Below -87.3 the
// reciprocal is flushed and the product is -0, off by less than 1.2e-36; -inf gives NaN, as x * (1 / (1 + expf(-x))) does.
__device__ __forceinline__ float logistic(float x) {
  const float c = fminf(fmaxf(x, -88.0f), 64.0f);
  const float t = c * -1.44269504f;
  const float lost = fmaf(c, -1.44269504f, -t) - c * 1.92596e-8f;  // log2 e = 1.44269502163 + 1.92596e-8
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t));
  e = fmaf(e, lost * 0.69314718f, e);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
  return r;
}
__device__ __forceinline__ float apply_act(float v, int act) {
  switch (act) {
    case MIMIR_B200_ELT_GELU: return gelu_ref(v);
    case MIMIR_B200_ELT_SILU: return __fmul_rn(v, 1.0f / (1.0f + expf(-v)));
    case MIMIR_B200_ELT_RELU: return fmaxf(v, 0.0f);
    case MIMIR_B200_ELT_TANH: return tanhf(v);
    case MIMIR_B200_ELT_SIGMOID: return 1.0f / (1.0f + expf(-v));
    default: return v;
  }
}

// The activations of the exact-fp32 kernels for a few rows (tanhf for GELU, as the reference writes it).
__device__ __forceinline__ float sk_act(float v, int act) {
  switch (act) {
    case MIMIR_B200_ELT_GELU: {
      const float c = 0.7978845608f;
      return v * (0.5f * (1.0f + tanhf(c * (v + 0.044715f * v * v * v))));
    }
    case MIMIR_B200_ELT_SILU: return v * (1.0f / (1.0f + expf(-v)));
    case MIMIR_B200_ELT_RELU: return fmaxf(0.0f, v);
    case MIMIR_B200_ELT_TANH: return tanhf(v);
    case MIMIR_B200_ELT_SIGMOID: return 1.0f / (1.0f + expf(-v));
    default: return v;
  }
}

}  // namespace
}  // namespace mb
