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
// 1 / (1 + exp(-x)) in four instructions, two of them on the special-function unit: 2^-21 of its value for x above -87, 0 below
__device__ __forceinline__ float logistic(float x) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -1.442695041f));
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
