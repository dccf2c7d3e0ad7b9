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
// Two single-precision operations in one issue slot
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// x / (1 + exp(-x)) of two values, with two special-function instructions each (expf and a division: a third more time on a GroupNorm) and the
// rest in pairs: the direct convolution that normalises 128 channels of 256^2 is bound by its issue slots.  exp(-x) = 2^t with t =
// -x log2 e.  What rounding t loses goes back in as a first-order factor, d = -x - t ln 2 with ln 2 in two parts (W. J. Cody and W. Waite, Software
// Manual for the Elementary Functions, 1980): |d| < 4e-6, the next term is 8e-12.  With 2^-22 for each of the two instructions the result is
// within 2^-21 of its value for -87.3 <= x, infinity included: above 64 it is x itself (2^t is 0 next to 1; the bound keeps d finite).
// Below -87.3 the reciprocal is flushed and the result is -0, off by less than 1.2e-36 (t ends at 126.9, and d, which then grows, only
// lengthens the sum); -inf gives NaN, as x * (1 / (1 + expf(-x))) does.
__device__ __forceinline__ void silu2(float& x0, float& x1) {
  const float n0 = fmaxf(-x0, -64.0f), n1 = fmaxf(-x1, -64.0f);
  const unsigned long long n = pack2(n0, n1);
  float t0, t1, e0, e1, r0, r1;
  unpack2(mul2(n, pack2(1.44269504f, 1.44269504f)), t0, t1);
  t0 = fminf(t0, 126.9f);
  t1 = fminf(t1, 126.9f);
  const unsigned long long t = pack2(t0, t1);
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(t0));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(t1));
  unsigned long long d = fma2(t, pack2(-0.693147182f, -0.693147182f), n);  // ln 2 = 0.693147182464600 - 1.904654e-9
  d = fma2(t, pack2(1.904654e-9f, 1.904654e-9f), d);
  unsigned long long e = pack2(e0, e1);
  e = fma2(e, d, e);
  unpack2(add2(e, pack2(1.0f, 1.0f)), r0, r1);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(r0));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(r1));
  unpack2(mul2(pack2(x0, x1), pack2(r0, r1)), x0, x1);
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
