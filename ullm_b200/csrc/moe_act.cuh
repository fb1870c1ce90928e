// Activations of the routed experts' grouped products (moe.cu, moe_tcgen05.cu), in 32-bit.
#pragma once

#include "common.cuh"

__device__ __forceinline__ float moe_gate_act(int act, float g, float u, float limit, float alpha) {
  if (act == 2) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.f + expf(-alpha * g)) * (u + 1.f);
  }
  return (act == 0 ? act_silu(g) : act_gelu_tanh(g)) * u;
}

// The same with the activation fixed at compile time and without a branch, so that a thread's elements run beside one another: all
// three are u' g' / (1 + e^-z) (z = g; 2 sqrt(2 / pi) (g + 0.044715 g^3), since (1 + tanh v) / 2 = 1 / (1 + e^-2v); alpha g'), the
// quotient from a reciprocal with one step of Newton's method.  From 2^126 on the denominator counts as infinite.
template <int ACT>
__device__ __forceinline__ float moe_gate_act_flat(float g, float u, float limit, float alpha) {
  float z = g;
  if (ACT == 2) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit) + 1.f;
    z = alpha * g;
  } else if (ACT != 0) {
    z = 1.5957691216057308f * (g + 0.044715f * g * g * g);
  }
  const float y = 1.f + expf(-z), r = __fdividef(1.f, y), q = g * r;
  const float s = fabsf(g) <= 3.4028234e38f ? fmaf(fmaf(-q, y, g), r, q) : q;
  return (y < 8.5e37f ? s : (y == y ? g * 0.f : y)) * u;
}

// the activation of a product without gate rows
__device__ __forceinline__ float moe_plain_act(int act, float v) {
  if (act == 3) {
    v = fmaxf(v, 0.f);
    return v * v;
  }
  return v;
}
