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

// The same with the activation fixed at compile time and without a branch.
template <int ACT>
__device__ __forceinline__ float moe_gate_act_flat(float g, float u, float limit, float alpha) {
  if (ACT == 2) {
    g = fminf(g, limit);
    return gate_flat(g, alpha * g) * (fminf(fmaxf(u, -limit), limit) + 1.f);
  }
  return (ACT == 0 ? gate_flat(g, g) : act_gelu_tanh_flat(g)) * u;
}

// the activation of a product without gate rows
__device__ __forceinline__ float moe_plain_act(int act, float v) {
  if (act == 3) {
    v = fmaxf(v, 0.f);
    return v * v;
  }
  return v;
}
