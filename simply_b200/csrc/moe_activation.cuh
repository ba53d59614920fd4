// Activations of the experts' products, shared by the kernels that form them (moe.cu, moe_tc.cu):
// 0 gelu (tanh form), 1 silu, 2 relu, 3 the clamped form (with a gate only), 4 the exact gelu.
#pragma once

__device__ __forceinline__ float moe_activation(float g, int act) {
  if (act == 0) {
    const float c = 0.7978845608028654f;
    return 0.5f * g * (1.0f + tanhf(c * (g + 0.044715f * g * g * g)));
  }
  if (act == 1) return g / (1.0f + expf(-g));
  if (act == 4) return 0.5f * g * (1.0f + erff(g * 0.7071067811865476f));  // the exact gelu
  return fmaxf(g, 0.f);
}

// act(gate) * up; activation 3 is the clamped form, which acts on both halves:
// g' = min(g, limit), u' = clamp(u, -limit, limit), g' sigmoid(1.702 g') (u' + 1).
__device__ __forceinline__ float moe_gated_pair(float g, float u, int act, float limit) {
  if (act == 3) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.0f + expf(-1.702f * g)) * (u + 1.0f);
  }
  return moe_activation(g, act) * u;
}
