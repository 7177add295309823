// The activations of gated feed-forward layers: kind 0 SiLU, else GELU by its tanh form.
#pragma once

namespace tb {

__device__ __forceinline__ float act_fwd(float g, int kind) {
  if (kind == 0) return g / (1.f + __expf(-g));  // SiLU
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;  // tanh-approximate GELU
  return 0.5f * g * (1.f + tanhf(k0 * (g + k1 * g * g * g)));
}
__device__ __forceinline__ float act_bwd(float g, int kind) {
  if (kind == 0) {
    const float s = 1.f / (1.f + __expf(-g));
    return s * (1.f + g * (1.f - s));
  }
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float t = tanhf(k0 * (g + k1 * g * g * g));
  return 0.5f * (1.f + t) + 0.5f * g * (1.f - t * t) * k0 * (1.f + 3.f * k1 * g * g);
}

}  // namespace tb
