// The activation of gated experts with limits (experts.cu says of which form).
#pragma once

__device__ __forceinline__ float limited_one(float g, float u, float w, float limit, float alpha, float offset) {
  g = fminf(w * g, limit);
  u = fminf(fmaxf(w * u, -limit), limit);
  return g / (1.0f + expf(-alpha * g)) * (u + offset);
}
