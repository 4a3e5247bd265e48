// Activation functions shared by the kernels that apply them in an epilogue or on their own (fp32 arithmetic).
#pragma once
#include <cuda_runtime.h>

namespace b200 {

// a_pos z^2 + z / 2 for z > 0, a_neg (exp(z) - 1 - z) + z / 2 for z <= 0
__device__ __forceinline__ float xielu(float z, float a_pos, float a_neg) {
  const float n = fminf(z, 0.f);
  return fmaf(z > 0.f ? a_pos * z : 0.5f, z, z > 0.f ? 0.5f * z : a_neg * (expm1f(n) - n));
}

// The same with the hardware exponential (absolute error of exp below 2^-21 for z <= 0): for results that are rounded to bf16.
__device__ __forceinline__ float xielu_fast(float z, float a_pos, float a_neg) {
  const float e = __expf(fminf(z, 0.f));
  return fmaf(z > 0.f ? a_pos * z : 0.5f, z, z > 0.f ? 0.5f * z : a_neg * (e - 1.0f - z));
}

// A gated unit: min(g, limit) sigmoid(slope min(g, limit)) (clamp(u, -limit, limit) + up_offset); without `clamp` the limit is
// infinite.  FAST: the hardware exponential and quotient, about 2^-21 of the unit ahead of its rounding.
template <bool FAST>
__device__ __forceinline__ float gated_unit(float g, float u, bool clamp, float limit, float slope, float up_offset) {
  if (clamp) { g = fminf(g, limit); u = fminf(fmaxf(u, -limit), limit); }
  if (FAST) return __fdividef(g, 1.0f + __expf(-slope * g)) * (u + up_offset);
  return g * (1.0f / (1.0f + expf(-(slope * g)))) * (u + up_offset);     // accurate functions, as norm_act.cu's glu_clamped
}

}  // namespace b200
