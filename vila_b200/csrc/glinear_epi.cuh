// Epilogue pieces of vila_glinear shared by its CUDA-core and its tcgen05 kernels.
#pragma once
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "dtype_any.cuh"

namespace vb {

// clamped gated unit: g = min(zg, limit), u = clamp(zu, +-limit), g * sigmoid(alpha * g) * (u + 1)
__device__ __forceinline__ float glu_clamp_f(float zg, float zu, const vila_glinear_ext& x) {
  const float g = fminf(zg, x.act_limit), u = fminf(fmaxf(zu, -x.act_limit), x.act_limit);
  return g * sigmoid_f(x.act_alpha * g) * (u + 1.0f);
}

__device__ __forceinline__ float gelu_tanh_exact_f(float z) {
  return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ float activate(float z, int act, const vila_glinear_ext& x) {
  switch (act) {
    case VILA_ACT_SILU: return silu_exact_f(z);
    case VILA_ACT_RELU2: z = fmaxf(z, 0.f); return z * z;
    case VILA_ACT_GELU_TANH: return gelu_tanh_exact_f(z);
    case VILA_ACT_GELU_ERF: return gelu_erf_f(z);
    case VILA_ACT_XIELU: return xielu_f(z, x.act_pos, x.act_neg);
    case VILA_ACT_SOFTCAP: return x.act_pos * tanhf(z / x.act_pos);
    default: return z;
  }
}
// the two columns of a gated unit (flags: which one)
constexpr int kGluFlags = VILA_FLAG_SWIGLU | VILA_FLAG_GLU_CLAMP | VILA_FLAG_GEGLU;
__device__ __forceinline__ float glu(float g, float u, int flags, const vila_glinear_ext& x) {
  if (flags & VILA_FLAG_GLU_CLAMP) return glu_clamp_f(g, u, x);
  return (flags & VILA_FLAG_GEGLU ? gelu_tanh_exact_f(g) : silu_exact_f(g)) * u;
}

// bias and activation of one output
__device__ __forceinline__ float finish(const vila_glinear_params& p, const vila_glinear_ext& x, float z, int g, int n) {
  if (p.bias) z += ld_any(p.bias, p.w_dtype, static_cast<size_t>(g) * p.bias_group_stride + n);
  return activate(z, p.act, x);
}

// scale of the INPUT row behind sorted position i (= output row: in_scale is only taken without o_rows)
__device__ __forceinline__ float in_scale_of(const vila_glinear_params& p, const vila_glinear_ext& x, int i) {
  return x.in_scale ? x.in_scale[p.a_rows ? p.a_rows[i] : i] : 1.0f;
}

}  // namespace vb
