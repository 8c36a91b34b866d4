// Masks, block lists and score options of vila_paged_attention, shared by its CUDA-core and its tensor-core kernels.
#pragma once
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "dtype_any.cuh"

namespace vb {

constexpr float kNegBig = -1e30f;

__host__ __device__ __forceinline__ int maps_of(int maps) { return maps > 1 ? maps : 1; }

__device__ __forceinline__ size_t pool_row(const int32_t* pt, int page, int j) {
  return static_cast<size_t>(pt[j / page]) * page + (j % page);
}

// first key a query at position pos can see
__device__ __forceinline__ int first_key(const vila_paged_attn_params& p, int pos) {
  return p.chunk > 0 ? (pos / p.chunk) * p.chunk : 0;
}
// may the query at position pos see key j?
__device__ __forceinline__ bool sees(const vila_paged_attn_params& p, int pos, int j) {
  return j <= pos && j >= first_key(p, pos) && (p.window <= 0 || pos - j < p.window || j < p.keep_first);
}
// Key blocks of BK keys a tile visits, in order: [0, kb) then [wb, nblocks).
struct BlockList {
  int kb, wb, count;
  __device__ __forceinline__ int block(int v) const { return v < kb ? v : wb + (v - kb); }
};
__device__ __forceinline__ BlockList visible_blocks(const vila_paged_attn_params& p, int pos0, int nkeys, int BK) {
  BlockList b;
  const int nblocks = (nkeys + BK - 1) / BK;
  if (p.window <= 0) {
    b.kb = 0;
    b.wb = first_key(p, pos0) / BK;
  } else {
    b.kb = min((min(p.keep_first, nkeys) + BK - 1) / BK, nblocks);
    b.wb = max(b.kb, max(max(pos0 - p.window + 1, 0), first_key(p, pos0)) / BK);
  }
  b.count = b.kb + max(nblocks - b.wb, 0);
  return b;
}
__device__ __forceinline__ float head_scale(const vila_paged_attn_params& p, int h) {
  return p.head_scale ? p.scale * p.head_scale[h] : p.scale;
}
// A head's own scaled score, bounded to (-softcap, softcap) when a cap is set: cap tanh(s / cap).  Scores up to the cap itself
// take s R((s / cap)^2) with R(u) = tanh(sqrt u) / sqrt u, an entire quotient on [0, 1] whose nearest pole (-pi^2 / 4) lets
// Chebyshev interpolation of degree 7 be 4e-9 close: 3.3e-8 off in fp32 (rms; a correctly rounded quotient, tanh and product
// 4.2e-8) at 10 multiply-adds where the quotient and tanhf took 50 instructions.  Scores above the cap take
// cap (1 - 2 / (e^(2 s / cap) + 1)), whose quotient is below 0.24 there, so that the approximate exponential and reciprocal cost
// less than a rounding of the result: 1.8e-8 - 4.0e-8 off (rms; at most 1.4e-7) over 1 < s / cap < 9 for caps of 0.01 - 50, where
// cap tanhf(s / cap) is 1.8e-8 - 4.4e-8 (1.7e-7).  By the score alone, so that it does not depend on its neighbours.
__device__ __forceinline__ constexpr float cap_poly(int k) {
  constexpr float c[8] = {1.0f, -0.33333277702331543f, 0.1333213895559311f, -0.05386970564723015f,
                          0.02146141044795513f, -0.007912484928965569f, 0.002278647618368268f, -0.000352328090230003f};
  return c[k];
}
__device__ __forceinline__ float cap_inverse(const vila_paged_attn_params& p) { return p.softcap > 1e-30f ? 1.0f / p.softcap : 0.f; }
__device__ __forceinline__ bool over_cap(const vila_paged_attn_params& p, float s) { return !(fabsf(s) <= p.softcap); }
__device__ __forceinline__ float cap_inverse_over(float inverse) { return inverse > 0.f ? 2.8853900817779268f * inverse : INFINITY; }   // 2 log2 e / cap
__device__ __forceinline__ float capped_over(float cap, float inverse_over, float s) {
  float e, q;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(fabsf(s) * inverse_over));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(e + 1.0f));
  return copysignf(fmaf(-2.0f * cap, q, cap), s);
}
__device__ __forceinline__ float capped(const vila_paged_attn_params& p, float s, float inv) {   // inv: cap_inverse
  if (over_cap(p, s)) return capped_over(p.softcap, cap_inverse_over(inv), s);
  const float x = s * inv, u = __fmul_rn(x, x);
  float r = cap_poly(7);
#pragma unroll
  for (int k = 6; k >= 0; --k) r = fmaf(r, u, cap_poly(k));
  return s * r;
}
__device__ __forceinline__ float capped(const vila_paged_attn_params& p, float s) { return p.softcap > 0.f ? capped(p, s, cap_inverse(p)) : s; }
__device__ __forceinline__ float dist_bias(const vila_paged_attn_params& p, int dist, int h) {
  return __ldg(p.dist_bias + static_cast<size_t>(min(dist, p.dist_rows - 1)) * p.H + h);
}
// Score head h counts the maps singly: model head h / maps, map h % maps.  Its key head (also counted with maps) and
// value head; rep = query heads per key / value head.
__device__ __forceinline__ int key_head(int h, int maps, int rep) { return maps == 1 ? h / rep : ((h >> 1) / rep) * 2 + (h & 1); }
__device__ __forceinline__ int value_head(int h, int maps, int rep) { return maps == 1 ? h / rep : (h >> 1) / rep; }
__device__ __forceinline__ float out_gate(const vila_paged_attn_params& p, int row, int h) {
  return p.gate ? sigmoid_f(ld_any(p.gate, p.gate_dtype, static_cast<size_t>(row) * p.ldg + h)) : 1.0f;
}

}  // namespace vb
