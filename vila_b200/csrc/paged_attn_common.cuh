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

constexpr float kLog2e = 1.44269504f;   // 1 / ln 2

// two fp32 numbers at a time
using f2 = unsigned long long;
__device__ __forceinline__ f2 pair(float x, float y) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void unpair(f2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ void fma2(float& ax, float& ay, float m, float cx, float cy) {   // a = a m + c
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pair(ax, ay)), "l"(pair(m, m)), "l"(pair(cx, cy)));
  unpair(r, ax, ay);
}
__device__ __forceinline__ void add2(float& ax, float& ay, float cx, float cy) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pair(ax, ay)), "l"(pair(cx, cy)));
  unpair(r, ax, ay);
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// capped() of two scores up to the cap, the same operations
__device__ __forceinline__ void cap2(float& a, float& b, float inv) {
  const f2 s = pair(a, b), x = mul2(s, pair(inv, inv)), u = mul2(x, x);
  f2 r = pair(cap_poly(7), cap_poly(7));
#pragma unroll
  for (int k = 6; k >= 0; --k) r = fma2(r, u, pair(cap_poly(k), cap_poly(k)));
  unpair(mul2(s, r), a, b);
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// log2(e) x, rounded (never fused into what follows: a maximum's value has to be the same wherever it is used)
__device__ __forceinline__ float log2_units(float x) { return __fmul_rn(x, kLog2e); }

// A row of one score head again, key by key in fp32 multiply-adds, into dst (V numbers, divided by their weights' sum): what
// the CUDA-core kernels compute.  Rows that met an infinite or NaN number come here, because the parts of a finite number
// hold zeros and zero times infinity is NaN where the whole number times infinity is not.  A warp per row.
template <int D, int MAPS, int V>
__device__ __noinline__ void row_again(const vila_paged_attn_params& p, int row, int pos, int slot, int h, int map, float* dst) {
  constexpr int DL = D / 32, VL = V / 32;                 // columns of a lane
  const int lane = threadIdx.x & 31, g = h / (p.H / p.G);
  const int32_t* pt = p.page_tables + static_cast<size_t>(slot) * p.pt_stride;
  const size_t prow = static_cast<size_t>(p.G) * (MAPS * D + V);
  const __nv_bfloat16* pool = static_cast<const __nv_bfloat16*>(p.pool);
  const size_t koff = static_cast<size_t>(g * MAPS + map) * D + DL * lane, voff = static_cast<size_t>(p.G) * MAPS * D + static_cast<size_t>(g) * V + VL * lane;
  const float sc = head_scale(p, h);
  float q[DL], acc[VL];
#pragma unroll
  for (int e = 0; e < DL; ++e) q[e] = p.q[((static_cast<size_t>(row) * p.H + h) * MAPS + map) * D + DL * lane + e] * sc;
#pragma unroll
  for (int e = 0; e < VL; ++e) acc[e] = 0.f;
  float m = p.sink ? p.sink[h] : kNegBig, l = p.sink ? 1.0f : 0.0f;
  for (int j = 0; j <= pos; ++j) {
    if (!sees(p, pos, j)) continue;
    const __nv_bfloat16* at = pool + pool_row(pt, p.page, j) * prow;
    float s = 0.f;
#pragma unroll
    for (int e = 0; e < DL; ++e) s = fmaf(q[e], __bfloat162float(at[koff + e]), s);
    s = capped(p, warp_sum(s));
    if (p.dist_bias) s += dist_bias(p, pos - j, h);
    const float mn = fmaxf(m, s), w = expf(s - mn), alpha = expf(m - mn);
    l = fmaf(l, alpha, w);
    m = mn;
#pragma unroll
    for (int e = 0; e < VL; ++e) acc[e] = fmaf(w, __bfloat162float(at[voff + e]), acc[e] * alpha);
  }
#pragma unroll
  for (int e = 0; e < VL; ++e) dst[VL * lane + e] = acc[e] * (1.0f / l);
}

}  // namespace vb
