// Grouped-query attention over a paged K/V pool for ragged batches, with the pieces a parallel-sublayer
// decoder adds to it:
//   rope_append_kernel   rotary positions on the first rot_dims columns of every q / k head (pairs
//                        (2i, 2i+1) or (i, i + rot_dims / 2), angle = position * inv_freq[i], evaluated in
//                        double so that far positions keep their phase; cos and sin optionally scaled by
//                        one magnitude), optional unit norm per head (fp32), q out as fp32,
//                        k | v appended to the pool row of the token
//   paged_attn_kernel    fp32 scores of ALL H heads of a (query, key) pair, optional head mixing
//                        s_h <- sum_g talk[h, g] s_g before the softmax, online softmax whose running
//                        (max, sum) starts at (sink_h, 1) when a sink is given, fp32 weighted sum.
//                        A CTA owns BQ consecutive rows of one sequence x all heads (BQ * H "score rows");
//                        prompt portions use BQ up to 16, decoded tokens BQ = 1 with the key blocks of a
//                        row dealt to nsplit CTAs
//   paged_attn_merge_kernel  merges the nsplit partial (max, sum, weighted sum) triples of a decoded token
// Options another architecture can combine freely: an additive bias looked up by the distance between
// query and key (dist_bias [dist_rows, H], the last row serves every larger distance; added after scale and
// mixing), a chunked mask (a query sees the keys of its own block of `chunk` positions only; the key loop
// starts at the block of the tile's first row), and a per-(token, head) sigmoid gate on the output.
// A cap bounds every head's own scaled score to softcap * tanh(score / softcap) before mixing, bias and softmax.
// The append kernel can mix another layer's values of the same tokens into the cached ones.
// A sliding window with kept first tokens (a key is seen if it is at most window - 1 positions back, or among the
// first keep_first of its sequence) is a mask plus a shorter block list: the blocks that hold kept tokens, then
// the blocks from the window of the tile's first row on.  A per-head multiplier of the scores is folded into the
// staged queries.  talk_after mixes the heads' softmax WEIGHTS: that needs every head's final (max, sum) before
// any value is added, so the kernels first run over the key blocks with the scores only (pass 0), then again with
// weights exp(s - max) / sum, mixed over heads, times the values (pass 1; nothing is rescaled).  When the keys of
// a decoded token are dealt to several CTAs, pass 0 and pass 1 are two launches: the first leaves every CTA's
// (max, sum) of its share in the partial records, the second merges them in split order and adds its share.
// Differential attention (maps == 2): every query / key head comes as two maps side by side, each an attention of its own
// over the same value head; a CTA always holds both maps of its heads, so the pair is combined where the sums end,
//   o = rms(a1 - lambda a2) * diff_scale   (rms over the head's vdim values), then the gate,
// in the epilogue of the tiled and the one-row kernel or in the merge of a decoded token's key splits.
// Every reduction over keys runs in key order inside a block and block by block, so a row's result does
// not depend on what else is in the launch.
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "kernels.h"
#include "dtype_any.cuh"
#include "paged_attn_common.cuh"

namespace vb {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

__host__ __device__ __forceinline__ int round4(int r) { return (r + 3) & ~3; }
// Floats between the K rows of consecutive keys in shared memory: all G heads of a key (G * DS, DS = D4 + 4)
// plus a pad that makes the stride 4 mod 32, so that the float4 reads of 8 consecutive keys (same head, same
// column) fall into 8 different bank groups.
__host__ __device__ __forceinline__ int key_stride(int G, int DS) { return G * DS + ((36 - (G * DS) % 32) % 32); }


// ---- rotary + unit norm + append ---------------------------------------------------------------------
// One CTA per token; warp w takes the heads w, w + 8, ... of q then k; v is copied by all threads.
__global__ void __launch_bounds__(kThreads) rope_append_kernel(const vila_rope_append_params p) {
  extern __shared__ float cs[];   // cos [rot/2] | sin [rot/2]
  const int t = blockIdx.x, half = p.rot_dims >> 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const double pos = static_cast<double>(p.positions[t]);
  const float mag = p.rot_mscale != 0.f ? p.rot_mscale : 1.0f;
  for (int i = tid; i < half; i += kThreads) {
    double s, c;
    sincos(pos * p.inv_freq[i], &s, &c);
    cs[i] = static_cast<float>(c) * mag;
    cs[half + i] = static_cast<float>(s) * mag;
  }
  __syncthreads();
  // column c of the rotated part: its partner, its pair index and whether it is the second of its pair
  const bool halves = p.rot_layout == 1;
  auto partner = [&](int c) { return halves ? (c < half ? c + half : c - half) : (c ^ 1); };
  auto pair_of = [&](int c) { return halves ? (c < half ? c : c - half) : (c >> 1); };
  auto second = [&](int c) { return halves ? c >= half : (c & 1) != 0; };
  const size_t in0 = static_cast<size_t>(t) * p.ldq;
  const int maps = maps_of(p.maps), HQ = p.H * maps, GK = p.G * maps;   // query / key heads with their maps counted singly
  const size_t koff = static_cast<size_t>(GK) * p.dim;                  // where a pool row's values start
  const size_t prow = static_cast<size_t>(p.cache_rows[t]) * (koff + static_cast<size_t>(p.G) * p.vdim);
  for (int hh = warp; hh < HQ + GK; hh += kWarps) {
    const bool is_q = hh < HQ;
    const size_t src = in0 + static_cast<size_t>(hh) * p.dim;   // q heads then k heads are contiguous
    // pass 1: rotated values -> sum of squares (recomputed in pass 2: dim is small, no buffer needed)
    float ss = 0.f;
    for (int c = lane; c < p.dim; c += 32) {
      float v = ld_any(p.qkv, p.qkv_dtype, src + c);
      if (c < p.rot_dims) {
        const float o = ld_any(p.qkv, p.qkv_dtype, src + partner(c));
        const float co = cs[pair_of(c)], si = cs[half + pair_of(c)];
        v = second(c) ? fmaf(v, co, o * si) : fmaf(v, co, -(o * si));
      }
      ss = fmaf(v, v, ss);
    }
    ss = warp_sum(ss);
    const float r = p.unit_norm ? 1.0f / sqrtf(ss / static_cast<float>(p.dim) + p.eps) : 1.0f;
    const float* nw = is_q ? p.q_norm_w : p.k_norm_w;
    for (int c = lane; c < p.dim; c += 32) {
      float v = ld_any(p.qkv, p.qkv_dtype, src + c);
      if (p.v_from_k && !is_q)   // the value is the key as it came in
        st_any(p.pool, p.pool_dtype, prow + koff + static_cast<size_t>(hh - HQ) * p.dim + c, v);
      if (c < p.rot_dims) {
        const float o = ld_any(p.qkv, p.qkv_dtype, src + partner(c));
        const float co = cs[pair_of(c)], si = cs[half + pair_of(c)];
        v = second(c) ? fmaf(v, co, o * si) : fmaf(v, co, -(o * si));
      }
      v *= r;
      if (nw) v *= nw[c];
      if (is_q) p.q_out[(static_cast<size_t>(t) * HQ + hh) * p.dim + c] = v;
      else st_any(p.pool, p.pool_dtype, prow + static_cast<size_t>(hh - HQ) * p.dim + c, v);
    }
  }
  if (p.v_from_k) return;
  const size_t vsrc = in0 + static_cast<size_t>(HQ + GK) * p.dim, vdst = prow + koff;
  for (int c = tid; c < p.G * p.vdim; c += kThreads) {
    float v = ld_any(p.qkv, p.qkv_dtype, vsrc + c);
    if (p.v_first)   // part of the value comes from another layer's value of the same token
      v = fmaf(p.v_mix, ld_any(p.v_first, p.v_first_dtype, static_cast<size_t>(t) * p.ld_vf + c), (1.0f - p.v_mix) * v);
    st_any(p.pool, p.pool_dtype, vdst + c, v);
  }
}

// The same for even head sizes, a pair of columns (rotated together, or neighbours past the rotated part) at a time: a lane
// loads its NP pairs of a head once, all in flight, and keeps them over the norm; the first head's are on their way while
// the angles are evaluated.  The general form reads every element twice, one after the other (2048 tokens of 24 heads:
// 33 us, here 13.8; 8 tokens 7.2 and 3.3).
template <bool BF16, int NP>
__global__ void __launch_bounds__(kThreads) rope_append_pairs_kernel(const vila_rope_append_params p) {
  extern __shared__ float cs[];   // cos [rot/2] | sin [rot/2]
  const int t = blockIdx.x, half = p.rot_dims >> 1, npair = p.dim >> 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool halves = p.rot_layout == 1;
  const int maps = maps_of(p.maps), HQ = p.H * maps, GK = p.G * maps, heads = HQ + GK;
  const size_t koff = static_cast<size_t>(GK) * p.dim, in0 = static_cast<size_t>(t) * p.ldq;
  auto first_of = [&](int i) { return !halves || i >= half ? (halves ? p.rot_dims + 2 * (i - half) : 2 * i) : i; };
  auto second_of = [&](int i) { return halves && i < half ? i + half : first_of(i) + 1; };
  auto fetch = [&](int hh, uint32_t (&x)[NP], uint32_t (&y)[NP]) {
    const size_t src = in0 + static_cast<size_t>(hh) * p.dim;
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const int i = lane + 32 * k;
      x[k] = i < npair ? ld_raw(p.qkv, BF16 ? VILA_DT_BF16 : VILA_DT_F32, src + first_of(i)) : 0u;
      y[k] = i < npair ? ld_raw(p.qkv, BF16 ? VILA_DT_BF16 : VILA_DT_F32, src + second_of(i)) : 0u;
    }
  };
  uint32_t x[NP], y[NP];
  if (warp < heads) fetch(warp, x, y);
  const double pos = static_cast<double>(p.positions[t]);
  const float mag = p.rot_mscale != 0.f ? p.rot_mscale : 1.0f;
  for (int i = tid; i < half; i += kThreads) {
    double s, c;
    sincos(pos * p.inv_freq[i], &s, &c);
    cs[i] = static_cast<float>(c) * mag;
    cs[half + i] = static_cast<float>(s) * mag;
  }
  const size_t prow = static_cast<size_t>(p.cache_rows[t]) * (koff + static_cast<size_t>(p.G) * p.vdim);
  __syncthreads();
  for (int hh = warp; hh < heads; hh += kWarps) {
    const bool is_q = hh < HQ;
    float a[NP], b[NP], raw_a[NP], raw_b[NP], ss = 0.f;
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const int i = lane + 32 * k;
      a[k] = raw_a[k] = raw_to_float(x[k], BF16 ? VILA_DT_BF16 : VILA_DT_F32);
      b[k] = raw_b[k] = raw_to_float(y[k], BF16 ? VILA_DT_BF16 : VILA_DT_F32);
      if (i < half) {
        const float co = cs[i], si = cs[half + i];
        a[k] = fmaf(raw_a[k], co, -(raw_b[k] * si));
        b[k] = fmaf(raw_b[k], co, raw_a[k] * si);
      }
      ss = fmaf(a[k], a[k], fmaf(b[k], b[k], ss));
    }
    if (hh + kWarps < heads) fetch(hh + kWarps, x, y);
    float r = 1.0f;
    if (p.unit_norm) r = 1.0f / sqrtf(warp_sum(ss) / static_cast<float>(p.dim) + p.eps);
    const float* nw = is_q ? p.q_norm_w : p.k_norm_w;
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const int i = lane + 32 * k;
      if (i >= npair) continue;
      const int c0 = first_of(i), c1 = second_of(i);
      float u = a[k] * r, v = b[k] * r;
      if (nw) {
        u *= nw[c0];
        v *= nw[c1];
      }
      if (is_q) {
        float* q = p.q_out + (static_cast<size_t>(t) * HQ + hh) * p.dim;
        q[c0] = u;
        q[c1] = v;
      } else {
        const size_t kd = prow + static_cast<size_t>(hh - HQ) * p.dim;
        st_any(p.pool, p.pool_dtype, kd + c0, u);
        st_any(p.pool, p.pool_dtype, kd + c1, v);
        if (p.v_from_k) {   // the value is the key as it came in
          st_any(p.pool, p.pool_dtype, kd + koff + c0, raw_a[k]);
          st_any(p.pool, p.pool_dtype, kd + koff + c1, raw_b[k]);
        }
      }
    }
  }
  if (p.v_from_k) return;
  const size_t vsrc = in0 + static_cast<size_t>(heads) * p.dim, vdst = prow + koff;
#pragma unroll 2
  for (int c = tid; c < p.G * p.vdim; c += kThreads) {
    float v = raw_to_float(ld_raw(p.qkv, BF16 ? VILA_DT_BF16 : VILA_DT_F32, vsrc + c), BF16 ? VILA_DT_BF16 : VILA_DT_F32);
    if (p.v_first)   // part of the value comes from another layer's value of the same token
      v = fmaf(p.v_mix, ld_any(p.v_first, p.v_first_dtype, static_cast<size_t>(t) * p.ld_vf + c), (1.0f - p.v_mix) * v);
    st_any(p.pool, p.pool_dtype, vdst + c, v);
  }
}

// Head sizes of 64, 128 and 256.  The form above is bound by its instructions (220 a head: 2-byte accesses, a whole warp and
// 64-bit addresses for one head), not by its bytes, so here a lane has eight columns, two runs of four that are rotated with
// each other, and a warp 4, 2 or 1 heads at a time; from more than four CTAs an SM on, two tokens share a CTA and the latency
// of their angles (double sincos).  bf16 in and out, us, before and now: 16 heads of 128 over 4 on 8 / 592 / 800 / 2048 / 4096
// tokens 3.9 / 6.2 / 7.8 / 15.0 / 27.5, now 3.0 / 4.2 / 4.9 / 9.0 / 15.0; 32 of 64 over 32 6.6 / 9.7 / 12.8 / 24.2 / 51.5, now
// 3.4 / 5.1 / 6.8 / 12.4 / 29.3 (4.0 TB/s).  One token a CTA: 592 and 800 tokens 4.2 and 6.4, two 4.6 and 4.9; four tokens a CTA
// are 0.2 - 0.9 ahead of two where there are few heads and 1 - 3 behind where there are 64.
template <bool BF16>
struct Four {
  uint4 raw;
  __device__ __forceinline__ void load(const void* p, size_t at) {
    if (BF16) {
      const uint2 v = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(p) + at);
      raw.x = v.x;
      raw.y = v.y;
    } else {
      raw = *reinterpret_cast<const uint4*>(static_cast<const float*>(p) + at);
    }
  }
  __device__ __forceinline__ void get(float (&v)[4]) const {
    if (BF16) {
      v[0] = bf_lo(raw.x), v[1] = bf_hi(raw.x), v[2] = bf_lo(raw.y), v[3] = bf_hi(raw.y);
    } else {
      v[0] = __uint_as_float(raw.x), v[1] = __uint_as_float(raw.y), v[2] = __uint_as_float(raw.z), v[3] = __uint_as_float(raw.w);
    }
  }
};
__device__ __forceinline__ void store_four(void* p, int dt, size_t at, const float (&v)[4]) {
  if (dt) *reinterpret_cast<float4*>(static_cast<float*>(p) + at) = make_float4(v[0], v[1], v[2], v[3]);
  else *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p) + at) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
}

template <bool BF16, int LPH, int TOK>   // LPH: lanes of a head
__global__ void __launch_bounds__(kThreads) rope_append_vec_kernel(const vila_rope_append_params p) {
  extern __shared__ __align__(16) float cs[];   // of each token: cos [rot/2] | sin [rot/2]
  constexpr int kDim = LPH * 8, kHeads = 32 / LPH;
  const int t0 = blockIdx.x * TOK, nt = min(TOK, p.T - t0), half = p.rot_dims >> 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, sub = lane / LPH, j = lane % LPH;
  const int maps = maps_of(p.maps), HQ = p.H * maps, GK = p.G * maps, heads = HQ + GK, V = p.G * p.vdim;
  const int groups = (heads + kHeads - 1) / kHeads;
  const int koff = GK * kDim, width = koff + V;
  const bool halves = p.rot_layout == 1, turned = (halves ? 4 * j < half : 8 * j < p.rot_dims);
  const int c0 = !halves ? 8 * j : turned ? 4 * j : p.rot_dims + 8 * j - 2 * half;
  const int c1 = halves && turned ? c0 + half : c0 + 4;
  // this warp's groups of heads, of all tokens one after the other
  int tok = 0, gr = warp - kWarps;
  auto step = [&]() {
    gr += kWarps;
    while (gr >= groups && tok < nt) {
      gr -= groups;
      ++tok;
    }
  };
  Four<BF16> x, y;
  auto fetch = [&]() {
    const int hh = gr * kHeads + sub;
    if (hh >= heads) return;
    const size_t src = static_cast<size_t>(t0 + tok) * p.ldq + hh * kDim;
    x.load(p.qkv, src + c0);
    y.load(p.qkv, src + c1);
  };
  step();
  if (tok < nt) fetch();
  const float mag = p.rot_mscale != 0.f ? p.rot_mscale : 1.0f;
  for (int c = tid; c < nt * half; c += kThreads) {
    const int at = TOK == 1 ? 0 : c / half, i = c - at * half;
    double s, co;
    sincos(static_cast<double>(p.positions[t0 + at]) * p.inv_freq[i], &s, &co);
    cs[at * p.rot_dims + i] = static_cast<float>(co) * mag;
    cs[at * p.rot_dims + half + i] = static_cast<float>(s) * mag;
  }
  __syncthreads();
  while (tok < nt) {
    const int t = t0 + tok, hh = gr * kHeads + sub;
    const bool live = hh < heads, is_q = hh < HQ;
    float u[4] = {}, v[4] = {}, ru[4], rv[4];
    if (live) {
      x.get(u);
      y.get(v);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) ru[k] = u[k], rv[k] = v[k];
    if (turned) {
      const float* angle = cs + tok * p.rot_dims;
      if (halves) {
        const float4 c = *reinterpret_cast<const float4*>(angle + 4 * j), s = *reinterpret_cast<const float4*>(angle + half + 4 * j);
        const float co[4] = {c.x, c.y, c.z, c.w}, si[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          u[k] = fmaf(ru[k], co[k], -(rv[k] * si[k]));
          v[k] = fmaf(rv[k], co[k], ru[k] * si[k]);
        }
      } else {
        const float4 c = *reinterpret_cast<const float4*>(angle + 4 * j), s = *reinterpret_cast<const float4*>(angle + half + 4 * j);
        u[0] = fmaf(ru[0], c.x, -(ru[1] * s.x));
        u[1] = fmaf(ru[1], c.x, ru[0] * s.x);
        u[2] = fmaf(ru[2], c.y, -(ru[3] * s.y));
        u[3] = fmaf(ru[3], c.y, ru[2] * s.y);
        v[0] = fmaf(rv[0], c.z, -(rv[1] * s.z));
        v[1] = fmaf(rv[1], c.z, rv[0] * s.z);
        v[2] = fmaf(rv[2], c.w, -(rv[3] * s.w));
        v[3] = fmaf(rv[3], c.w, rv[2] * s.w);
      }
    }
    step();
    if (tok < nt) fetch();
    if (p.unit_norm) {
      float ss = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) ss = fmaf(u[k], u[k], fmaf(v[k], v[k], ss));
#pragma unroll
      for (int o = LPH / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float r = 1.0f / sqrtf(ss / static_cast<float>(kDim) + p.eps);
#pragma unroll
      for (int k = 0; k < 4; ++k) u[k] *= r, v[k] *= r;
    }
    if (!live) continue;
    const float* nw = is_q ? p.q_norm_w : p.k_norm_w;
    if (nw) {
#pragma unroll
      for (int k = 0; k < 4; ++k) u[k] *= nw[c0 + k], v[k] *= nw[c1 + k];
    }
    if (is_q) {
      const size_t q = (static_cast<size_t>(t) * HQ + hh) * kDim;
      store_four(p.q_out, VILA_DT_F32, q + c0, u);
      store_four(p.q_out, VILA_DT_F32, q + c1, v);
    } else {
      const size_t kd = static_cast<size_t>(p.cache_rows[t]) * width + (hh - HQ) * kDim;
      store_four(p.pool, p.pool_dtype, kd + c0, u);
      store_four(p.pool, p.pool_dtype, kd + c1, v);
      if (p.v_from_k) {   // the value is the key as it came in
        store_four(p.pool, p.pool_dtype, kd + koff + c0, ru);
        store_four(p.pool, p.pool_dtype, kd + koff + c1, rv);
      }
    }
  }
  if (p.v_from_k) return;
  const int per = V >> 2;
  for (int c = tid; c < nt * per; c += kThreads) {
    const int at = TOK == 1 ? 0 : c / per, i = (c - at * per) * 4, t = t0 + at;
    Four<BF16> in;
    in.load(p.qkv, static_cast<size_t>(t) * p.ldq + heads * kDim + i);
    float v[4];
    in.get(v);
    if (p.v_first)   // part of the value comes from another layer's value of the same token
#pragma unroll
      for (int k = 0; k < 4; ++k)
        v[k] = fmaf(p.v_mix, ld_any(p.v_first, p.v_first_dtype, static_cast<size_t>(t) * p.ld_vf + i + k), (1.0f - p.v_mix) * v[k]);
    store_four(p.pool, p.pool_dtype, static_cast<size_t>(p.cache_rows[t]) * width + koff + i, v);
  }
}

// ---- attention -----------------------------------------------------------------------------------------
struct AttnShape {
  int BQ;      // query rows per CTA
  int BK;      // keys per block (<= 32: one lane per key in the softmax step)
  int sub;     // CTAs per 16-row tile (grid.y)
  int hsplit;  // head groups per tile (grid.z of the tiled kernel, inside grid.y of the other): 1 = all heads in one
               // CTA, G = one K/V head and its query heads per CTA (possible when the heads' scores are not mixed)
  int phase;   // weights mixed after the softmax with the keys of a row dealt to several CTAs: 0 = this launch only
               // leaves every CTA's running (max, sum) in its partial record, 1 = this launch merges those records and
               // adds its share of the values; -1 = one CTA does both passes itself
};

// K | V rows of a key block, widened to fp32.  16-byte loads when the head sizes allow (bf16: multiples of 8, fp32:
// multiples of 4; the pool row is then 16-byte aligned as well): the block's pieces are dealt to all threads (a warp per
// key where rows are wide), and a thread has kLoads of them in flight before it stores the first.  Otherwise a warp per key, element by element.
// g0, G: the value heads g0 .. g0 + G - 1 of the pool row are loaded with their key heads (as many, or one per map).
constexpr int kLoads = 4;

template <bool BF16>
__device__ __forceinline__ void load_kv_vec(float* Ks, float* Vs, const vila_paged_attn_params& p, const int32_t* pt, int j0,
                                            int nkeys, int BK, int DS, int V4, int nthreads, int g0, int G, bool with_v) {
  constexpr int E = BF16 ? 8 : 4;   // elements of a piece
  const int maps = maps_of(p.maps), GK = G * maps, D = p.dim, V = p.vdim, KS = key_stride(GK, DS);
  const size_t prw = static_cast<size_t>(p.G) * (maps * D + V);
  const size_t koff = static_cast<size_t>(g0) * maps * D;
  const size_t voff = static_cast<size_t>(p.G) * maps * D + static_cast<size_t>(g0) * V;
  const int kq = GK * D / E, per = kq + (with_v ? G * V / E : 0);   // pieces of a key: k, all
  auto fetch = [&](size_t row, int x) {
    const size_t at = row * prw + (x < kq ? koff + x * E : voff + (x - kq) * E);
    return BF16 ? __ldg(reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.pool) + at))
                : __ldg(reinterpret_cast<const uint4*>(static_cast<const float*>(p.pool) + at));
  };
  auto store = [&](int jj, int x, uint4 u) {
    const int e = x * E, g = e / D;
    float* d = x < kq ? Ks + jj * KS + g * DS + (e - g * D) : Vs + jj * G * V4 + (x - kq) * E;
    if (BF16) {
      *reinterpret_cast<float4*>(d) = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u),
                                                  __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
      *reinterpret_cast<float4*>(d + 4) = make_float4(__uint_as_float(u.z << 16), __uint_as_float(u.z & 0xffff0000u),
                                                      __uint_as_float(u.w << 16), __uint_as_float(u.w & 0xffff0000u));
    } else {
      *reinterpret_cast<uint4*>(d) = u;
    }
  };
  if (per >= 96) {   // wide rows (several heads): a warp per key
    for (int jj = threadIdx.x >> 5; jj < BK; jj += nthreads >> 5) {
      const bool ok = j0 + jj < nkeys;
      const size_t row = ok ? pool_row(pt, p.page, j0 + jj) : 0;
      for (int first = threadIdx.x & 31; first < per; first += 32 * kLoads) {
        uint4 u[kLoads];
#pragma unroll
        for (int i = 0; i < kLoads; ++i)
          u[i] = ok && first + 32 * i < per ? fetch(row, first + 32 * i) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int i = 0; i < kLoads; ++i)
          if (first + 32 * i < per) store(jj, first + 32 * i, u[i]);
      }
    }
    return;
  }
  for (int first = threadIdx.x; first < BK * per; first += kLoads * nthreads) {   // narrow rows: pieces dealt to all threads
    uint4 u[kLoads];
    int jj[kLoads], x[kLoads];
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      const int item = first + i * nthreads;
      jj[i] = item / per;
      x[i] = item - jj[i] * per;
      u[i] = item < BK * per && j0 + jj[i] < nkeys ? fetch(pool_row(pt, p.page, j0 + jj[i]), x[i]) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < kLoads; ++i)
      if (first + i * nthreads < BK * per) store(jj[i], x[i], u[i]);
  }
}

__device__ __forceinline__ void load_kv_block(float* Ks, float* Vs, const vila_paged_attn_params& p,
                                              const int32_t* pt, int j0, int nkeys, int BK, int D4, int DS, int V4,
                                              int nwarps, int g0, int G, bool with_v) {
  const int maps = maps_of(p.maps), GK = G * maps, D = p.dim, V = p.vdim;
  if (p.pool_dtype == VILA_DT_BF16 && (D & 7) == 0 && (V & 7) == 0) {
    load_kv_vec<true>(Ks, Vs, p, pt, j0, nkeys, BK, DS, V4, 32 * nwarps, g0, G, with_v);
    return;
  }
  if (p.pool_dtype == VILA_DT_F32 && (D & 3) == 0 && (V & 3) == 0) {
    load_kv_vec<false>(Ks, Vs, p, pt, j0, nkeys, BK, DS, V4, 32 * nwarps, g0, G, with_v);
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, KS = key_stride(GK, DS);
  const size_t prw = static_cast<size_t>(p.G) * (maps * D + V);
  const size_t koff = static_cast<size_t>(g0) * maps * D;
  const size_t voff = static_cast<size_t>(p.G) * maps * D + static_cast<size_t>(g0) * V;
  for (int jj = warp; jj < BK; jj += nwarps) {
    const int j = j0 + jj;
    float* kd = Ks + jj * KS;
    float* vd = Vs + jj * G * V4;
    if (j >= nkeys) {
      for (int x = lane; x < KS; x += 32) kd[x] = 0.f;
      for (int x = lane; x < G * V4; x += 32) vd[x] = 0.f;
      continue;
    }
    const size_t src = pool_row(pt, p.page, j) * prw, vsrc = src + voff;
    for (int x = lane; x < GK * D4; x += 32) {
      const int g = x / D4, k = x - g * D4;
      kd[g * DS + k] = k < D ? ld_any(p.pool, p.pool_dtype, src + koff + static_cast<size_t>(g) * D + k) : 0.f;
    }
    for (int x = lane; with_v && x < G * V4; x += 32) {
      const int g = x / V4, k = x - g * V4;
      vd[x] = k < V ? ld_any(p.pool, p.pool_dtype, vsrc + static_cast<size_t>(g) * V + k) : 0.f;
    }
  }
}

// Differential attention: a warp turns the two maps' finished rows of one head (fp32 in shared memory, V values each)
// into the head's output.
__device__ __forceinline__ void combine_maps(const vila_paged_attn_params& p, const float* a1, const float* a2, int row, int h) {
  const int lane = threadIdx.x & 31, V = p.vdim;
  float ss = 0.f;
  for (int c = lane; c < V; c += 32) {
    const float o = fmaf(-p.diff_lambda, a2[c], a1[c]);
    ss = fmaf(o, o, ss);
  }
  ss = warp_sum(ss);
  const float r = p.diff_scale / sqrtf(ss / static_cast<float>(V) + p.diff_eps) * out_gate(p, row, h);
  const size_t ob = (static_cast<size_t>(row) * p.H + h) * V;
  for (int c = lane; c < V; c += 32) st_any(p.out, p.out_dtype, ob + c, fmaf(-p.diff_lambda, a2[c], a1[c]) * r);
}

// Shared memory (floats):  Qs [BQ * H][D4] (scale folded in) | Ks [BK][G][DS] | Vs [BK][G][V4] |
//   Ss [BQ * H][BK] raw scores | Ps [BQ * H][BK] weights | talk [H * H] | m, l, alpha [BQ * H]
// H and G count score heads (a head's maps singly), the value heads are GV = G / maps.
// DS = D4 + 4: consecutive keys start 4 banks apart, so the float4 reads of 8 keys do not collide.
// CAP: with capped scores, whose instructions are not in the other form (uncapped prompts of mixed heads ran 3 % slower for
// them in tiles of 4 rows).
template <int NACC, bool CAP>   // few accumulators: registers for four CTAs on an SM, whose loads and barriers then overlap
__global__ void __launch_bounds__(kThreads, NACC <= 2 ? 4 : (NACC <= 8 ? 2 : 1)) paged_attn_kernel(const vila_paged_attn_params p, const AttnShape sh) {
  extern __shared__ __align__(16) float sm[];
  // H, G: the heads this CTA serves (all of them, or one value head with its key and query heads: h0 + h, g0 + g)
  const int maps = maps_of(p.maps), HT = p.H * maps, hs = blockIdx.y % sh.hsplit;
  const int H = HT / sh.hsplit, GV = p.G / sh.hsplit, G = GV * maps, h0 = hs * H, g0 = hs * GV;
  const int D = p.dim, V = p.vdim, BQ = sh.BQ, BK = sh.BK;
  const int D4 = round4(D), DS = D4 + 4, V4 = round4(V), R = BQ * H, rep = H / G, KS = key_stride(G, DS);
  float* Qs = sm;
  float* Ks = Qs + R * D4;
  float* Vs = Ks + BK * KS;
  float* Ss = Vs + BK * GV * V4;
  float* Ps = Ss + R * BK;
  float* Tk = Ps + R * BK;
  float* m_s = Tk + H * H;
  float* l_s = m_s + R;
  float* a_s = l_s + R;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int* tile = p.tiles + 4 * blockIdx.x;
  const int i0 = blockIdx.y / sh.hsplit * BQ;
  const int n_tile = tile[1];
  if (i0 >= n_tile) return;
  const int row0 = tile[0] + i0, n = min(BQ, n_tile - i0), pos0 = tile[2] + i0;
  const int32_t* pt = p.page_tables + static_cast<size_t>(tile[3]) * p.pt_stride;
  const int split = blockIdx.z, nsplit = gridDim.z;

  for (int idx = tid; idx < R * D4; idx += kThreads) {
    const int r = idx / D4, k = idx - r * D4, i = r / H, h = r - i * H;
    Qs[idx] = (i < n && k < D) ? p.q[(static_cast<size_t>(row0 + i) * HT + h0 + h) * D + k] * head_scale(p, h0 + h) : 0.f;
  }
  for (int idx = tid; idx < H * H; idx += kThreads) Tk[idx] = p.talk ? p.talk[idx] : ((idx / H) == (idx % H) ? 1.f : 0.f);
  const bool after = p.talk_after != 0 && p.talk != nullptr;
  for (int r = tid; r < R; r += kThreads) {
    const bool first = split == 0 && p.sink != nullptr && !after;
    m_s[r] = first ? p.sink[h0 + r % H] : kNegBig;
    l_s[r] = first ? 1.0f : 0.0f;
  }
  float4 acc[NACC];
#pragma unroll
  for (int a = 0; a < NACC; ++a) acc[a] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int vq = V4 >> 2;                 // float4 columns of a head
  const int nout = R * vq;                // float4 accumulators of the CTA: index o -> (r, c4)
  const int nkeys = pos0 + n;             // keys 0 .. nkeys - 1 are visible to the last row
  const BlockList bl = visible_blocks(p, pos0, nkeys, BK);

  const int pass_begin = after && sh.phase != 1 ? 0 : 1, pass_end = after && sh.phase == 0 ? 1 : 2;
  for (int pass = pass_begin; pass < pass_end; ++pass) {
  const bool stats = pass == 0;   // scores only: every head's running max and sum over the visible keys
  if (after && !stats) {
    __syncthreads();
    for (int r = tid; r < R; r += kThreads) {
      if (sh.phase == 1) {   // (max, sum) of every split's share, merged in split order
        const int i = r / H, h = r - i * H;
        float mx = kNegBig, l = 0.f;
        if (i < n) {
          const float* rec = p.partial + (static_cast<size_t>(row0 + i) * nsplit * H + h) * (V + 2) + V;
          const size_t step = static_cast<size_t>(H) * (V + 2);
          for (int s = 0; s < nsplit; ++s) mx = fmaxf(mx, rec[s * step]);
          for (int s = 0; s < nsplit; ++s) l += expf(rec[s * step] - mx) * rec[s * step + 1];
        }
        m_s[r] = mx;
        l_s[r] = l;
      }
      l_s[r] = l_s[r] > 0.f ? 1.0f / l_s[r] : 0.f;
    }
  }
  const bool all_blocks = stats && sh.phase < 0;
  for (int vb_ = all_blocks ? 0 : split; vb_ < bl.count; vb_ += all_blocks ? 1 : nsplit) {
    const int j0 = bl.block(vb_) * BK;
    __syncthreads();
    load_kv_block(Ks, Vs, p, pt, j0, nkeys, BK, D4, DS, V4, kWarps, g0, GV, !stats);
    __syncthreads();
    // raw scores of every (score row, key)
    for (int idx = tid; idx < R * BK; idx += kThreads) {
      const int r = idx / BK, jj = idx - r * BK, h = r % H;
      const float4* qr = reinterpret_cast<const float4*>(Qs + r * D4);
      const float4* kr = reinterpret_cast<const float4*>(Ks + jj * KS + key_head(h, maps, rep) * DS);
      float s = 0.f;
#pragma unroll 4
      for (int k = 0; k < (D4 >> 2); ++k) {
        const float4 a = qr[k], c = kr[k];
        s = fmaf(a.x, c.x, s); s = fmaf(a.y, c.y, s); s = fmaf(a.z, c.z, s); s = fmaf(a.w, c.w, s);
      }
      Ss[idx] = CAP ? capped(p, s) : s;
    }
    __syncthreads();
    if (after) {
      if (stats) {
        // every head's own scores: running max and sum, nothing else
        for (int r = warp; r < R; r += kWarps) {
          const int i = r / H;
          const bool valid = lane < BK && i < n && sees(p, pos0 + i, j0 + lane);
          const float s = valid ? Ss[r * BK + lane] : kNegBig;
          const float m_old = m_s[r];
          const float m_new = fmaxf(m_old, warp_max(s));
          const float ps = warp_sum(valid ? expf(s - m_new) : 0.f);
          if (lane == 0) {
            l_s[r] = l_s[r] * expf(m_old - m_new) + ps;
            m_s[r] = m_new;
          }
        }
        continue;
      }
      // final weights of every head (l_s holds 1 / sum), then their mix over heads; no rescaling of the sums
      for (int idx = tid; idx < R * BK; idx += kThreads) {
        const int r = idx / BK, jj = idx - r * BK, i = r / H;
        Ss[idx] = (i < n && sees(p, pos0 + i, j0 + jj)) ? expf(Ss[idx] - m_s[r]) * l_s[r] : 0.f;
      }
      __syncthreads();
      for (int r = warp; r < R; r += kWarps) {
        const int i = r / H, h = r - i * H;
        if (lane < BK) {
          const float* tk = Tk + h * H;
          const float* sr = Ss + (i * H) * BK + lane;
          float w = 0.f;
          for (int g = 0; g < H; ++g) w = fmaf(tk[g], sr[g * BK], w);
          Ps[r * BK + lane] = w;
        }
        if (lane == 0) a_s[r] = 1.0f;
      }
    } else
    // head mixing + mask + online softmax: a warp per score row, a lane per key
    for (int r = warp; r < R; r += kWarps) {
      const int i = r / H, h = r - i * H;
      const bool valid = lane < BK && i < n && sees(p, pos0 + i, j0 + lane);
      float s = 0.f;
      if (lane < BK) {
        if (p.talk) {
          const float* tk = Tk + h * H;
          const float* sr = Ss + (i * H) * BK + lane;
          for (int g = 0; g < H; ++g) s = fmaf(tk[g], sr[g * BK], s);
        } else {
          s = Ss[r * BK + lane];
        }
      }
      if (valid && p.dist_bias) s += dist_bias(p, pos0 + i - (j0 + lane), h0 + h);
      s = valid ? s : kNegBig;
      const float m_old = m_s[r];
      const float m_new = fmaxf(m_old, warp_max(s));
      const float pj = valid ? expf(s - m_new) : 0.f;
      const float ps = warp_sum(pj);
      if (lane < BK) Ps[r * BK + lane] = pj;
      if (lane == 0) {
        const float alpha = expf(m_old - m_new);
        a_s[r] = alpha;
        l_s[r] = l_s[r] * alpha + ps;
        m_s[r] = m_new;
      }
    }
    __syncthreads();
    // weighted sum of the values
#pragma unroll
    for (int a = 0; a < NACC; ++a) {
      const int o = tid + a * kThreads;
      if (o < nout) {
        const int r = o / vq, c4 = o - r * vq, h = r % H;
        const float alpha = a_s[r];
        float4 v = acc[a];
        v.x *= alpha; v.y *= alpha; v.z *= alpha; v.w *= alpha;
        const float* pr = Ps + r * BK;
        const float* vr = Vs + value_head(h, maps, rep) * V4 + 4 * c4;
        for (int jj = 0; jj < BK; ++jj) {
          const float pj = pr[jj];
          const float4 c = *reinterpret_cast<const float4*>(vr + jj * GV * V4);
          v.x = fmaf(pj, c.x, v.x); v.y = fmaf(pj, c.y, v.y); v.z = fmaf(pj, c.z, v.z); v.w = fmaf(pj, c.w, v.w);
        }
        acc[a] = v;
      }
    }
  }
  }
  __syncthreads();
  if (maps > 1 && nsplit == 1) {   // finished rows to shared memory (over the operands), then a warp per (row, head)
#pragma unroll
    for (int a = 0; a < NACC; ++a) {
      const int o = tid + a * kThreads;
      if (o < nout) {
        const float inv = 1.0f / l_s[o / vq];
        acc[a].x *= inv; acc[a].y *= inv; acc[a].z *= inv; acc[a].w *= inv;
      }
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < NACC; ++a) {
      const int o = tid + a * kThreads;
      if (o < nout) *reinterpret_cast<float4*>(sm + 4 * o) = acc[a];   // [R][V4]
    }
    __syncthreads();
    const int HM = H / maps;   // heads of this CTA
    for (int u = warp; u < n * HM; u += kWarps) {
      const int i = u / HM, h = u - i * HM;
      const float* a1 = sm + (i * H + 2 * h) * V4;
      combine_maps(p, a1, a1 + V4, row0 + i, h0 / maps + h);
    }
    return;
  }
#pragma unroll
  for (int a = 0; a < NACC; ++a) {
    const int o = tid + a * kThreads;
    if (o >= nout) continue;
    const int r = o / vq, c4 = o - r * vq, i = r / H, h = r - i * H;
    if (i >= n) continue;
    const float v[4] = {acc[a].x, acc[a].y, acc[a].z, acc[a].w};
    if (nsplit == 1) {
      const float inv = after ? out_gate(p, row0 + i, h0 + h) : out_gate(p, row0 + i, h0 + h) / l_s[r];
      const size_t ob = (static_cast<size_t>(row0 + i) * HT + h0 + h) * V + 4 * c4;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (4 * c4 + e < V) st_any(p.out, p.out_dtype, ob + e, v[e] * inv);
    } else {
      float* part = p.partial + ((static_cast<size_t>(row0 + i) * nsplit + split) * HT + h0 + h) * (V + 2);
      if (!(after && sh.phase == 0)) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (4 * c4 + e < V) part[4 * c4 + e] = v[e];
      }
      // with the weights mixed afterwards the (max, sum) slots belong to the first launch: the second one reads them
      if (c4 == 0 && !(after && sh.phase == 1)) { part[V] = m_s[r]; part[V + 1] = l_s[r]; }
    }
  }
}

// Prompt portions that neither tensor-core kernel takes: BQ (a multiple of 4) rows x all heads per CTA, register-tiled.  Score rows are ordered
// head-major (r = h * BQ + i) so that 4 consecutive score rows are 4 query rows of ONE head: they share
// the key / value head, and a thread that owns such a block of 4 keeps
//   scores:        TR (4, or 2 with 512 threads) rows x 2 keys (jp and jp + BK / 2) per thread, q and k as float4
//                  pieces: 6 shared loads per 32 multiply-adds (4 per 16)
//   weighted sum:  4 rows x 4 value columns per accumulator, the 4 weights of a key as ONE float4
//                  (Ps is [row block][key][4]): 2 shared loads per 16 multiply-adds
// Shared memory (floats): Qs [R][D4] | Ks [BK][G][DS] | Vs [BK][G][V4] | Ss [R][BK] | Ps [R / 4][BK][4] |
//   m, l, alpha [R] | talk [H * H]
template <int NACC, int NT, int TR, bool CAP>
__global__ void __launch_bounds__(NT) paged_attn_tile4_kernel(const vila_paged_attn_params p, const AttnShape sh) {
  extern __shared__ __align__(16) float sm[];
  // H, G: the heads this CTA serves (all of them, or one K/V head with its query heads: global heads h0 + h, g0 + g)
  const int maps = maps_of(p.maps), HT = p.H * maps;
  const int H = HT / sh.hsplit, GV = p.G / sh.hsplit, G = GV * maps, h0 = blockIdx.z * H, g0 = blockIdx.z * GV;
  const int D = p.dim, V = p.vdim, BQ = sh.BQ, BK = sh.BK, HK = sh.BK >> 1;
  const int D4 = round4(D), DS = D4 + 4, V4 = round4(V), R = BQ * H, NB = R >> 2, rep = H / G, KS = key_stride(G, DS);
  float* Qs = sm;
  float* Ks = Qs + R * D4;
  float* Vs = Ks + BK * KS;
  float* Ss = Vs + BK * GV * V4;
  float* Ps = Ss + R * BK;
  float* m_s = Ps + R * BK;
  float* l_s = m_s + R;
  float* a_s = l_s + R;
  float* Tk = a_s + R;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int* tile = p.tiles + 4 * blockIdx.x;
  const int i0 = blockIdx.y * BQ;
  const int n_tile = tile[1];
  if (i0 >= n_tile) return;
  const int row0 = tile[0] + i0, n = min(BQ, n_tile - i0), pos0 = tile[2] + i0;
  const int32_t* pt = p.page_tables + static_cast<size_t>(tile[3]) * p.pt_stride;

  for (int idx = tid; idx < R * D4; idx += NT) {
    const int r = idx / D4, k = idx - r * D4, h = r / BQ, i = r - h * BQ;
    Qs[idx] = (i < n && k < D) ? p.q[(static_cast<size_t>(row0 + i) * HT + h0 + h) * D + k] * head_scale(p, h0 + h) : 0.f;
  }
  for (int idx = tid; idx < H * H; idx += NT) Tk[idx] = p.talk ? p.talk[idx] : ((idx / H) == (idx % H) ? 1.f : 0.f);
  const bool after = p.talk_after != 0 && p.talk != nullptr;
  for (int r = tid; r < R; r += NT) {
    const bool sink = p.sink != nullptr && !after;
    m_s[r] = sink ? p.sink[h0 + r / BQ] : kNegBig;
    l_s[r] = sink ? 1.0f : 0.0f;
  }
  float4 acc[NACC][4];
#pragma unroll
  for (int a = 0; a < NACC; ++a)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[a][k] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int vq = V4 >> 2;
  const int nout = NB * vq;               // accumulator items of the CTA: o -> (row block, float4 column)
  const int nkeys = pos0 + n;
  const int d4n = D4 >> 2;

  const BlockList bl = visible_blocks(p, pos0, nkeys, BK);
  for (int pass = after ? 0 : 1; pass < 2; ++pass) {
  const bool stats = pass == 0;   // scores only: every head's running max and sum over all visible keys
  if (after && !stats) {
    __syncthreads();
    for (int r = tid; r < R; r += NT) l_s[r] = l_s[r] > 0.f ? 1.0f / l_s[r] : 0.f;
  }
  for (int vb_ = 0; vb_ < bl.count; ++vb_) {
    const int j0 = bl.block(vb_) * BK;
    __syncthreads();
    load_kv_block(Ks, Vs, p, pt, j0, nkeys, BK, D4, DS, V4, NT / 32, g0, GV, !stats);
    __syncthreads();
    for (int item = tid; item < (R / TR) * HK; item += NT) {
      const int rbs = item / HK, jp = item - rbs * HK, r0 = rbs * TR;     // TR score rows of one head x 2 keys
      const int g = key_head(r0 / BQ, maps, rep);
      const float4* q0 = reinterpret_cast<const float4*>(Qs + r0 * D4);
      const float4* k0 = reinterpret_cast<const float4*>(Ks + jp * KS + g * DS);
      const float4* k1 = reinterpret_cast<const float4*>(Ks + (jp + HK) * KS + g * DS);
      float s[TR][2];
#pragma unroll
      for (int a = 0; a < TR; ++a) s[a][0] = s[a][1] = 0.f;
#pragma unroll 2
      for (int k = 0; k < d4n; ++k) {
        const float4 ka = k0[k], kb = k1[k];
#pragma unroll
        for (int a = 0; a < TR; ++a) {
          const float4 qv = q0[a * d4n + k];
          s[a][0] = fmaf(qv.x, ka.x, s[a][0]); s[a][0] = fmaf(qv.y, ka.y, s[a][0]);
          s[a][0] = fmaf(qv.z, ka.z, s[a][0]); s[a][0] = fmaf(qv.w, ka.w, s[a][0]);
          s[a][1] = fmaf(qv.x, kb.x, s[a][1]); s[a][1] = fmaf(qv.y, kb.y, s[a][1]);
          s[a][1] = fmaf(qv.z, kb.z, s[a][1]); s[a][1] = fmaf(qv.w, kb.w, s[a][1]);
        }
      }
#pragma unroll
      for (int a = 0; a < TR; ++a) {
        Ss[(r0 + a) * BK + jp] = CAP ? capped(p, s[a][0]) : s[a][0];
        Ss[(r0 + a) * BK + jp + HK] = CAP ? capped(p, s[a][1]) : s[a][1];
      }
    }
    __syncthreads();
    if (after) {
      if (stats) {
        for (int r = warp; r < R; r += NT / 32) {
          const int i = r % BQ;
          const bool valid = lane < BK && i < n && sees(p, pos0 + i, j0 + lane);
          const float s = valid ? Ss[r * BK + lane] : kNegBig;
          const float m_old = m_s[r];
          const float m_new = fmaxf(m_old, warp_max(s));
          const float ps = warp_sum(valid ? expf(s - m_new) : 0.f);
          if (lane == 0) {
            l_s[r] = l_s[r] * expf(m_old - m_new) + ps;
            m_s[r] = m_new;
          }
        }
        continue;
      }
      for (int idx = tid; idx < R * BK; idx += NT) {
        const int r = idx / BK, jj = idx - r * BK, i = r % BQ;
        Ss[idx] = (i < n && sees(p, pos0 + i, j0 + jj)) ? expf(Ss[idx] - m_s[r]) * l_s[r] : 0.f;
      }
      __syncthreads();
      for (int r = warp; r < R; r += NT / 32) {
        const int h = r / BQ, i = r - h * BQ;
        if (lane < BK) {
          const float* tk = Tk + h * H;
          const float* sr = Ss + i * BK + lane;
          float w = 0.f;
          for (int g = 0; g < H; ++g) w = fmaf(tk[g], sr[g * BQ * BK], w);
          Ps[(((r >> 2) * BK + lane) << 2) + (r & 3)] = w;
        }
        if (lane == 0) a_s[r] = 1.0f;
      }
    } else
    // head mixing + mask + online softmax: a warp takes 4 score rows at a time (rows warp, warp + 8, ...), a
    // lane per key; the 4 rows' reductions are interleaved so that their shuffles overlap
    for (int rbase = warp; rbase < R; rbase += 4 * (NT / 32)) {
      float sv[4], mo[4], mn[4], pj[4], ps[4];
      bool ok[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = rbase + u * (NT / 32);
        sv[u] = kNegBig;
        ok[u] = false;
        mo[u] = kNegBig;
        if (r < R) {
          const int h = r / BQ, i = r - h * BQ;
          ok[u] = lane < BK && i < n && sees(p, pos0 + i, j0 + lane);
          if (lane < BK) {
            float s0 = 0.f, s1 = 0.f;
            if (p.talk) {
              const float* tk = Tk + h * H;
              const float* sr = Ss + i * BK + lane;
              int g = 0;
              for (; g + 1 < H; g += 2) {
                s0 = fmaf(tk[g], sr[g * BQ * BK], s0);
                s1 = fmaf(tk[g + 1], sr[(g + 1) * BQ * BK], s1);
              }
              if (g < H) s0 = fmaf(tk[g], sr[g * BQ * BK], s0);
            } else {
              s0 = Ss[r * BK + lane];
            }
            if (ok[u]) sv[u] = s0 + s1 + (p.dist_bias ? dist_bias(p, pos0 + i - (j0 + lane), h0 + h) : 0.f);
          }
          mo[u] = m_s[r];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) mn[u] = sv[u];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < 4; ++u) mn[u] = fmaxf(mn[u], __shfl_xor_sync(0xffffffffu, mn[u], o));
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        mn[u] = fmaxf(mn[u], mo[u]);
        pj[u] = ok[u] ? expf(sv[u] - mn[u]) : 0.f;
        ps[u] = pj[u];
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < 4; ++u) ps[u] += __shfl_xor_sync(0xffffffffu, ps[u], o);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = rbase + u * (NT / 32);
        if (r < R) {
          if (lane < BK) Ps[(((r >> 2) * BK + lane) << 2) + (r & 3)] = pj[u];
          if (lane == 0) {
            const float alpha = expf(mo[u] - mn[u]);
            a_s[r] = alpha;
            l_s[r] = l_s[r] * alpha + ps[u];
            m_s[r] = mn[u];
          }
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < NACC; ++a) {
      const int o = tid + a * NT;
      if (o < nout) {
        const int rb = o / vq, c4 = o - rb * vq;
        const int g = value_head((rb << 2) / BQ, maps, rep);
        const float4 al = *reinterpret_cast<const float4*>(a_s + (rb << 2));
        const float alv[4] = {al.x, al.y, al.z, al.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          acc[a][k].x *= alv[k]; acc[a][k].y *= alv[k]; acc[a][k].z *= alv[k]; acc[a][k].w *= alv[k];
        }
        const float4* pr = reinterpret_cast<const float4*>(Ps + ((rb * BK) << 2));
        const float* vr = Vs + g * V4 + 4 * c4;
#pragma unroll 4
        for (int jj = 0; jj < BK; ++jj) {
          const float4 pw = pr[jj];
          const float4 c = *reinterpret_cast<const float4*>(vr + jj * GV * V4);
          const float pv[4] = {pw.x, pw.y, pw.z, pw.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            acc[a][k].x = fmaf(pv[k], c.x, acc[a][k].x); acc[a][k].y = fmaf(pv[k], c.y, acc[a][k].y);
            acc[a][k].z = fmaf(pv[k], c.z, acc[a][k].z); acc[a][k].w = fmaf(pv[k], c.w, acc[a][k].w);
          }
        }
      }
    }
  }
  }
  __syncthreads();
  if (maps > 1) {   // finished rows to shared memory (over the operands), then a warp per (row, head)
#pragma unroll
    for (int a = 0; a < NACC; ++a) {
      const int o = tid + a * NT;
      if (o < nout) {
        const int r0 = (o / vq) << 2;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float inv = 1.0f / l_s[r0 + k];
          acc[a][k].x *= inv; acc[a][k].y *= inv; acc[a][k].z *= inv; acc[a][k].w *= inv;
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < NACC; ++a) {
      const int o = tid + a * NT;
      if (o < nout) {
        const int rb = o / vq, c4 = o - rb * vq;
#pragma unroll
        for (int k = 0; k < 4; ++k) *reinterpret_cast<float4*>(sm + ((rb << 2) + k) * V4 + 4 * c4) = acc[a][k];   // [R][V4]
      }
    }
    __syncthreads();
    const int HM = H / maps;   // heads of this CTA
    for (int u = warp; u < n * HM; u += NT / 32) {
      const int i = u / HM, h = u - i * HM;
      const float* a1 = sm + (2 * h * BQ + i) * V4;
      combine_maps(p, a1, a1 + BQ * V4, row0 + i, h0 / maps + h);
    }
    return;
  }
#pragma unroll
  for (int a = 0; a < NACC; ++a) {
    const int o = tid + a * NT;
    if (o >= nout) continue;
    const int rb = o / vq, c4 = o - rb * vq;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int r = (rb << 2) + k, h = r / BQ, i = r - h * BQ;
      if (i >= n) continue;
      const float inv = after ? out_gate(p, row0 + i, h0 + h) : out_gate(p, row0 + i, h0 + h) / l_s[r];
      const float v[4] = {acc[a][k].x, acc[a][k].y, acc[a][k].z, acc[a][k].w};
      const size_t ob = (static_cast<size_t>(row0 + i) * p.H + h0 + h) * V + 4 * c4;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (4 * c4 + e < V) st_any(p.out, p.out_dtype, ob + e, v[e] * inv);
    }
  }
}

// one CTA per (decoded row, head): combine the nsplit partial triples in split order
__global__ void __launch_bounds__(128) paged_attn_merge_kernel(const vila_paged_attn_params p) {
  const int* tile = p.tiles + 4 * blockIdx.x;
  const int row = tile[0], h = blockIdx.y, V = p.vdim, ns = p.nsplit;
  const float* part = p.partial + (static_cast<size_t>(row) * ns * p.H + h) * (V + 2);
  const size_t stride = static_cast<size_t>(p.H) * (V + 2);
  if (p.talk_after != 0 && p.talk != nullptr) {   // the partial sums carry final weights: add them in split order
    const float gt = out_gate(p, row, h);
    for (int k = threadIdx.x; k < V; k += blockDim.x) {
      float a = 0.f;
      for (int s = 0; s < ns; ++s) a += part[s * stride + k];
      st_any(p.out, p.out_dtype, (static_cast<size_t>(row) * p.H + h) * V + k, a * gt);
    }
    return;
  }
  float mx = kNegBig;
  for (int s = 0; s < ns; ++s) mx = fmaxf(mx, part[s * stride + V]);
  float den = 0.f;
  for (int s = 0; s < ns; ++s) den += expf(part[s * stride + V] - mx) * part[s * stride + V + 1];
  const float inv = out_gate(p, row, h) / den;
  for (int k = threadIdx.x; k < V; k += blockDim.x) {
    float a = 0.f;
    for (int s = 0; s < ns; ++s) a += expf(part[s * stride + V] - mx) * part[s * stride + k];
    st_any(p.out, p.out_dtype, (static_cast<size_t>(row) * p.H + h) * V + k, a * inv);
  }
}

// one CTA per (decoded row, head) of differential attention: both maps' partial triples in split order, then the pair
__global__ void __launch_bounds__(128) paged_attn_merge_maps_kernel(const vila_paged_attn_params p) {
  extern __shared__ float o_s[];   // [V] a1 - lambda a2 | [4] partial sums of squares
  const int* tile = p.tiles + 4 * blockIdx.x;
  const int row = tile[0], h = blockIdx.y, V = p.vdim, ns = p.nsplit, HT = 2 * p.H;
  const float* part = p.partial + (static_cast<size_t>(row) * ns * HT + 2 * h) * (V + 2);
  const size_t stride = static_cast<size_t>(HT) * (V + 2);
  float mx[2], inv[2];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const float* pm = part + m * (V + 2) + V;
    mx[m] = kNegBig;
    for (int s = 0; s < ns; ++s) mx[m] = fmaxf(mx[m], pm[s * stride]);
    float den = 0.f;
    for (int s = 0; s < ns; ++s) den += expf(pm[s * stride] - mx[m]) * pm[s * stride + 1];
    inv[m] = 1.0f / den;
  }
  float ss = 0.f;
  for (int k = threadIdx.x; k < V; k += blockDim.x) {
    float a[2] = {0.f, 0.f};
    for (int s = 0; s < ns; ++s)
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const float* pm = part + s * stride + m * (V + 2);
        a[m] += expf(pm[V] - mx[m]) * pm[k];
      }
    const float o = fmaf(-p.diff_lambda, a[1] * inv[1], a[0] * inv[0]);
    o_s[k] = o;
    ss = fmaf(o, o, ss);
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) o_s[V + (threadIdx.x >> 5)] = ss;
  __syncthreads();
  ss = (o_s[V] + o_s[V + 1]) + (o_s[V + 2] + o_s[V + 3]);
  const float r = p.diff_scale / sqrtf(ss / static_cast<float>(V) + p.diff_eps) * out_gate(p, row, h);
  for (int k = threadIdx.x; k < V; k += blockDim.x)
    st_any(p.out, p.out_dtype, (static_cast<size_t>(row) * p.H + h) * V + k, o_s[k] * r);
}

// H, G: heads of the CTA (of the model, maps not counted singly)
size_t attn_smem(const vila_paged_attn_params& p, int BQ, int BK, int H = 0, int G = 0) {
  if (H == 0) { H = p.H; G = p.G; }
  const int maps = maps_of(p.maps), GV = G;
  H *= maps;
  G *= maps;
  const int D4 = round4(p.dim), V4 = round4(p.vdim), R = BQ * H;
  const size_t work = static_cast<size_t>(R) * D4 + static_cast<size_t>(BK) * key_stride(G, D4 + 4) +
                      static_cast<size_t>(BK) * GV * V4 + 2 * static_cast<size_t>(R) * BK + H * H + 3 * R;
  const size_t rows = maps > 1 ? static_cast<size_t>(R) * V4 : 0;   // the maps' finished rows, over the same memory
  return sizeof(float) * (work > rows ? work : rows);
}

}  // namespace

int rope_append(const vila_rope_append_params& p, cudaStream_t stream) {
  if (p.T <= 0) return 0;
  VB_CHECK(p.H >= 1 && p.G >= 1 && p.dim >= 1 && p.vdim >= 1 && p.rot_dims >= 0 && p.rot_dims <= p.dim &&
               p.rot_dims % 2 == 0 && (p.rot_dims == 0 || p.inv_freq != nullptr) && (!p.v_from_k || p.vdim == p.dim) &&
               (p.rot_layout == 0 || p.rot_layout == 1) && p.maps >= 0 && p.maps <= 2 && (p.maps < 2 || !p.v_from_k),
           "rope_append: H=%d G=%d dim=%d vdim=%d rot_dims=%d v_from_k=%d", p.H, p.G, p.dim, p.vdim, p.rot_dims,
           p.v_from_k);
  const size_t cs_bytes = sizeof(float) * (p.rot_dims + 2);
  // four columns at a time: every run of four starts on 8 bytes (bf16) or 16 (fp32)
  const bool fours = (p.dim == 64 || p.dim == 128 || p.dim == 256) && p.rot_dims % 8 == 0 && p.vdim % 4 == 0 && p.ldq % 4 == 0 &&
                     (reinterpret_cast<uintptr_t>(p.qkv) & (p.qkv_dtype == VILA_DT_BF16 ? 7 : 15)) == 0 &&
                     (reinterpret_cast<uintptr_t>(p.pool) & (p.pool_dtype == VILA_DT_BF16 ? 7 : 15)) == 0 &&
                     (reinterpret_cast<uintptr_t>(p.q_out) & 15) == 0;
  if (fours) {
    const size_t angles = sizeof(float) * p.rot_dims;
#define VB_ROPE_TOK(LPH, TOK)                                                                                                     \
  do {                                                                                                                            \
    const dim3 grid((p.T + TOK - 1) / TOK);                                                                                       \
    if (p.qkv_dtype == VILA_DT_BF16)                                                                                              \
      VB_CUDA(launch_serial(rope_append_vec_kernel<true, LPH, TOK>, grid, dim3(kThreads), TOK * angles, stream, p));              \
    else                                                                                                                          \
      VB_CUDA(launch_serial(rope_append_vec_kernel<false, LPH, TOK>, grid, dim3(kThreads), TOK * angles, stream, p));             \
  } while (0)
#define VB_ROPE_VEC(LPH)                         \
  do {                                           \
    if (p.T > 4 * num_sms()) VB_ROPE_TOK(LPH, 2); \
    else VB_ROPE_TOK(LPH, 1);                    \
  } while (0)
    if (p.dim == 64) VB_ROPE_VEC(8);
    else if (p.dim == 128) VB_ROPE_VEC(16);
    else VB_ROPE_VEC(32);
#undef VB_ROPE_VEC
#undef VB_ROPE_TOK
    return 0;
  }
  if (p.dim % 2 == 0 && p.dim <= 256) {
#define VB_ROPE(NP)                                                                                                    \
  do {                                                                                                                 \
    if (p.qkv_dtype == VILA_DT_BF16)                                                                                   \
      VB_CUDA(launch_serial(rope_append_pairs_kernel<true, NP>, dim3(p.T), dim3(kThreads), cs_bytes, stream, p));      \
    else                                                                                                               \
      VB_CUDA(launch_serial(rope_append_pairs_kernel<false, NP>, dim3(p.T), dim3(kThreads), cs_bytes, stream, p));     \
  } while (0)
    if (p.dim <= 64) VB_ROPE(1);
    else if (p.dim <= 128) VB_ROPE(2);
    else VB_ROPE(4);
#undef VB_ROPE
    return 0;
  }
  VB_CUDA(launch_serial(rope_append_kernel, dim3(p.T), dim3(kThreads), sizeof(float) * (p.rot_dims + 2), stream, p));
  return 0;
}

int paged_attention(const vila_paged_attn_params& p, cudaStream_t stream, int tries) {
  if (p.ntiles <= 0) return 0;
  VB_CHECK(p.H >= 1 && p.G >= 1 && p.H % p.G == 0 && p.dim >= 1 && p.vdim >= 1 && p.page >= 1 && p.nsplit >= 1 &&
               p.nsplit <= 64 && (p.nsplit == 1 || p.partial != nullptr),
           "paged_attention: H=%d G=%d dim=%d vdim=%d page=%d nsplit=%d", p.H, p.G, p.dim, p.vdim, p.page, p.nsplit);
  constexpr size_t kSmemMax = 224 * 1024;
  VB_CHECK(p.chunk >= 0 && (p.dist_bias == nullptr || p.dist_rows >= 1), "paged_attention: chunk=%d dist_rows=%d",
           p.chunk, p.dist_rows);
  VB_CHECK(p.softcap >= 0.f, "paged_attention: softcap=%f", p.softcap);
  VB_CHECK(p.window >= 0 && p.keep_first >= 0 && (p.talk_after == 0 || (p.talk != nullptr && p.sink == nullptr)),
           "paged_attention: window=%d keep_first=%d; talk_after needs talk and no sink", p.window, p.keep_first);
  VB_CHECK(p.maps >= 0 && p.maps <= 2 &&
               (p.maps < 2 || (p.talk == nullptr && p.sink == nullptr && p.dist_bias == nullptr && p.head_scale == nullptr)),
           "paged_attention: maps=%d (two maps per head take no head mixing, sink, distance bias or head scale)", p.maps);
  VB_CHECK(p.max_rows >= 1 && p.max_rows <= 16 && (p.nsplit == 1 || p.max_rows == 1),
           "paged_attention: max_rows=%d nsplit=%d (key splitting serves one-row tiles)", p.max_rows, p.nsplit);
  if (paged_attention_tc_takes(p)) return paged_attention_tc(p, stream, tries);
  VB_CHECK(tries == -1, "paged_attention: the kernel with limited waits does not take this call");
  if (paged_attention_mma_takes(p)) return paged_attention_mma(p, stream);
  if (paged_attention_mix_takes(p)) return paged_attention_mix(p, stream);
  if (paged_attention_decode_takes(p)) return paged_attention_decode(p, stream);
  AttnShape sh;
  sh.phase = -1;
  // Without head mixing the K/V-head groups are independent: a CTA then serves ONE K/V head and its query heads, holds
  // a quarter .. an eighth of the K | V block, and takes more rows of the sequence instead.
  sh.hsplit = p.talk == nullptr ? p.G : 1;
  const int maps = maps_of(p.maps), Hl = p.H / sh.hsplit, Gl = p.G / sh.hsplit, Sl = Hl * maps;   // Sl: score heads of a CTA
  if (p.max_rows > 1 && Sl <= 32) {
    // prompt portions: the register-tiled kernel, 4 .. 16 rows per CTA (about 64 score rows, 128 at most)
    sh.BQ = 16;
    while (sh.BQ > 4 && sh.BQ * Sl > 64) sh.BQ >>= 1;
    sh.BK = 32;
    while (attn_smem(p, sh.BQ, sh.BK, Hl, Gl) > kSmemMax && sh.BK > 8) sh.BK >>= 1;
    const size_t smem4 = attn_smem(p, sh.BQ, sh.BK, Hl, Gl);
    const int items = (sh.BQ * Sl / 4) * (round4(p.vdim) >> 2);      // accumulator items (4 rows x 4 columns)
    // 512 threads (16 warps on the SM, 2-row score tiles) when there is accumulator work for them
    const int nt = items >= 512 ? 512 : 256;
    const int nacc4 = (items + nt - 1) / nt;
    if (smem4 <= kSmemMax && nacc4 <= (nt == 512 ? 2 : 4)) {
      sh.sub = (p.max_rows + sh.BQ - 1) / sh.BQ;
      const dim3 grid4(p.ntiles, sh.sub, sh.hsplit);
#define VB_PAGED4(N, NT, TR)                                                                                     \
  do {                                                                                                           \
    const auto kernel = p.softcap > 0.f ? paged_attn_tile4_kernel<N, NT, TR, true> : paged_attn_tile4_kernel<N, NT, TR, false>; \
    if (smem4 > 48 * 1024)                                                                                       \
      VB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem4))); \
    VB_CUDA(launch_serial(kernel, grid4, dim3(NT), smem4, stream, p, sh));                                       \
  } while (0)
      if (nt == 512) {
        if (nacc4 <= 1) VB_PAGED4(1, 512, 2);
        else VB_PAGED4(2, 512, 2);
      } else if (nacc4 <= 1) VB_PAGED4(1, 256, 4);
      else if (nacc4 <= 2) VB_PAGED4(2, 256, 4);
      else VB_PAGED4(4, 256, 4);
#undef VB_PAGED4
      return 0;
    }
  }
  // decoded tokens (one-row tiles, keys optionally split over CTAs) and shapes the tiled kernel does not take
  sh.BQ = 1;
  while (sh.BQ < p.max_rows) sh.BQ <<= 1;
  while (sh.BQ > 1 && sh.BQ * Sl > 64) sh.BQ >>= 1;
  sh.BK = 32;
  while (attn_smem(p, sh.BQ, sh.BK, Hl, Gl) > kSmemMax && sh.BK > 4) sh.BK >>= 1;
  while (attn_smem(p, sh.BQ, sh.BK, Hl, Gl) > kSmemMax && sh.BQ > 1) sh.BQ >>= 1;
  const size_t smem = attn_smem(p, sh.BQ, sh.BK, Hl, Gl);
  VB_CHECK(smem <= kSmemMax, "paged_attention: H=%d G=%d dim=%d vdim=%d need %zu bytes of shared memory", p.H, p.G,
           p.dim, p.vdim, smem);
  sh.sub = (p.max_rows + sh.BQ - 1) / sh.BQ;
  const int nacc = (sh.BQ * Sl * (round4(p.vdim) >> 2) + kThreads - 1) / kThreads;
  VB_CHECK(nacc <= 16, "paged_attention: H=%d vdim=%d: %d accumulators per thread", p.H, p.vdim, nacc);
  const dim3 grid(p.ntiles, sh.sub * sh.hsplit, p.nsplit);
#define VB_PAGED(N)                                                                                              \
  do {                                                                                                           \
    const auto kernel = p.softcap > 0.f ? paged_attn_kernel<N, true> : paged_attn_kernel<N, false>;              \
    if (smem > 48 * 1024)                                                                                        \
      VB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem))); \
    VB_CUDA(launch_serial(kernel, grid, dim3(kThreads), smem, stream, p, sh));                                   \
  } while (0)
  // weights mixed after the softmax + split keys: the (max, sum) launch, then the launch that adds the values
  const int launches = (p.talk_after != 0 && p.nsplit > 1) ? 2 : 1;
  for (int l = 0; l < launches; ++l) {
    sh.phase = launches == 2 ? l : -1;
    if (nacc <= 1) VB_PAGED(1);
    else if (nacc <= 2) VB_PAGED(2);
    else if (nacc <= 4) VB_PAGED(4);
    else if (nacc <= 8) VB_PAGED(8);
    else VB_PAGED(16);
  }
#undef VB_PAGED
  if (p.nsplit > 1 && maps > 1)
    VB_CUDA(launch_serial(paged_attn_merge_maps_kernel, dim3(p.ntiles, p.H), dim3(128), sizeof(float) * (p.vdim + 4), stream, p));
  else if (p.nsplit > 1)
    VB_CUDA(launch_serial(paged_attn_merge_kernel, dim3(p.ntiles, p.H), dim3(128), 0, stream, p));
  return 0;
}

}  // namespace vb
