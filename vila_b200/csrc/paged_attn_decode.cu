// vila_paged_attention for decoded tokens over a bf16 pool (heads not mixed).
//
// What bounds a decoded token is latency: a few hundred keys per CTA, and the general kernel goes from global memory
// through shared memory, a barrier, the scores, a barrier, the softmax, a barrier, the values, for every 32 keys, and
// merges the key splits in a second launch.  Here a warp is on its own: it takes 16 keys at a time, half a warp per key,
// requests their 8 key and 8 value pieces per lane at once (16 bytes each, straight to registers), reduces the scores of
// all its heads with one transposing tree, keeps its own running (max, sum) and weighted sums, and meets the others only
// at the end: the 8 warps of a CTA through shared memory, the CTAs of a (token, key head) as a cluster through each
// other's shared memory, in warp and rank order.  fp32 throughout.
// 8 tokens x 1024 keys, 16 heads over 4: 25 us there with the merge, 11 here; 3 x 3000 keys 38 and 12, 8 x 4000
// 69 and 20 (two CTAs have to fit an SM: at 138 registers, one, the first took 26).
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "kernels.h"
#include "dtype_any.cuh"
#include "paged_attn_common.cuh"

namespace vb {
namespace {

constexpr int kWarps = 8, kThreads = 32 * kWarps, kKeys = 16, kV = 128;
constexpr unsigned kAll = 0xffffffffu;

// 16 bytes or zeros, requested where it is written.  The compiler moves other loads to their use, behind the scores: how many
// stayed in flight hung on what stands between (without the cap's branch 24 x 4000 keys of 8 heads over 2 took 50.2 us, with
// its quotient and tanhf 41.5, with the polynomial 41.8; now 37.8, with a cap 42.0 and 40.2).
__device__ __forceinline__ uint4 ld_now(const __nv_bfloat16* p, bool on) {
  uint4 v;
  asm volatile("{.reg .pred q;\nsetp.ne.b32 q, %5, 0;\nmov.b32 %0, 0;\nmov.b32 %1, 0;\nmov.b32 %2, 0;\nmov.b32 %3, 0;\n@q ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];}"
               : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w) : "l"(p), "r"(static_cast<int>(on)));
  return v;
}

// HM: model heads of a key head, MAPS: maps of a head (MAPS * D = 128 key columns).  Lane l of a half-warp holds key columns
// 8 l .. 8 l + 7 (of map l / R) and value columns 8 l .. 8 l + 7.
template <int HM, int MAPS>
__global__ void __launch_bounds__(kThreads, HM * MAPS <= 4 ? 2 : 1) paged_attn_decode_kernel(const vila_paged_attn_params p) {
  constexpr int SH = HM * MAPS, D = 128 / MAPS, R = 16 / MAPS;   // score heads, columns and lanes of a map
  constexpr int NV = HM * 8;                                     // scores of a lane's map: 8 keys x HM heads
  constexpr int PER = NV >= R ? NV / R : 1, DUP = NV >= R ? 1 : R / NV;   // scores a lane ends up with, lanes that share one
  constexpr int REC = kV + 2;
  __shared__ float rec_s[kWarps][SH][REC];                       // sums | max | sum of weights
  __shared__ float cta_s[SH][REC];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, hf = lane >> 4, l16 = lane & 15;
  const int map = l16 / R, r = l16 - map * R;
  const int C = gridDim.z, rank = blockIdx.z, g = blockIdx.y;
  const int* tile = p.tiles + 4 * blockIdx.x;
  if (tile[1] < 1) return;                                       // the same for the whole cluster
  const int row0 = tile[0], pos = tile[2];
  const int32_t* pt = p.page_tables + static_cast<size_t>(tile[3]) * p.pt_stride;
  const size_t prow = static_cast<size_t>(p.G) * (128 + kV);
  const __nv_bfloat16* pool = static_cast<const __nv_bfloat16*>(p.pool);
  const size_t koff = static_cast<size_t>(g) * 128 + 8 * l16, voff = static_cast<size_t>(p.G) * 128 + static_cast<size_t>(g) * kV + 8 * l16;

  float q[HM][8];
#pragma unroll
  for (int h = 0; h < HM; ++h) {
    const float sc = head_scale(p, g * HM + h);
    const float* src = p.q + ((static_cast<size_t>(row0) * p.H + g * HM + h) * MAPS + map) * D + 8 * r;
    const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
    q[h][0] = a.x * sc; q[h][1] = a.y * sc; q[h][2] = a.z * sc; q[h][3] = a.w * sc;
    q[h][4] = b.x * sc; q[h][5] = b.y * sc; q[h][6] = b.z * sc; q[h][7] = b.w * sc;
  }
  // the scores this lane owns: head oh, keys 8 hf + ok .. + PER - 1 of a group
  const int vi = NV >= R ? r * PER : r / DUP, oh = vi >> 3, ok = vi & 7;
  float m = kNegBig, l = 0.f;                                    // of score head (oh, map), over this warp's keys
  float acc[SH][8];
#pragma unroll
  for (int s = 0; s < SH; ++s)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[s][e] = 0.f;

  const float cap_inv = cap_inverse(p);
  const BlockList bl = visible_blocks(p, pos, pos + 1, kKeys);
  for (int v = rank * kWarps + warp; v < bl.count; v += C * kWarps) {
    const int j0 = bl.block(v) * kKeys, jl = j0 + l16;
    const bool seen = sees(p, pos, jl);                          // lane l16 answers for key l16
    const unsigned long long at = seen ? pool_row(pt, p.page, jl) * prow : 0ull;
    const unsigned mask = __ballot_sync(kAll, seen) & 0xffffu;
    if (mask == 0u) continue;
    uint4 kr[8], vr[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const unsigned long long row = __shfl_sync(kAll, at, 8 * hf + i);
      const bool on = (mask >> (8 * hf + i)) & 1u;
      kr[i] = ld_now(pool + row + koff, on);
      vr[i] = ld_now(pool + row + voff, on);
    }
    float s[NV];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float kf[8] = {bf_lo(kr[i].x), bf_hi(kr[i].x), bf_lo(kr[i].y), bf_hi(kr[i].y), bf_lo(kr[i].z), bf_hi(kr[i].z), bf_lo(kr[i].w), bf_hi(kr[i].w)};
#pragma unroll
      for (int h = 0; h < HM; ++h) {
        float a = 0.f, b = 0.f;
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          a = fmaf(q[h][e], kf[e], a);
          b = fmaf(q[h][e + 1], kf[e + 1], b);
        }
        s[h * 8 + i] = a + b;
      }
    }
    // transposing tree over the R lanes of a map: every step halves the values that a lane carries
    {
      int n = NV;
#pragma unroll
      for (int off = R / 2; off >= 1; off >>= 1) {
        if (n > 1) {
          n >>= 1;
          const bool hi = (r & off) != 0;
#pragma unroll
          for (int i = 0; i < NV / 2; ++i)
            if (i < n) {
              const float send = hi ? s[i] : s[i + n], keep = hi ? s[i + n] : s[i];
              s[i] = keep + __shfl_xor_sync(kAll, send, off);
            }
        } else {
          s[0] += __shfl_xor_sync(kAll, s[0], off);
        }
      }
    }
    const int head = g * HM + oh;
    float mx = m;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int key = 8 * hf + ok + i;
      float z = p.softcap > 0.f ? capped(p, s[i], cap_inv) : s[i];
      if (p.dist_bias) z += dist_bias(p, max(pos - (j0 + key), 0), head);
      s[i] = (mask >> key) & 1u ? z : kNegBig;
      mx = fmaxf(mx, s[i]);
    }
#pragma unroll
    for (int off = DUP; off < R / HM; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(kAll, mx, off));   // the head's other lanes
    mx = fmaxf(mx, __shfl_xor_sync(kAll, mx, 16));                                                 // the other half's keys
    const float alpha = expf(m - mx);
    float ps = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      s[i] = (mask >> (8 * hf + ok + i)) & 1u ? expf(s[i] - mx) : 0.f;
      ps += s[i];
    }
#pragma unroll
    for (int off = DUP; off < R / HM; off <<= 1) ps += __shfl_xor_sync(kAll, ps, off);
    ps += __shfl_xor_sync(kAll, ps, 16);
    l = l * alpha + ps;
    m = mx;
#pragma unroll
    for (int t = 0; t < SH; ++t) {
      const int h = t / MAPS, mp = t % MAPS;
      const float al = __shfl_sync(kAll, alpha, mp * R + (h * 8 / PER) * DUP);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[t][e] *= al;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float vf[8] = {bf_lo(vr[i].x), bf_hi(vr[i].x), bf_lo(vr[i].y), bf_hi(vr[i].y), bf_lo(vr[i].z), bf_hi(vr[i].z), bf_lo(vr[i].w), bf_hi(vr[i].w)};
#pragma unroll
      for (int t = 0; t < SH; ++t) {
        const int h = t / MAPS, mp = t % MAPS, at_ = h * 8 + i;
        const float w = __shfl_sync(kAll, s[at_ % PER], 16 * hf + mp * R + (at_ / PER) * DUP);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[t][e] = fmaf(w, vf[e], acc[t][e]);
      }
    }
  }
  // both halves' keys, then the warp's record
#pragma unroll
  for (int t = 0; t < SH; ++t) {
    float o[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = acc[t][e] + __shfl_xor_sync(kAll, acc[t][e], 16);
    if (hf == 0) {
#pragma unroll
      for (int e = 0; e < 8; e += 2) *reinterpret_cast<float2*>(&rec_s[warp][t][8 * l16 + e]) = make_float2(o[e], o[e + 1]);
    }
  }
  if (hf == 0 && r == (oh * 8 / PER) * DUP) {   // the first lane of a head
    rec_s[warp][oh * MAPS + map][kV] = m;
    rec_s[warp][oh * MAPS + map][kV + 1] = l;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < SH * kV; idx += kThreads) {
    const int t = idx / kV, c = idx - t * kV;
    float mx = kNegBig;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) mx = fmaxf(mx, rec_s[w][t][kV]);
    float a = 0.f, sum = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = expf(rec_s[w][t][kV] - mx);
      a = fmaf(f, rec_s[w][t][c], a);
      sum = fmaf(f, rec_s[w][t][kV + 1], sum);
    }
    cta_s[t][c] = a;
    if (c == 0) {
      cta_s[t][kV] = mx;
      cta_s[t][kV + 1] = sum;
    }
  }
  if (C > 1) cluster_sync_all();
  else __syncthreads();
  // the cluster's records: rank r finishes the model heads r, r + C, ..; 128 threads, one per value column
  __shared__ float ss_s[4];
  for (int h = rank; h < HM; h += C) {
    const int c = threadIdx.x;
    float o[MAPS];
    if (c < kV) {
#pragma unroll
      for (int mp = 0; mp < MAPS; ++mp) {
        const uint32_t own = smem_u32(&cta_s[h * MAPS + mp][0]);
        float pm[8], mx = p.sink ? p.sink[g * HM + h] : kNegBig;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          pm[k] = k < C ? (C > 1 ? ld_dsmem_f32(mapa_u32(own, k) + 4 * kV) : cta_s[h * MAPS + mp][kV]) : kNegBig;
          mx = fmaxf(mx, pm[k]);
        }
        float a = 0.f, den = p.sink ? expf(p.sink[g * HM + h] - mx) : 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < C) {
            const float f = expf(pm[k] - mx);
            const uint32_t rem = C > 1 ? mapa_u32(own, k) : 0u;
            a = fmaf(f, C > 1 ? ld_dsmem_f32(rem + 4 * c) : cta_s[h * MAPS + mp][c], a);
            den = fmaf(f, C > 1 ? ld_dsmem_f32(rem + 4 * kV + 4) : cta_s[h * MAPS + mp][kV + 1], den);
          }
        o[mp] = a / den;
      }
    }
    float out = c < kV ? o[0] : 0.f;
    if (MAPS == 2) {
      out = c < kV ? fmaf(-p.diff_lambda, o[MAPS - 1], o[0]) : 0.f;
      const float ss = warp_sum(out * out);
      __syncthreads();
      if (c < kV && lane == 0) ss_s[warp] = ss;
      __syncthreads();
      out *= p.diff_scale / sqrtf(((ss_s[0] + ss_s[1]) + (ss_s[2] + ss_s[3])) / static_cast<float>(kV) + p.diff_eps);
    }
    if (c < kV) st_any(p.out, p.out_dtype, (static_cast<size_t>(row0) * p.H + g * HM + h) * kV + c, out * out_gate(p, row0, g * HM + h));
  }
  if (C > 1) cluster_sync_all();   // nobody's shared memory goes away under a reader
}

template <int HM, int MAPS>
int launch(const vila_paged_attn_params& p, int C, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.ntiles, p.G, C);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = C;
  cfg.attrs = attr;
  cfg.numAttrs = C > 1 ? 1 : 0;
  VB_CUDA(cudaLaunchKernelEx(&cfg, paged_attn_decode_kernel<HM, MAPS>, p));
  return 0;
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace

// one-row tiles; a key head's row of 128 columns (one map, or two of 64) and 128 value columns are a half-warp's 16-byte pieces
bool paged_attention_decode_takes(const vila_paged_attn_params& p) {
  const int maps = maps_of(p.maps), hm = p.H / p.G;
  return p.max_rows == 1 && p.pool_dtype == VILA_DT_BF16 && p.talk == nullptr && p.vdim == kV && maps * p.dim == 128 &&
         (hm == 1 || hm == 2 || hm == 4 || (hm == 8 && maps == 1)) && p.G <= 65535 && aligned16(p.pool) && aligned16(p.q);
}

int paged_attention_decode(const vila_paged_attn_params& p, cudaStream_t stream) {
  // CTAs per (token, key head): what the caller would deal the keys to, as far as a cluster reaches; never more or fewer by
  // what else is in the launch, so that a row's sums do not depend on it
  const int C = p.nsplit >= 8 ? 8 : p.nsplit >= 4 ? 4 : p.nsplit >= 2 ? 2 : 1, hm = p.H / p.G;
  if (p.maps == 2) {
    if (hm == 1) return launch<1, 2>(p, C, stream);
    if (hm == 2) return launch<2, 2>(p, C, stream);
    return launch<4, 2>(p, C, stream);
  }
  if (hm == 1) return launch<1, 1>(p, C, stream);
  if (hm == 2) return launch<2, 1>(p, C, stream);
  if (hm == 4) return launch<4, 1>(p, C, stream);
  return launch<8, 1>(p, C, stream);
}

}  // namespace vb
