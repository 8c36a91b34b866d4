// vila_paged_attention of prompt portions whose heads are mixed (talk), over a bf16 pool, on the tensor cores in fp32 precision.
//
// A mixed score needs the scores of all H heads of its (query, key) pair, so a CTA holds eight rows of one sequence and all
// the heads, a warp one head (two from 17 heads on).  The rows are the n of mma.sync m16n8k16: scores^T = K q^T, 16 keys x 8
// rows, and O^T = V^T w^T, 16 columns x 8 rows, so that a head's sums are 32 registers and 32 heads of 128 columns fit a CTA.
// Between the two products a block of 16 keys goes through shared memory: every warp leaves its head's scores (weights, where
// those are mixed) and takes its row of the mixing matrix times all of them, in fp32 multiply-adds; two buffers, one barrier
// a block.
//
// Keys and values come from global memory in fragment order, without shared memory: the order of a contraction's terms and of
// an output's columns is free, so that a lane's 16 bytes of a key's row are two steps' operands, and its 16 bytes of four
// values' rows are, two halves at a time, those of four column tiles.  A stage of 64 columns is asked for one stage ahead.
//
// Queries (fp32, scaled) and weights are cut into three bf16 parts as in paged_attn_mma.cu, and what the tensor core sums
// goes into fresh accumulators: a score's first parts (8 truncating additions at 128 columns) apart from the others, a block's
// 16 products of a value column; they join by rounded additions.  A tile whose rows come out infinite or NaN is computed again
// key by key: zero parts meet an infinite number where the number itself does not.
//
// Bound by latency: a block of 16 heads takes 9100 clocks, of which the tensor pipe works 1540 and shared memory's 2000; the
// loads of a stage and the barrier of a block are what the 16 warps wait for.  Two heads of 128 columns a warp (17 heads and more) do
// not fit its 128 registers: 150 - 200 bytes are stored and 360 - 500 loaded a block besides.
// The tiles on the CUDA cores (paged_attn_tile4_kernel) hold whole key blocks of all heads in shared memory, 32 keys of 4
// heads, 4 of 32.  Scores mixed / weights mixed there and here: 2048 causal rows of 16 heads over 4 1923 / 2115 -> 532 / 620 us,
// 1024 rows on 500 keys of 32 heads over 32 21700 / 24500 -> 1007 / 963, 40 rows on 300 keys 163 / 240 -> 106 / 139.
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "kernels.h"
#include "dtype_any.cuh"
#include "paged_attn_common.cuh"
#include "mma_bf16.cuh"

namespace vb {
namespace {

constexpr int kBK = 16;       // keys of a block
constexpr int kRows = 8;

__device__ __forceinline__ uint4 ld_pool(const __nv_bfloat16* p) {   // stays where it is written, a stage ahead of its use
  uint4 v;
  asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t word(const uint4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }

template <int D>
__host__ __device__ constexpr int q_stride() { return D + 4; }   // floats: eight rows' 16-byte pieces in different banks
__host__ __device__ __forceinline__ int talk_stride(int H) { return (H + 3) & ~3; }
template <int D>
size_t smem_bytes(int H) { return sizeof(float) * (static_cast<size_t>(H) * (kRows * q_stride<D>() + 2 * kBK * kRows + talk_stride(H)) + 4); }

// The tile's rows again, key by key in fp32 multiply-adds.  xs: H floats of shared memory.
template <int D, int HW, bool AFTER>
__device__ __noinline__ void tile_again(const vila_paged_attn_params& p, const float* Qs, const float* talk, float* xs, const int32_t* pt,
                                        int row0, int n, int pos0) {
  constexpr int C = D / 32;
  const int H = p.H, lane = threadIdx.x & 31, h0 = (threadIdx.x >> 5) * HW, rep = H / p.G;
  const size_t prow = static_cast<size_t>(p.G) * 2 * D;
  const __nv_bfloat16* pool = static_cast<const __nv_bfloat16*>(p.pool);
  for (int i = 0; i < n; ++i) {
    const int pos = pos0 + i;
    float m[HW], l[HW], o[HW][C];
#pragma unroll
    for (int u = 0; u < HW; ++u) {
      const bool sink = !AFTER && p.sink != nullptr && h0 + u < H;
      m[u] = sink ? p.sink[h0 + u] : kNegBig;
      l[u] = sink ? 1.0f : 0.0f;
#pragma unroll
      for (int c = 0; c < C; ++c) o[u][c] = 0.f;
    }
    for (int pass = AFTER ? 0 : 1; pass < 2; ++pass)
      for (int j = 0; j <= pos; ++j) {
        if (!sees(p, pos, j)) continue;
        const __nv_bfloat16* at = pool + pool_row(pt, p.page, j) * prow;
#pragma unroll
        for (int u = 0; u < HW; ++u) {
          const int h = h0 + u;
          if (h >= H) continue;
          float s = 0.f;
#pragma unroll
          for (int c = 0; c < C; ++c)
            s = fmaf(Qs[(h * kRows + i) * q_stride<D>() + C * lane + c], __bfloat162float(at[static_cast<size_t>(h / rep) * D + C * lane + c]), s);
          s = capped(p, warp_sum(s));
          if (AFTER && pass == 0) {
            const float mn = fmaxf(m[u], s);
            l[u] = fmaf(l[u], expf(m[u] - mn), expf(s - mn));
            m[u] = mn;
          } else if (lane == 0) {
            xs[h] = AFTER ? expf(s - m[u]) / l[u] : s;
          }
        }
        if (pass == 0) continue;
        __syncthreads();
#pragma unroll
        for (int u = 0; u < HW; ++u) {
          const int h = h0 + u;
          if (h >= H) continue;
          const float s = warp_sum(lane < H ? talk[h * talk_stride(H) + lane] * xs[lane] : 0.f);
          float w = s, alpha = 1.f;
          if (!AFTER) {
            const float z = p.dist_bias ? s + dist_bias(p, pos - j, h) : s, mn = fmaxf(m[u], z);
            w = expf(z - mn);
            alpha = expf(m[u] - mn);
            l[u] = fmaf(l[u], alpha, w);
            m[u] = mn;
          }
#pragma unroll
          for (int c = 0; c < C; ++c)
            o[u][c] = fmaf(w, __bfloat162float(at[static_cast<size_t>(p.G + h / rep) * D + C * lane + c]), o[u][c] * alpha);
        }
        __syncthreads();
      }
#pragma unroll
    for (int u = 0; u < HW; ++u) {
      const int h = h0 + u;
      if (h >= H) continue;
      const float inv = AFTER ? out_gate(p, row0 + i, h) : out_gate(p, row0 + i, h) / l[u];
#pragma unroll
      for (int c = 0; c < C; ++c) st_any(p.out, p.out_dtype, (static_cast<size_t>(row0 + i) * H + h) * D + C * lane + c, o[u][c] * inv);
    }
  }
}

// D: columns of a key and of a value, HW: heads of a warp, AFTER: the weights are mixed, not the scores
template <int D, int HW, bool AFTER>
__global__ void __launch_bounds__(512, 1) paged_attn_mix_kernel(const __grid_constant__ vila_paged_attn_params p) {
  constexpr int QS = q_stride<D>(), NS = D / 64;             // stages of 64 columns
  extern __shared__ __align__(16) float sm[];
  const int H = p.H, rep = H / p.G, TS = talk_stride(H);
  float* Qs = sm;                                            // [H][8][QS]
  float* X = Qs + H * kRows * QS;                            // two buffers [H][8 rows][4 lanes: keys 2 t, 2 t + 1, 2 t + 8, 2 t + 9]
  float* talk = X + 2 * H * kRows * kBK;                     // [H][TS]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const int at = static_cast<int>(gridDim.x) - 1 - blockIdx.x, parts = (p.max_rows + kRows - 1) / kRows;   // late rows, which see most keys, first
  const int* tile = p.tiles + 4 * (at / parts);
  const int i0 = at % parts * kRows;
  if (i0 >= tile[1]) return;
  const int row0 = tile[0] + i0, n = min(kRows, tile[1] - i0), pos0 = tile[2] + i0;
  const int32_t* pt = p.page_tables + static_cast<size_t>(tile[3]) * p.pt_stride;
  const int h0 = warp * HW;
  const bool softcap = p.softcap > 0.f;
  const float cap_inv = cap_inverse(p);

  for (int x = tid; x < H * kRows * (D / 4); x += blockDim.x) {
    const int c = x % (D / 4), r = x / (D / 4), h = r / kRows, i = r - h * kRows;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n) v = *reinterpret_cast<const float4*>(p.q + (static_cast<size_t>(row0 + i) * H + h) * D + 4 * c);
    const float sc = head_scale(p, h);
    *reinterpret_cast<float4*>(Qs + r * QS + 4 * c) = make_float4(v.x * sc, v.y * sc, v.z * sc, v.w * sc);
  }
  for (int x = tid; x < H * TS; x += blockDim.x) talk[x] = x % TS < H ? p.talk[(x / TS) * H + x % TS] : 0.f;

  float o[HW][4 * NS][4];
#pragma unroll
  for (int u = 0; u < HW; ++u)
#pragma unroll
    for (int t = 0; t < 4 * NS; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[u][t][e] = 0.f;
  // scores mixed: m and l of row gid.  Weights mixed: of rows 2 tig and 2 tig + 1 (the layout of the scores)
  float m[HW][2], l[HW][2];
#pragma unroll
  for (int u = 0; u < HW; ++u) {
    const bool sink = !AFTER && p.sink != nullptr && h0 + u < H;
    const float z = sink ? p.sink[h0 + u] : kNegBig;
    const bool none = !sink || z < kNegBig;                  // a sink below every score (-inf: switched off) weighs nothing
    m[u][0] = m[u][1] = none ? kNegBig : z;
    l[u][0] = l[u][1] = none ? 0.f : ex2(fmaf(z, kLog2e, -log2_units(z)));
  }
  // what a row sees: keys lo .. pos, and of those the last `window` or the first keep_first
  struct Sight {
    int pos, lo, wlo;
  };
  auto sight = [&](int i) {
    const int pos = i < n ? pos0 + i : -1;
    return Sight{pos, first_key(p, max(pos, 0)), p.window > 0 ? pos - p.window + 1 : 0};
  };
  const int keep = p.window > 0 ? p.keep_first : 0;
  auto seen = [&](const Sight& s, int j) { return j <= s.pos && j >= s.lo && (j >= s.wlo || j < keep); };
  const Sight sg = sight(gid), s2[2] = {sight(2 * tig), sight(2 * tig + 1)};
  const int nkeys = pos0 + n;
  const BlockList bl = visible_blocks(p, pos0, nkeys, kBK);
  const size_t prow = static_cast<size_t>(p.G) * 2 * D;
  const __nv_bfloat16* pool = static_cast<const __nv_bfloat16*>(p.pool);
  __syncthreads();

  auto pool_rows = [&](int v) {   // of block v's keys, one to a lane (twice); behind the last key that one
    return v < bl.count ? static_cast<int>(pool_row(pt, p.page, min(bl.block(v) * kBK + (lane & 15), nkeys - 1))) : 0;
  };
  auto key_at = [&](int rows, int k, int h) {
    return pool + static_cast<size_t>(static_cast<unsigned>(__shfl_sync(0xffffffffu, rows, k))) * prow + static_cast<size_t>(h / rep) * D;
  };
  uint4 in[4];   // the stage that comes next
  auto load_k = [&](int rows, int h, int st) {
    const __nv_bfloat16 *a = key_at(rows, gid, h) + 64 * st + 8 * tig, *b = key_at(rows, gid + 8, h) + 64 * st + 8 * tig;
    in[0] = ld_pool(a);
    in[1] = ld_pool(b);
    in[2] = ld_pool(a + 32);
    in[3] = ld_pool(b + 32);
  };
  auto load_v = [&](int rows, int h, int st) {
    const size_t off = static_cast<size_t>(p.G) * D + 64 * st + 8 * gid;
    in[0] = ld_pool(key_at(rows, 2 * tig, h) + off);
    in[1] = ld_pool(key_at(rows, 2 * tig + 1, h) + off);
    in[2] = ld_pool(key_at(rows, 2 * tig + 8, h) + off);
    in[3] = ld_pool(key_at(rows, 2 * tig + 9, h) + off);
  };
  auto head = [&](int u) { return min(h0 + u, H - 1); };     // a warp without a head computes the last one's and leaves nothing
  // scores of 16 keys x 8 rows: keys gid (e < 2) and gid + 8, rows 2 tig + (e & 1).  `next` asks for the stage behind them.
  auto scores = [&](int rows, int u, float (&s)[4], auto next) {
    float lo[4];
    const float* q = Qs + (head(u) * kRows + gid) * QS + 8 * tig;
#pragma unroll
    for (int st = 0; st < NS; ++st) {
      const uint4 k[4] = {in[0], in[1], in[2], in[3]};
      if (st + 1 < NS) load_k(rows, head(u), st + 1);
      else next();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float4 q0 = *reinterpret_cast<const float4*>(q + 64 * st + 32 * c), q1 = *reinterpret_cast<const float4*>(q + 64 * st + 32 * c + 4);
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          const float4 qv = w ? q1 : q0;
          uint32_t b0[3], b1[3];
          split3(qv.x, qv.y, b0[0], b0[1], b0[2]);
          split3(qv.z, qv.w, b1[0], b1[1], b1[2]);
          const uint32_t a[4] = {word(k[2 * c], 2 * w), word(k[2 * c + 1], 2 * w), word(k[2 * c], 2 * w + 1), word(k[2 * c + 1], 2 * w + 1)};
          if (st + c + w == 0) {
            mma_bf16_first(lo, a, b0[2], b1[2]);
            mma_bf16_first(s, a, b0[0], b1[0]);
          } else {
            mma_bf16(lo, a, b0[2], b1[2]);
            mma_bf16(s, a, b0[0], b1[0]);
          }
          mma_bf16(lo, a, b0[1], b1[1]);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      s[e] += lo[e];
      if (softcap) s[e] = capped(p, s[e], cap_inv);
    }
  };

  for (int pass = AFTER ? 0 : 1; pass < 2; ++pass) {
    const bool stats = AFTER && pass == 0;
    if (AFTER && !stats) {
#pragma unroll
      for (int u = 0; u < HW; ++u)
#pragma unroll
        for (int r = 0; r < 2; ++r) l[u][r] = l[u][r] > 0.f ? 1.0f / l[u][r] : 0.f;
    }
    int rows = pool_rows(0);
    if (bl.count > 0) load_k(rows, head(0), 0);
    for (int v = 0; v < bl.count; ++v) {
      const int j0 = bl.block(v) * kBK, rows_next = pool_rows(v + 1);
      float* xb = X + (v & 1) * H * kRows * kBK;
#pragma unroll
      for (int u = 0; u < HW; ++u) {
        float s[4];
        scores(rows, u, s, [&]() {
          if (u + 1 < HW) load_k(rows, head(u + 1), 0);
          else if (!stats) load_v(rows, head(0), 0);
          else if (v + 1 < bl.count) load_k(rows_next, head(0), 0);
        });
        if (AFTER) {
          bool ok[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) ok[e] = seen(s2[e & 1], j0 + gid + 8 * (e >> 1));
          if (stats) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              float mn = fmaxf(ok[r] ? s[r] : kNegBig, ok[r + 2] ? s[r + 2] : kNegBig);
#pragma unroll
              for (int x = 4; x < 32; x <<= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, x));
              mn = fmaxf(mn, m[u][r]);
              const float ml = log2_units(mn);
              float ps = (ok[r] ? ex2(fmaf(s[r], kLog2e, -ml)) : 0.f) + (ok[r + 2] ? ex2(fmaf(s[r + 2], kLog2e, -ml)) : 0.f);
#pragma unroll
              for (int x = 4; x < 32; x <<= 1) ps += __shfl_xor_sync(0xffffffffu, ps, x);
              l[u][r] = l[u][r] * ex2(__fsub_rn(log2_units(m[u][r]), ml)) + ps;
              m[u][r] = mn;
            }
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) s[e] = ok[e] ? ex2(fmaf(s[e], kLog2e, -log2_units(m[u][e & 1]))) * l[u][e & 1] : 0.f;
          }
        }
        if (!stats && h0 + u < H) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            xb[((h0 + u) * kRows + 2 * tig + (e & 1)) * kBK + (gid >> 1) * 4 + (gid & 1) + (e & 2)] = s[e];
        }
      }
      if (!stats) {
        __syncthreads();
#pragma unroll
        for (int u = 0; u < HW; ++u) {
          // this head's row of the mixing matrix x all heads: row gid, keys 2 tig, 2 tig + 1, 2 tig + 8, 2 tig + 9
          float z[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f};
          const float* tk = talk + head(u) * TS;
          const float* x = xb + lane * 4;
          int g = 0;
          for (; g + 4 <= H; g += 4) {
            const float4 t4 = *reinterpret_cast<const float4*>(tk + g);
            const float t[4] = {t4.x, t4.y, t4.z, t4.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float4 xv = *reinterpret_cast<const float4*>(x + (g + k) * kRows * kBK);
              float(&d)[4] = k & 1 ? y : z;
              d[0] = fmaf(t[k], xv.x, d[0]);
              d[1] = fmaf(t[k], xv.y, d[1]);
              d[2] = fmaf(t[k], xv.z, d[2]);
              d[3] = fmaf(t[k], xv.w, d[3]);
            }
          }
          for (; g < H; ++g) {
            const float4 xv = *reinterpret_cast<const float4*>(x + g * kRows * kBK);
            z[0] = fmaf(tk[g], xv.x, z[0]);
            z[1] = fmaf(tk[g], xv.y, z[1]);
            z[2] = fmaf(tk[g], xv.z, z[2]);
            z[3] = fmaf(tk[g], xv.w, z[3]);
          }
          float w[4], al[2] = {1.f, 1.f};
          if (AFTER) {
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = z[e] + y[e];
          } else {
            bool ok[4];
            float mn = m[u][0];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int j = j0 + 2 * tig + (e & 1) + 4 * (e & 2);
              ok[e] = seen(sg, j);
              w[e] = z[e] + y[e];
              if (p.dist_bias) w[e] += dist_bias(p, max(sg.pos - j, 0), head(u));
              mn = fmaxf(mn, ok[e] ? w[e] : kNegBig);
            }
            mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
            mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
            const float ml = log2_units(mn), alpha = ex2(__fsub_rn(log2_units(m[u][0]), ml));
            float ps = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              w[e] = ok[e] ? ex2(fmaf(w[e], kLog2e, -ml)) : 0.f;
              ps += w[e];
            }
            ps += __shfl_xor_sync(0xffffffffu, ps, 1);
            ps += __shfl_xor_sync(0xffffffffu, ps, 2);
            l[u][0] = l[u][0] * alpha + ps;
            m[u][0] = mn;
            al[0] = __shfl_sync(0xffffffffu, alpha, 8 * tig);        // rows 2 tig, 2 tig + 1
            al[1] = __shfl_sync(0xffffffffu, alpha, 8 * tig + 4);
          }
          uint32_t b0[3], b1[3];
          split3(w[0], w[1], b0[0], b0[1], b0[2]);
          split3(w[2], w[3], b1[0], b1[1], b1[2]);
#pragma unroll
          for (int st = 0; st < NS; ++st) {
            const uint4 vv[4] = {in[0], in[1], in[2], in[3]};
            if (st + 1 < NS) load_v(rows, head(u), st + 1);
            else if (u + 1 < HW) load_v(rows, head(u + 1), 0);
            else if (v + 1 < bl.count) load_k(rows_next, head(0), 0);
#pragma unroll
            for (int t = 0; t < 4; ++t) {   // columns 64 st + 8 gid + 2 t (e < 2) and + 1, rows 2 tig + (e & 1)
              const uint32_t x0 = word(vv[0], t), x1 = word(vv[1], t), x2 = word(vv[2], t), x3 = word(vv[3], t);
              const uint32_t a[4] = {__byte_perm(x0, x1, 0x5410), __byte_perm(x0, x1, 0x7632), __byte_perm(x2, x3, 0x5410),
                                     __byte_perm(x2, x3, 0x7632)};
              float c[4];
              mma_bf16_first(c, a, b0[2], b1[2]);
              mma_bf16(c, a, b0[1], b1[1]);
              mma_bf16(c, a, b0[0], b1[0]);
              float(&d)[4] = o[u][4 * st + t];
#pragma unroll
              for (int e = 0; e < 4; ++e) d[e] = AFTER ? d[e] + c[e] : fmaf(d[e], al[e & 1], c[e]);
            }
          }
        }
      }
      rows = rows_next;
    }
  }

  bool odd = false;
#pragma unroll
  for (int u = 0; u < HW; ++u) {
    float z = AFTER ? 0.f : l[u][0] * 0.f;
#pragma unroll
    for (int t = 0; t < 4 * NS; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) z = fmaf(o[u][t][e], 0.f, z);
    odd |= !(z == 0.f);
  }
  if (__syncthreads_or(odd)) {
    tile_again<D, HW, AFTER>(p, Qs, talk, X, pt, row0, n, pos0);
    return;
  }
#pragma unroll
  for (int u = 0; u < HW; ++u) {
    const int h = h0 + u;
    float lr[2] = {1.f, 1.f};
    if (!AFTER) {
      lr[0] = __shfl_sync(0xffffffffu, l[u][0], 8 * tig);
      lr[1] = __shfl_sync(0xffffffffu, l[u][0], 8 * tig + 4);
    }
    if (h >= H) continue;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int i = 2 * tig + r;
      if (i >= n) continue;
      const float inv = out_gate(p, row0 + i, h) / lr[r];
#pragma unroll
      for (int st = 0; st < NS; ++st) {
        const size_t at = (static_cast<size_t>(row0 + i) * H + h) * D + 64 * st + 8 * gid;
        float y[8];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          y[2 * t] = o[u][4 * st + t][r] * inv;
          y[2 * t + 1] = o[u][4 * st + t][2 + r] * inv;
        }
        if (p.out_dtype == VILA_DT_F32) {
          float* d = static_cast<float*>(p.out) + at;
          *reinterpret_cast<float4*>(d) = make_float4(y[0], y[1], y[2], y[3]);
          *reinterpret_cast<float4*>(d + 4) = make_float4(y[4], y[5], y[6], y[7]);
        } else {
          *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.out) + at) =
              make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
        }
      }
    }
  }
}

template <int D, int HW, bool AFTER>
int launch(const vila_paged_attn_params& p, cudaStream_t stream) {
  auto kernel = paged_attn_mix_kernel<D, HW, AFTER>;
  static PerDeviceOnce once;
  if (once.first()) VB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_bytes<D>(16 * HW))));
  const long ctas = static_cast<long>(p.ntiles) * ((p.max_rows + kRows - 1) / kRows);
  VB_CHECK(ctas < (1L << 31), "paged_attention: too many tiles");
  VB_CUDA(launch_serial(kernel, dim3(static_cast<unsigned>(ctas)), dim3(32 * ((p.H + HW - 1) / HW)), smem_bytes<D>(p.H), stream, p));
  return 0;
}
template <int D>
int launch_form(const vila_paged_attn_params& p, cudaStream_t stream) {
  if (p.H <= 16) return p.talk_after ? launch<D, 1, true>(p, stream) : launch<D, 1, false>(p, stream);
  return p.talk_after ? launch<D, 2, true>(p, stream) : launch<D, 2, false>(p, stream);
}

bool aligned(const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; }

}  // namespace

// Mixed heads over a bf16 pool: 64 or 128 columns of key and value, up to 32 heads, rows on 16-byte boundaries.
bool paged_attention_mix_takes(const vila_paged_attn_params& p) {
  return p.talk != nullptr && p.max_rows > 1 && p.nsplit == 1 && maps_of(p.maps) == 1 && p.pool_dtype == VILA_DT_BF16 && p.H <= 32 &&
         (p.dim == 64 || p.dim == 128) && p.vdim == p.dim && aligned(p.pool, 16) && aligned(p.q, 16) && aligned(p.out, 16);
}

int paged_attention_mix(const vila_paged_attn_params& p, cudaStream_t stream) {
  return p.dim == 64 ? launch_form<64>(p, stream) : launch_form<128>(p, stream);
}

}  // namespace vb
