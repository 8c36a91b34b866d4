// vila_paged_attention for prompt portions over a bf16 pool on the tensor cores, in fp32 precision.
//
// The keys and values are bf16 numbers; the queries and the softmax weights are fp32 and stay so: each is cut into
// three bf16 parts (8 + 8 + 8 bits) whose products with a bf16 number are exact, and the three products are summed
// in fp32.  Three bf16 products are cheaper than two tf32 ones and need no range assumptions.
//
// A warp owns 16 rows of one sequence x one score head (mma.sync m16n8k16: rows x 8 keys, then rows x 8 value columns),
// its queries' parts in registers (96 of them at 128 columns) for the whole key loop, scores and sums never leave
// registers.  A CTA serves one key / value head: the score heads that share it x as many consecutive 16-row tiles as make
// four warps.  Blocks of 64 keys come by cp.async into a double buffer of 16-byte pieces swizzled over 8 rows (the
// ldmatrix reads of 8 keys fall into different banks).  CTAs of late positions, which see most keys, start first.
//
// Bound by the tensor pipe: six products where bf16 attention issues two.  Tiled on the CUDA cores the same
// attention ran at 10 TFLOP/s (two shared-memory reads per 16 multiply-adds): MEASURED_ATTN.
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "kernels.h"
#include "dtype_any.cuh"
#include "paged_attn_common.cuh"

namespace vb {
namespace {

constexpr int kBK = 64;      // keys of a block
constexpr int kMaxWarps = 8;

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two fp32 numbers -> three packed pairs of bf16 that add up to them (the last part takes what 16 bits leave)
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16(x, y);
  const float x1 = x - bf_lo(hi), y1 = y - bf_hi(hi);
  mid = pack_bf16(x1, y1);
  lo = pack_bf16(x1 - bf_lo(mid), y1 - bf_hi(mid));
}
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool ok) {
  const uint32_t n = ok ? 16u : 0u;   // 0: zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// D: columns of a map, MAPS: maps of a head, V: value columns.  A key's row in shared memory: MAPS * D columns.
template <int D, int MAPS, int V>
__global__ void __launch_bounds__(32 * kMaxWarps) paged_attn_mma_kernel(const vila_paged_attn_params p, int tiles_per_cta) {
  constexpr int KB = MAPS * D * 2, VB = V * 2;             // bytes of a key's / value's row
  constexpr int kBuf = kBK * (KB + VB);                     // one of two buffers: keys, then values
  extern __shared__ __align__(128) uint8_t sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int rep = p.H / p.G, SH = rep * MAPS, g = blockIdx.y;
  const int tile0 = (gridDim.x - 1 - blockIdx.x) * tiles_per_cta, ntile = min(tiles_per_cta, p.ntiles - tile0);
  const int my_tile = warp / SH, sh = warp - my_tile * SH;  // this warp's tile and score head
  const int h = g * rep + sh / MAPS, map = sh % MAPS;
  const bool active = my_tile < ntile;
  const int* tile = p.tiles + 4 * (tile0 + (active ? my_tile : 0));
  const int row0 = tile[0], n = active ? tile[1] : 0, pos0 = tile[2];
  const int gid = lane >> 2, tig = lane & 3;                // rows gid, gid + 8; columns 2 tig, 2 tig + 1 of an 8-column tile
  const uint32_t sm0 = smem_u32(sm);

  // queries, scaled, in three parts
  uint32_t q[3][D / 16][4];
  {
    const float sc = head_scale(p, h);
#pragma unroll
    for (int k = 0; k < D / 16; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = gid + 8 * (e & 1), c = 16 * k + 8 * (e >> 1) + 2 * tig;
        float2 v = make_float2(0.f, 0.f);
        if (active && i < n)
          v = *reinterpret_cast<const float2*>(p.q + (static_cast<size_t>(row0 + i) * p.H * MAPS + h * MAPS + map) * D + c);
        split3(v.x * sc, v.y * sc, q[0][k][e], q[1][k][e], q[2][k][e]);
        // the parts of an infinite query are itself and zeros
        if (isinf(v.x * sc)) q[1][k][e] &= 0xffff0000u, q[2][k][e] &= 0xffff0000u;
        if (isinf(v.y * sc)) q[1][k][e] &= 0xffffu, q[2][k][e] &= 0xffffu;
      }
  }
  float o[V / 8][4];
#pragma unroll
  for (int t = 0; t < V / 8; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[t][e] = 0.f;
  float m[2], l[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    m[r] = p.sink ? p.sink[h] : kNegBig;
    l[r] = p.sink ? 1.0f : 0.0f;
  }
  // positions of this thread's two rows and what they see: keys lo .. pos, and of those the last `window` or the first keep_first
  int pos[2], lo[2], wlo[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    pos[r] = gid + 8 * r < n ? pos0 + gid + 8 * r : -1;
    lo[r] = first_key(p, max(pos[r], 0));
    wlo[r] = p.window > 0 ? pos[r] - p.window + 1 : 0;
  }
  const int keep = p.window > 0 ? p.keep_first : 0;
  const int row_max = pos0 + n - 1;
  const size_t prow = static_cast<size_t>(p.G) * (MAPS * D + V);   // elements of a pool row
  const __nv_bfloat16* pool = static_cast<const __nv_bfloat16*>(p.pool);
  const size_t koff = static_cast<size_t>(g) * MAPS * D, voff = static_cast<size_t>(p.G) * MAPS * D + static_cast<size_t>(g) * V;

  // the CTA's tiles in runs of one sequence (nearly always a single run)
  for (int run = 0; run < ntile;) {
    const int slot = p.tiles[4 * (tile0 + run) + 3];
    int end = run, first_pos = 0x7fffffff, nkeys = 0;
    for (; end < ntile && p.tiles[4 * (tile0 + end) + 3] == slot; ++end) {
      const int* t = p.tiles + 4 * (tile0 + end);
      first_pos = min(first_pos, t[2]);
      nkeys = max(nkeys, t[2] + t[1]);
    }
    const bool mine = active && my_tile >= run && my_tile < end;
    run = end;
    const int32_t* pt = p.page_tables + static_cast<size_t>(slot) * p.pt_stride;
    const BlockList bl = visible_blocks(p, first_pos, nkeys, kBK);

    // block v to buffer b: a warp takes every nwarps-th key, its lanes the row's pieces
    auto fetch = [&](int v, int b) {
      const int j0 = bl.block(v) * kBK;
      constexpr int kPieces = (KB + VB) / 16;
      const uint32_t base = sm0 + b * kBuf;
      for (int k0 = warp * 32; k0 < kBK; k0 += 32 * nwarps) {       // rows of 32 keys, a lane each
        const int j = j0 + k0 + lane;
        const unsigned long long at = j < nkeys ? pool_row(pt, p.page, j) * prow : 0ull;
        for (int jj = 0; jj < 32; ++jj) {
          const unsigned long long row = __shfl_sync(0xffffffffu, at, jj);
          const int key = k0 + jj;
          const bool ok = j0 + key < nkeys;
          for (int x = lane; x < kPieces; x += 32) {
            const bool is_k = x < KB / 16;
            const int c = is_k ? x : x - KB / 16;
            const uint32_t dst = base + (is_k ? key * KB : kBK * KB + key * VB) + ((c ^ (key & 7)) << 4);
            cp16(dst, pool + row + (is_k ? koff : voff) + c * 8, ok);
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (bl.count > 0) fetch(0, 0);
    for (int v = 0; v < bl.count; ++v) {
      if (v + 1 < bl.count) {
        fetch(v + 1, (v + 1) & 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncthreads();
      const int j0 = bl.block(v) * kBK, j1 = j0 + kBK - 1;
      // does any row of this warp see a key of the block; do all of them see all of its keys
      const bool some = mine && j0 <= row_max && j1 >= first_key(p, pos0) &&
                        (p.window <= 0 || j1 > pos0 - p.window || j0 < keep);
      const bool all = j1 <= pos0 && n == 16 && j0 >= first_key(p, row_max) && (p.window <= 0 || j0 > row_max - p.window || j1 < keep);
      if (some) {
        const uint32_t kb = sm0 + (v & 1) * kBuf, vb = kb + kBK * KB;
        float s[kBK / 8][4];
#pragma unroll
        for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) s[t][e] = 0.f;
        // lanes 0-7 / 8-15 / 16-23 / 24-31 address the matrices (keys 0-7, d 0-7), (same keys, d 8-15), (keys 8-15, ..)
        const int lkey = (lane & 7) + ((lane >> 4) << 3), lc = (lane >> 3) & 1;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
#pragma unroll
          for (int t = 0; t < kBK / 16; ++t) {
            uint32_t b[4];
            ldsm4(kb + (16 * t + lkey) * KB + (((map * D / 8 + 2 * k + lc) ^ (lkey & 7)) << 4), b);
#pragma unroll
            for (int part = 2; part >= 0; --part) {
              mma_bf16(s[2 * t], q[part][k], b[0], b[1]);
              mma_bf16(s[2 * t + 1], q[part][k], b[2], b[3]);
            }
          }
        }
        // cap, bias, mask; the block's maximum per row
        float mn[2] = {m[0], m[1]};
        if (p.softcap > 0.f) {
#pragma unroll
          for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[t][e] = capped(p, s[t][e]);
        }
        if (p.dist_bias) {
#pragma unroll
          for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[t][e] += dist_bias(p, max(pos[e >> 1] - (j0 + 8 * t + 2 * tig + (e & 1)), 0), h);
        }
        if (!all) {
#pragma unroll
          for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int j = j0 + 8 * t + 2 * tig + (e & 1), r = e >> 1;
              if (!(j <= pos[r] && j >= lo[r] && (j >= wlo[r] || j < keep))) s[t][e] = kNegBig;
            }
        }
#pragma unroll
        for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) mn[e >> 1] = fmaxf(mn[e >> 1], s[t][e]);
        float ps[2] = {0.f, 0.f}, alpha[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          mn[r] = quad_max(mn[r]);
          alpha[r] = expf(m[r] - mn[r]);
          m[r] = mn[r];
        }
#pragma unroll
        for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            // a hidden key weighs nothing, also while its row has seen no key at all (maximum still kNegBig)
            s[t][e] = s[t][e] == kNegBig ? 0.f : expf(s[t][e] - mn[e >> 1]);
            ps[e >> 1] += s[t][e];
          }
#pragma unroll
        for (int r = 0; r < 2; ++r) l[r] = l[r] * alpha[r] + quad_sum(ps[r]);
#pragma unroll
        for (int t = 0; t < V / 8; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[t][e] *= alpha[e >> 1];
        // weights (three parts) x values: 16 keys x 16 columns per ldmatrix
        const int vkey = (lane & 7) + (((lane >> 3) & 1) << 3), vc = lane >> 4;
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k) {
          uint32_t a[3][4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float* w = &s[2 * k + (e >> 1)][2 * (e & 1)];
            split3(w[0], w[1], a[0][e], a[1][e], a[2][e]);
          }
#pragma unroll
          for (int t = 0; t < V / 16; ++t) {
            uint32_t b[4];
            ldsm4_t(vb + (16 * k + vkey) * VB + (((2 * t + vc) ^ (vkey & 7)) << 4), b);
#pragma unroll
            for (int part = 2; part >= 0; --part) {
              mma_bf16(o[2 * t], a[part], b[0], b[1]);
              mma_bf16(o[2 * t + 1], a[part], b[2], b[3]);
            }
          }
        }
      }
      __syncthreads();   // everyone has read the buffer that the next block but one overwrites
    }
  }

  if (MAPS == 2) {
    // the second map's rows through shared memory to the warp of the first, which combines, norms and gates them
    float* a2 = reinterpret_cast<float*>(sm) + (warp >> 1) * 16 * V;
    if (active && map == 1) {
#pragma unroll
      for (int t = 0; t < V / 8; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) a2[(gid + 8 * (e >> 1)) * V + 8 * t + 2 * tig + (e & 1)] = o[t][e] * (1.0f / l[e >> 1]);
    }
    __syncthreads();
    if (!active || map == 1) return;
    float ss[2] = {0.f, 0.f};
#pragma unroll
    for (int t = 0; t < V / 8; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = e >> 1;
        o[t][e] = fmaf(-p.diff_lambda, a2[(gid + 8 * r) * V + 8 * t + 2 * tig + (e & 1)], o[t][e] * (1.0f / l[r]));
        ss[r] = fmaf(o[t][e], o[t][e], ss[r]);
      }
#pragma unroll
    for (int r = 0; r < 2; ++r) l[r] = sqrtf(quad_sum(ss[r]) / static_cast<float>(V) + p.diff_eps) / p.diff_scale;
  }
  if (!active) return;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int i = gid + 8 * r;
    if (i >= n) continue;
    const float inv = out_gate(p, row0 + i, h) / l[r];
    const size_t ob = (static_cast<size_t>(row0 + i) * p.H + h) * V + 2 * tig;
#pragma unroll
    for (int t = 0; t < V / 8; ++t) {
      const float x = o[t][2 * r] * inv, y = o[t][2 * r + 1] * inv;
      if (p.out_dtype == VILA_DT_F32) *reinterpret_cast<float2*>(static_cast<float*>(p.out) + ob + 8 * t) = make_float2(x, y);
      else *reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(p.out) + ob + 8 * t) = pack_bf16(x, y);
    }
  }
}

template <int D, int MAPS, int V>
int launch(const vila_paged_attn_params& p, cudaStream_t stream) {
  constexpr int smem = 2 * kBK * (MAPS * D + V) * 2;
  const int SH = p.H / p.G * MAPS, tpc = SH >= 4 ? 1 : 4 / SH;   // four warps, or one tile of all the heads
  static PerDeviceOnce once;
  if (once.first())
    VB_CUDA(cudaFuncSetAttribute(paged_attn_mma_kernel<D, MAPS, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  VB_CUDA(launch_serial(paged_attn_mma_kernel<D, MAPS, V>, dim3((p.ntiles + tpc - 1) / tpc, p.G), dim3(32 * SH * tpc), smem, stream, p, tpc));
  return 0;
}

bool aligned(const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; }

}  // namespace

// Tiles of up to 16 rows (m16), head sizes that fit the registers, rows on 16-byte boundaries, all heads of a CTA in 8 warps.
bool paged_attention_mma_takes(const vila_paged_attn_params& p) {
  const int maps = maps_of(p.maps);
  return p.max_rows > 1 && p.nsplit == 1 && p.pool_dtype == VILA_DT_BF16 && p.talk == nullptr && p.H / p.G * maps <= kMaxWarps &&
         ((maps == 1 && p.dim == 128 && p.vdim == 128) || (maps == 2 && p.dim == 64 && p.vdim == 128) ||
          (maps == 1 && p.dim == 64 && p.vdim == 64)) &&
         p.G <= 65535 && aligned(p.pool, 16) && aligned(p.q, 8) && aligned(p.out, 8);
}

int paged_attention_mma(const vila_paged_attn_params& p, cudaStream_t stream) {
  if (p.maps == 2) return launch<64, 2, 128>(p, stream);
  if (p.dim == 64) return launch<64, 1, 64>(p, stream);
  return launch<128, 1, 128>(p, stream);
}

}  // namespace vb
