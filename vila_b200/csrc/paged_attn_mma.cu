// vila_paged_attention for prompt portions over a bf16 pool on the tensor cores, in fp32 precision: two maps, 64 columns, and 128
// columns off the 16-byte boundaries of paged_attn_tc.cu.
//
// The keys and values are bf16 numbers; the queries and the softmax weights are fp32 and stay so: each is cut into
// three bf16 parts (8 + 8 + 8 bits) whose products with a bf16 number are exact, and the three products are summed
// in fp32.  Three bf16 products are cheaper than two tf32 ones and need no range assumptions.  Only an infinite key or
// value cannot be taken so (it meets the zero parts of a number that one part holds): rows that come out infinite or NaN
// are computed again key by key.
//
// A warp owns 16 rows of one sequence x one score head (mma.sync m16n8k16: rows x 8 keys, then rows x 8 value columns);
// scores and sums never leave its registers, the queries' parts lie in shared memory in fragment order.  A CTA serves
// one key / value head: the score heads that share it x as many consecutive 16-row tiles as make four warps, twice: one
// set of warps takes the even blocks of 64 keys, the other the odd ones (by position, so that a row's sums do not depend
// on its tile), and the two are merged at the end.  The sets run freely against each other, one's softmax under the
// other's products, and the longest chain of blocks is half as long.  Blocks come by cp.async into double buffers of
// 16-byte pieces swizzled over 8 rows (the ldmatrix reads of 8 keys fall into different banks).  CTAs of late
// positions, which see most keys, start first, those of all key heads.
//
// Bound by the tensor pipe (mma.sync: 1024 multiply-adds per clock and SM measured), six products where bf16 attention
// issues two.  Tiled on the CUDA cores the same attention ran at 10 TFLOP/s (two shared-memory reads per 16
// multiply-adds).  2048 causal rows, 16 heads over 4, 128 columns: 1560 us there with capped scores, 193 here (186 without the
// cap; 251 with tanhf for every score).
//
// The tensor core truncates as it accumulates, and the truncations of a sum all go one way: with running sums over all keys
// the rows were 2.8e-6 off at 2048 keys and 2.6e-5 at 16384, where fp32 multiply-adds are 8e-7 and 2.3e-6 off.  So a block's
// products go into fresh sums, the parts in ascending size (four additions of full size for 64 keys), and join the row's
// sums by rounded additions; the first parts of a score's products (eight additions) are summed apart from the others.
// Error 7e-8 at 64 keys, 1.4e-7 at 2048, 2.6e-7 at 16384; the running sums took 219 and 153 us.
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "kernels.h"
#include "dtype_any.cuh"
#include "paged_attn_common.cuh"
#include "mma_bf16.cuh"

namespace vb {
namespace {

constexpr int kBK = 64;      // keys of a block
constexpr int kMaxWarps = 8;

__device__ __forceinline__ float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// D: columns of a map, MAPS: maps of a head, V: value columns, SETS: sets of warps that share the key blocks.  A key's row
// in shared memory has MAPS * D columns.
// exp(s - m) is taken as 2^(s log2 e - m log2 e) with one fused multiply-add: the rounded m log2 e is common to a row's
// weights and cancels in their quotient, which leaves the rounding of the difference, as in exp(s - m).
// CAP: with capped scores (a kernel of its own: the others were 4 % slower for its instructions).
template <int D, int MAPS, int V, int SETS, bool CAP>
__global__ void __launch_bounds__(32 * (SETS == 2 ? 8 : kMaxWarps), 1)
paged_attn_mma_kernel(const __grid_constant__ vila_paged_attn_params p, int tiles_per_cta) {
  constexpr int KB = MAPS * D * 2, VB = V * 2;             // bytes of a key's / value's row
  constexpr int kBuf = kBK * (KB + VB);                     // one of a set's two buffers: keys, then values
  constexpr int kQ = 3 * (D / 16) * 512;                    // bytes of a warp's query parts
  extern __shared__ __align__(128) uint8_t sm[];
  const int lane = threadIdx.x & 31, W = (blockDim.x >> 5) / SETS;   // warps of a set
  const int set = (threadIdx.x >> 5) / W, warp = (threadIdx.x >> 5) - set * W;
  const int rep = p.H / p.G, SH = rep * MAPS, g = blockIdx.x % p.G;
  const int tile0 = (gridDim.x / p.G - 1 - blockIdx.x / p.G) * tiles_per_cta, ntile = min(tiles_per_cta, p.ntiles - tile0);
  const int my_tile = warp / SH, sh = warp - my_tile * SH;  // this warp's tile and score head
  const int h = g * rep + sh / MAPS, map = sh % MAPS;
  const bool active = my_tile < ntile;
  const int* tile = p.tiles + 4 * (tile0 + (active ? my_tile : 0));
  const int row0 = tile[0], n = active ? tile[1] : 0, pos0 = tile[2];
  const int gid = lane >> 2, tig = lane & 3;                // rows gid, gid + 8; columns 2 tig, 2 tig + 1 of an 8-column tile
  uint4* q_s = reinterpret_cast<uint4*>(sm + warp * kQ) + lane;      // [part][D / 16] fragments, 32 lanes apart
  uint8_t* buf = sm + W * kQ + set * 2 * kBuf;
  const uint32_t buf0 = smem_u32(buf);

  // queries, scaled, in three parts (the sets share them: set s brings every SETS-th fragment)
  {
    const float sc = head_scale(p, h);
#pragma unroll
    for (int k0 = 0; k0 < D / 16; k0 += SETS) {
      const int k = k0 + set;
      uint32_t q[3][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = gid + 8 * (e & 1), c = 16 * k + 8 * (e >> 1) + 2 * tig;
        float2 v = make_float2(0.f, 0.f);
        if (active && i < n)
          v = *reinterpret_cast<const float2*>(p.q + (static_cast<size_t>(row0 + i) * p.H * MAPS + h * MAPS + map) * D + c);
        split3(v.x * sc, v.y * sc, q[0][e], q[1][e], q[2][e]);
        // the parts of an infinite query are itself and zeros
        if (isinf(v.x * sc)) q[1][e] &= 0xffff0000u, q[2][e] &= 0xffff0000u;
        if (isinf(v.y * sc)) q[1][e] &= 0xffffu, q[2][e] &= 0xffffu;
      }
#pragma unroll
      for (int part = 0; part < 3; ++part) q_s[(part * (D / 16) + k) * 32] = make_uint4(q[part][0], q[part][1], q[part][2], q[part][3]);
    }
  }
  float o[V / 8][4];
#pragma unroll
  for (int t = 0; t < V / 8; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[t][e] = 0.f;
  float m[2], l[2];
  const bool sink = p.sink != nullptr && set == 0;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    // a sink below every score (-inf: switched off) weighs nothing
    const float z = sink ? p.sink[h] : kNegBig;
    const bool none = !sink || z < kNegBig;
    m[r] = none ? kNegBig : z;
    l[r] = none ? 0.0f : ex2(fmaf(z, kLog2e, -log2_units(z)));
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
  const float cap_inv = cap_inverse(p);
  const int row_max = pos0 + n - 1, lo_min = first_key(p, pos0), lo_max = first_key(p, max(row_max, 0));
  const size_t prow = static_cast<size_t>(p.G) * (MAPS * D + V);   // elements of a pool row
  const __nv_bfloat16* pool = static_cast<const __nv_bfloat16*>(p.pool);
  const size_t koff = static_cast<size_t>(g) * MAPS * D, voff = static_cast<size_t>(p.G) * MAPS * D + static_cast<size_t>(g) * V;
  __syncthreads();   // queries

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
    auto next_block = [&](int v) {   // the first of this set's blocks from v on
      while (SETS == 2 && v < bl.count && (bl.block(v) & 1) != set) ++v;
      return v;
    };
    // block v to buffer b: a warp takes every W-th run of 32 keys, its lanes the rows' pieces
    auto fetch = [&](int v, int b) {
      const int j0 = bl.block(v) * kBK;
      constexpr int kPieces = (KB + VB) / 16;
      const uint32_t base = buf0 + b * kBuf;
      for (int k0 = warp * 16; k0 < kBK; k0 += 16 * W) {             // rows of 16 keys, a lane each
        const int j = j0 + k0 + (lane & 15);
        const unsigned long long at = j < nkeys ? pool_row(pt, p.page, j) * prow : 0ull;
#pragma unroll 4
        for (int jj = 0; jj < 16; ++jj) {
          const unsigned long long row = __shfl_sync(0xffffffffu, at, jj);
          const int key = k0 + jj;
          const bool ok = j0 + key < nkeys;
#pragma unroll
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
    auto set_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + set), "r"(32 * W) : "memory"); };
    int v = next_block(0), b = 0;
    if (v < bl.count) fetch(v, 0);
    while (v < bl.count) {
      const int after = next_block(v + 1);
      if (after < bl.count) {
        fetch(after, b ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      set_sync();
      const int j0 = bl.block(v) * kBK, j1 = j0 + kBK - 1;
      // does any row of this warp see a key of the block; do all of them see all of its keys
      const bool some = mine && j0 <= row_max && j1 >= lo_min && (p.window <= 0 || j1 > pos0 - p.window || j0 < keep);
      const bool all = j1 <= pos0 && n == 16 && j0 >= lo_max && (p.window <= 0 || j0 > row_max - p.window || j1 < keep);
      if (some) {
        const uint32_t kb = buf0 + b * kBuf, vb = kb + kBK * KB;
        float s[kBK / 8][4];
        // lanes 0-7 / 8-15 / 16-23 / 24-31 address the matrices (keys 0-7, d 0-7), (same keys, d 8-15), (keys 8-15, ..)
        const int lkey = (lane & 7) + ((lane >> 4) << 3), lc = (lane >> 3) & 1;
        // the queries' first parts in sums of their own: eight truncating additions of full size (four for 64 columns)
        float sl[kBK / 8][4];
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          uint32_t kf[kBK / 16][4];
#pragma unroll
          for (int t = 0; t < kBK / 16; ++t) ldsm4(kb + (16 * t + lkey) * KB + (((map * D / 8 + 2 * k + lc) ^ (lkey & 7)) << 4), kf[t]);
#pragma unroll
          for (int part = 2; part >= 0; --part) {
            const uint4 qv = q_s[(part * (D / 16) + k) * 32];
            const uint32_t qf[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
            for (int t = 0; t < kBK / 8; ++t) {
              float (&c)[4] = part == 0 ? s[t] : sl[t];
              if (k == 0 && part != 1) mma_bf16_first(c, qf, kf[t / 2][2 * (t & 1)], kf[t / 2][2 * (t & 1) + 1]);
              else mma_bf16(c, qf, kf[t / 2][2 * (t & 1)], kf[t / 2][2 * (t & 1) + 1]);
            }
          }
        }
#pragma unroll
        for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
          for (int e = 0; e < 4; e += 2) add2(s[t][e], s[t][e + 1], sl[t][e], sl[t][e + 1]);
        // cap, bias, mask; the block's maximum per row
        if (CAP) {
          bool over = false;
#pragma unroll
          for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) over |= over_cap(p, s[t][e]);
          if (__any_sync(0xffffffffu, over)) {
            const float cap_inv_over = cap_inverse_over(cap_inv);
#pragma unroll
            for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
              for (int e = 0; e < 4; e += 2) {
                const float a = s[t][e], b = s[t][e + 1];
                cap2(s[t][e], s[t][e + 1], cap_inv);
                if (over_cap(p, a)) s[t][e] = capped_over(p.softcap, cap_inv_over, a);
                if (over_cap(p, b)) s[t][e + 1] = capped_over(p.softcap, cap_inv_over, b);
              }
          } else {
#pragma unroll
            for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
              for (int e = 0; e < 4; e += 2) cap2(s[t][e], s[t][e + 1], cap_inv);
          }
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
        float mn[2] = {m[0], m[1]};
#pragma unroll
        for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) mn[e >> 1] = fmaxf(mn[e >> 1], s[t][e]);
        float ps[2] = {0.f, 0.f}, alpha[2], ml[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          mn[r] = quad_max(mn[r]);
          ml[r] = log2_units(mn[r]);
          alpha[r] = ex2(__fsub_rn(log2_units(m[r]), ml[r]));
          m[r] = mn[r];
        }
        if (all) {
#pragma unroll
          for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[t][e] = ex2(fmaf(s[t][e], kLog2e, -ml[e >> 1]));
        } else {
          // a hidden key weighs nothing, also while its row has seen no key at all (maximum still kNegBig)
#pragma unroll
          for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[t][e] = s[t][e] == kNegBig ? 0.f : ex2(fmaf(s[t][e], kLog2e, -ml[e >> 1]));
        }
#pragma unroll
        for (int t = 0; t < kBK / 8; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) ps[e >> 1] += s[t][e];
#pragma unroll
        for (int r = 0; r < 2; ++r) l[r] = l[r] * alpha[r] + quad_sum(ps[r]);
        // weights (three parts) x values: 16 keys x 16 columns per ldmatrix
        const int vkey = (lane & 7) + (((lane >> 3) & 1) << 3), vc = lane >> 4;
        uint32_t a[3][kBK / 16][4];
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float* w = &s[2 * k + (e >> 1)][2 * (e & 1)];
            split3(w[0], w[1], a[0][k][e], a[1][k][e], a[2][k][e]);
          }
#pragma unroll
        for (int t0 = 0; t0 < V / 16; t0 += 2) {
          uint32_t vf[kBK / 16][2][4];
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)
#pragma unroll
            for (int t = 0; t < 2; ++t) ldsm4_t(vb + (16 * k + vkey) * VB + (((2 * (t0 + t) + vc) ^ (vkey & 7)) << 4), vf[k][t]);
          float c[4][4];
#pragma unroll
          for (int part = 2; part >= 0; --part)
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                if (part == 2 && k == 0) mma_bf16_first(c[t], a[part][k], vf[k][t / 2][2 * (t & 1)], vf[k][t / 2][2 * (t & 1) + 1]);
                else mma_bf16(c[t], a[part][k], vf[k][t / 2][2 * (t & 1)], vf[k][t / 2][2 * (t & 1) + 1]);
              }
#pragma unroll
          for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int e = 0; e < 4; e += 2) fma2(o[2 * t0 + t][e], o[2 * t0 + t][e + 1], alpha[e >> 1], c[t][e], c[t][e + 1]);
        }
      }
      set_sync();   // the set has read the buffer that its next block but one overwrites
      v = after;
      b ^= 1;
    }
  }

  float* xch = reinterpret_cast<float*>(sm + W * kQ + (SETS - 1) * 2 * kBuf);   // the last set's buffers: rows handed over
  if (SETS == 2) {
    // the odd blocks' sums join the even blocks'
    constexpr int kRec = 16 * V + 64;
    float* rec = xch + warp * kRec;
    if (set == 1) {
#pragma unroll
      for (int t = 0; t < V / 8; ++t)
#pragma unroll
        for (int r = 0; r < 2; ++r)
          *reinterpret_cast<float2*>(rec + (gid + 8 * r) * V + 8 * t + 2 * tig) = make_float2(o[t][2 * r], o[t][2 * r + 1]);
#pragma unroll
      for (int r = 0; r < 2; ++r)
        if (tig == 0) {
          rec[16 * V + gid + 8 * r] = m[r];
          rec[16 * V + 16 + gid + 8 * r] = l[r];
        }
    }
    __syncthreads();
    if (set == 0) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float m1 = rec[16 * V + gid + 8 * r], l1 = rec[16 * V + 16 + gid + 8 * r], mx = fmaxf(m[r], m1);
        const float ml = log2_units(mx), f0 = ex2(__fsub_rn(log2_units(m[r]), ml));
        const float f1 = l1 == 0.f ? 0.f : ex2(__fsub_rn(log2_units(m1), ml));   // l1 == 0: no odd block was seen
        l[r] = l[r] * f0 + l1 * f1;
#pragma unroll
        for (int t = 0; t < V / 8; ++t) {
          const float2 x = *reinterpret_cast<const float2*>(rec + (gid + 8 * r) * V + 8 * t + 2 * tig);
          o[t][2 * r] = o[t][2 * r] * f0 + x.x * f1;
          o[t][2 * r + 1] = o[t][2 * r + 1] * f0 + x.y * f1;
        }
      }
    }
  }
  const bool writes = active && set == 0;
  if (writes) {
    unsigned odd[2];   // rows gid and gid + 8 that are not finite, a bit per lane
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float z = l[r] * 0.f;
#pragma unroll
      for (int t = 0; t < V / 8; ++t) z = fmaf(o[t][2 * r], 0.f, fmaf(o[t][2 * r + 1], 0.f, z));
      odd[r] = __ballot_sync(0xffffffffu, !(z == 0.f));
    }
    if (odd[0] | odd[1]) {
      float* rows = xch + warp * (SETS == 2 ? 16 * V + 64 : 16 * V);   // SETS == 2: this warp's record, already read
      __syncwarp();
      for (int i = 0; i < n; ++i) {
        const bool again = (odd[i >> 3] >> (4 * (i & 7))) & 15u;
        if (again) row_again<D, MAPS, V>(p, row0 + i, pos0 + i, tile[3], h, map, rows + i * V);
      }
      __syncwarp();
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if (gid + 8 * r >= n || ((odd[r] >> (4 * gid)) & 15u) == 0u) continue;
        l[r] = 1.f;
#pragma unroll
        for (int t = 0; t < V / 8; ++t) {
          const float2 x = *reinterpret_cast<const float2*>(rows + (gid + 8 * r) * V + 8 * t + 2 * tig);
          o[t][2 * r] = x.x;
          o[t][2 * r + 1] = x.y;
        }
      }
    }
  }
  if (MAPS == 2) __syncthreads();   // the records and rows have been read
  if (MAPS == 2) {
    // the second map's rows through shared memory to the warp of the first, which combines, norms and gates them
    float* a2 = xch + (warp >> 1) * 16 * V;
    if (writes && map == 1) {
#pragma unroll
      for (int t = 0; t < V / 8; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) a2[(gid + 8 * (e >> 1)) * V + 8 * t + 2 * tig + (e & 1)] = o[t][e] * (1.0f / l[e >> 1]);
    }
    __syncthreads();
    if (!writes || map == 1) return;
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
  if (!writes) return;
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

template <int D, int MAPS, int V, int SETS, bool CAP>
int launch_kernel(const vila_paged_attn_params& p, int warps, int tpc, cudaStream_t stream) {
  auto kernel = paged_attn_mma_kernel<D, MAPS, V, SETS, CAP>;
  const int smem = warps * 3 * (D / 16) * 512 + SETS * 2 * kBK * (MAPS * D + V) * 2;
  static PerDeviceOnce once;
  if (once.first()) VB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024));
  const long ctas = static_cast<long>((p.ntiles + tpc - 1) / tpc) * p.G;
  VB_CHECK(ctas < (1L << 31), "paged_attention: too many tiles");
  VB_CUDA(launch_serial(kernel, dim3(static_cast<unsigned>(ctas)), dim3(32 * warps * SETS), smem, stream, p, tpc));
  return 0;
}
template <int D, int MAPS, int V, int SETS>
int launch_sets(const vila_paged_attn_params& p, int warps, int tpc, cudaStream_t stream) {
  return p.softcap > 0.f ? launch_kernel<D, MAPS, V, SETS, true>(p, warps, tpc, stream) : launch_kernel<D, MAPS, V, SETS, false>(p, warps, tpc, stream);
}
template <int D, int MAPS, int V>
int launch(const vila_paged_attn_params& p, cudaStream_t stream) {
  const int SH = p.H / p.G * MAPS, tpc = SH >= 4 ? 1 : 4 / SH;   // four warps, or one tile of all the heads
  return SH * tpc <= 4 ? launch_sets<D, MAPS, V, 2>(p, SH * tpc, tpc, stream) : launch_sets<D, MAPS, V, 1>(p, SH * tpc, tpc, stream);
}

bool aligned(const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; }

}  // namespace

// Tiles of up to 16 rows (m16), head sizes that fit the registers, rows on 16-byte boundaries, all heads of a CTA in 8 warps.
bool paged_attention_mma_takes(const vila_paged_attn_params& p) {
  const int maps = maps_of(p.maps);
  return p.max_rows > 1 && p.nsplit == 1 && p.pool_dtype == VILA_DT_BF16 && p.talk == nullptr && p.H / p.G * maps <= kMaxWarps &&
         ((maps == 1 && p.dim == 128 && p.vdim == 128) || (maps == 2 && p.dim == 64 && p.vdim == 128) ||
          (maps == 1 && p.dim == 64 && p.vdim == 64)) &&
         aligned(p.pool, 16) && aligned(p.q, 8) && aligned(p.out, 8);
}

int paged_attention_mma(const vila_paged_attn_params& p, cudaStream_t stream) {
  if (p.maps == 2) return launch<64, 2, 128>(p, stream);
  if (p.dim == 64) return launch<64, 1, 64>(p, stream);
  return launch<128, 1, 128>(p, stream);
}

}  // namespace vb
