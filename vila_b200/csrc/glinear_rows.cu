// vila_glinear of few rows (up to 16, or 64 routed pairs) for bf16 operands: weights streamed once through mma.sync, every
// product of 16 columns into fresh sums that join by rounded additions.
//
// With a handful of rows the weight stream is the bound.  fp32 multiply-adds could not keep up with it from four rows on (8 rows
// of 32768 x 2048: 40 us, 16 rows 72), and a running tensor-core sum over K is truncated at every step (K = 2048 in one
// accumulator: 2.1e-6 off).  Sums of 16 products lose 1 - 2e-8, and their rounded additions in chains of 8 - 16 and a tree
// over the warps no more than the multiply-adds did: 7.8e-8 off at K = 2048 (7.9e-8), 8.3e-8 at 4096 (9.5e-8), 6.6e-8 at 704
// (6.5e-8).  Where all products have one sign the truncation is a bias, 1.3e-8 whatever K is: 4.0 - 4.6e-8 off at K = 512, 4.2 -
// 4.6e-8 at 2048, 4.5e-8 at 8192 (multiply-adds 3.9 - 4.3e-8, 3.9 - 4.5e-8, 4.5 - 4.8e-8).
// A tile is 16 weight rows x 8 or 16 token rows.  A lane's 16 bytes of a weight row are its share of two products' fragments,
// with the token rows' columns dealt alike, so both are loaded as they lie.  A sum's order depends on K, N and the number of
// groups, not on how many rows there are (pairs: from 4 M weights on they take the other form, see the rule).
//
// Measured, in brackets the multiply-adds: 32768 x 2048 on 1 | 8 | 16 rows 24.2 | 25.9 | 29.1 us (28 | 41 | 72), 65536 x 4096 on
// 8 rows 86 = 6.2 TB/s (132), 128 x 8192 on one row 6.1 (8.9), 1024 x 2048 on 8 rows 4.8 (5.8), routed 1408 x 2048 on 32
// pairs of 32 experts 23.7 (25.3 - 29), 2048 x 704 19.5 (18.7 - 20.4), 2816 x 4096 on 60 pairs of 64 experts 123 (142 - 158).
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "kernels.h"
#include "dtype_any.cuh"
#include "glinear_epi.cuh"
#include "mma_bf16.cuh"

namespace vb {
namespace {

__device__ __forceinline__ void add2(float& ax, float& ay, float cx, float cy) {
  asm("{.reg .b64 a, c;\nmov.b64 a, {%0, %1};\nmov.b64 c, {%2, %3};\nadd.rn.f32x2 a, a, c;\nmov.b64 {%0, %1}, a;}" : "+f"(ax), "+f"(ay) : "f"(cx), "f"(cy));
}
// Weights pass through L2 once: they are the first to make room there, so that activations and small tensors stay.
__device__ __forceinline__ uint64_t once_policy() {
  uint64_t v;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(v));
  return v;
}
__device__ __forceinline__ uint4 ld_once(const void* p, uint64_t policy) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0,%1,%2,%3}, [%4], %5;"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p), "l"(policy));
  return r;
}
__device__ __forceinline__ void cp16_once(uint32_t dst, const void* src, bool ok, uint64_t policy) {
  const uint32_t n = ok ? 16u : 0u;   // 0: zeros
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;" ::"r"(dst), "l"(src), "r"(n), "l"(policy) : "memory");
}
__device__ __forceinline__ uint32_t word(const uint4& u, int i) { return i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w; }
// 16 weight rows x 32 columns times 8 token rows: acc[s] takes the s-th 16 columns (a lane's 8 columns are two words of each)
__device__ __forceinline__ void piece(float (&acc)[2][4], const uint4& w0, const uint4& w1, const uint4& xv) {
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const uint32_t a[4] = {word(w0, 2 * s), word(w1, 2 * s), word(w0, 2 * s + 1), word(w1, 2 * s + 1)};
    float f[4];
    mma_bf16_first(f, a, word(xv, 2 * s), word(xv, 2 * s + 1));
    add2(acc[s][0], acc[s][1], f[0], f[1]);
    add2(acc[s][2], acc[s][3], f[2], f[3]);
  }
}
// ---- CTAs that stay ------------------------------------------------------------------------------------------------
// A CTA per SM, 16 warps.  KW of them share a tile of 16 weight rows, each with every KW-th piece of 32 columns; the pieces of a
// warp's tiles are one stream through its ring in shared memory, requested SLOTS - 1 ahead across the tiles, so that a tile's
// end (sums of the KW warps, epilogue) leaves the stream running.  The different token rows lie in shared memory where they fit
// beside the rings.  Routed: the tiles of every pass of eight pairs, of the groups that have any.
constexpr int kStay = 16;              // warps
constexpr int kStreamSmem = 188 * 1024;
constexpr int kMaxPairs = 64, kMaxPasses = kMaxPairs + kMaxPairs / 8;

template <int KW, int NT, int SLOTS, bool ROUTED>
__global__ void __launch_bounds__(32 * kStay, 1) glinear_stream_kernel(const vila_glinear_params p, const vila_glinear_ext x, int token_bytes) {
  constexpr int RW = kStay / KW;                          // tiles side by side
  static_assert(!ROUTED || NT == 1, "glinear: eight pairs a pass");
  extern __shared__ __align__(128) uint8_t ring[];        // [warp][slot][half][lane] 16 bytes: a lane reads its own
  __shared__ float red[2][kStay][8 * NT * 16 + 8];        // a warp's sums of a tile: [token][weight row]
  __shared__ int4 pass_s[ROUTED ? kMaxPasses : 1];        // group, first pair, pairs
  // of a pair (or token row): its row of a and where that lies in shared memory, its row of the output, in_scale and row_scale
  __shared__ int row_s[kMaxPairs], at_s[kMaxPairs], orow_s[kMaxPairs], uniq_s[kMaxPairs], counts_s[2];
  __shared__ float2 scale_s[kMaxPairs];
  uint8_t* const tok = ring + kStay * SLOTS * 1024;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int kw = warp % KW, rw = warp / KW;
  const int tiles = (p.N + 15) / 16, per_warp = ((p.K + 31) / 32 + KW - 1) / KW, pitch = (2 * p.K + 127) / 128 * 128 + 64;
  const int step = gridDim.x * RW, first = blockIdx.x * RW + rw;
  // Pairs outside [seg[0], seg[groups]) belong to no group (M only bounds them, identity choices lie there): nobody has written
  // their rows, nothing of them is read.
  const int live0 = ROUTED ? max(p.seg[0], 0) : 0, live1 = ROUTED ? min(p.M, p.seg[p.groups]) : p.M;
  if (ROUTED && warp == 0) {
    int count = 0;
    for (int g0 = 0; g0 < p.groups; g0 += 32) {
      const int g = g0 + lane, begin = g < p.groups ? p.seg[g] : 0, end = g < p.groups ? p.seg[g + 1] : 0, mine = (end - begin + 7) / 8;
      if (__ballot_sync(0xffffffffu, mine > 0) == 0u) continue;
      int at = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += v;
      }
      for (int i = 0; i < mine; ++i) pass_s[min(count + at - mine + i, kMaxPasses - 1)] = make_int4(g, begin + 8 * i, min(8, end - begin - 8 * i), 0);
      count += __shfl_sync(0xffffffffu, at, 31);
    }
    if (lane == 0) counts_s[0] = min(count, kMaxPasses);
  } else if (!ROUTED && warp == 1) {
    if (lane < p.M) row_s[lane] = uniq_s[lane] = p.a_rows ? p.a_rows[lane] / p.a_row_div : lane;
    at_s[lane] = lane;
    if (lane == 0) counts_s[1] = p.M;
  } else if (warp == 1) {
    // the rows of a without repetitions
    int before = 0;
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const int i = 32 * hf + lane;
      const bool live = i >= live0 && i < live1;
      const int row = live ? (p.a_rows ? p.a_rows[i] / p.a_row_div : i) : -1;
      row_s[i] = row;
      __syncwarp();
      int same = i;
      for (int j = min(32 * hf + 31, live1 - 1); j >= live0; --j)
        if (row_s[j] == row && j <= i) same = j;
      const unsigned fresh = __ballot_sync(0xffffffffu, same == i && live);
      if (same == i && live) {
        at_s[i] = before + __popc(fresh & ((1u << lane) - 1u));
        uniq_s[at_s[i]] = row;
      }
      __syncwarp();
      if (same != i && live) at_s[i] = at_s[same];
      before += __popc(fresh);
    }
    if (lane == 0) counts_s[1] = before;
  } else if (warp == 2 || warp == 3) {
    const int i = threadIdx.x - 64;
    if (i >= live0 && i < live1) {
      const int orow = p.o_rows ? p.o_rows[i] : i;
      orow_s[i] = orow;
      scale_s[i] = make_float2(in_scale_of(p, x, orow), p.row_scale ? p.row_scale[orow] : 1.0f);
    }
  }
  __syncthreads();
  const bool staged = counts_s[1] * pitch <= token_bytes;
  if (staged) {
    const int pieces = p.K / 8;
    for (int t = 0; t < counts_s[1]; ++t) {
      const __nv_bfloat16* row = static_cast<const __nv_bfloat16*>(p.a) + static_cast<size_t>(uniq_s[t]) * p.lda;
      for (int i = threadIdx.x; i < pieces; i += 32 * kStay) cp16(smem_u32(tok) + t * pitch + 16 * i, row + 8 * i, true);
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  const int total = ROUTED ? counts_s[0] * tiles : tiles;
  const int col = 32 * kw + 8 * tig;
  uint8_t* const mine = ring + warp * SLOTS * 1024 + lane * 16;
  const uint32_t mine_at = smem_u32(mine);
  const __nv_bfloat16 *w0 = nullptr, *w1 = nullptr;       // weight rows gid, gid + 8 of the tile that is being requested
  int req_tile = first, req_left = 0, req_k = 0, req_slot = 0;
  const uint64_t policy = once_policy();
  auto request = [&]() {
    if (req_left == 0 && req_tile < total) {
      int n = req_tile * 16 + gid;
      const __nv_bfloat16* W = static_cast<const __nv_bfloat16*>(p.w) + col;
      if (ROUTED) {
        const int u = req_tile / tiles;
        n -= u * tiles * 16;
        W += static_cast<size_t>(pass_s[u].x) * p.w_group_stride;
      }
      w0 = W + static_cast<size_t>(min(n, p.N - 1)) * p.ldw;
      w1 = W + static_cast<size_t>(min(n + 8, p.N - 1)) * p.ldw;
      req_left = per_warp;
      req_k = col;
      req_tile += step;
    }
    if (req_left > 0) {
      const bool in = req_k < p.K;
      cp16_once(mine_at + req_slot * 1024, in ? w0 : p.w, in, policy);
      cp16_once(mine_at + req_slot * 1024 + 512, in ? w1 : p.w, in, policy);
      w0 += 32 * KW;
      w1 += 32 * KW;
      req_k += 32 * KW;
      --req_left;
    }
    req_slot = req_slot == SLOTS - 1 ? 0 : req_slot + 1;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll 1
  for (int q = 0; q < SLOTS - 1; ++q) request();
  asm volatile("cp.async.wait_group %0;" ::"n"(SLOTS - 1) : "memory");
  __syncthreads();                                        // the token rows

  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  int buf = 0, slot = 0, turn = 0;
#pragma unroll 1
  for (int tile = first; tile < total; tile += step) {
    const int u = ROUTED ? tile / tiles : 0;
    const int4 ps = ROUTED ? pass_s[u] : make_int4(0, 0, p.M, 0);
    const uint8_t* xr[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int i = min(ps.y + min(8 * t + gid, ps.z - 1), kMaxPairs - 1);
      xr[t] = staged ? tok + at_s[i] * pitch : reinterpret_cast<const uint8_t*>(static_cast<const __nv_bfloat16*>(p.a) + static_cast<size_t>(row_s[i]) * p.lda);
    }
    float acc[NT][2][4];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[t][e >> 2][e & 3] = 0.f;
    int k = col;
#pragma unroll 2
    for (int left = per_warp; left > 0; --left, k += 32 * KW) {
      uint4 xv[NT];
#pragma unroll
      for (int t = 0; t < NT; ++t) xv[t] = k < p.K ? *reinterpret_cast<const uint4*>(xr[t] + 2 * k) : zero;
      asm volatile("cp.async.wait_group %0;" ::"n"(SLOTS - 2) : "memory");
      const uint4 wa = *reinterpret_cast<const uint4*>(mine + slot * 1024), wb = *reinterpret_cast<const uint4*>(mine + slot * 1024 + 512);
      request();                                          // into the slot of the piece before
      slot = slot == SLOTS - 1 ? 0 : slot + 1;
#pragma unroll
      for (int t = 0; t < NT; ++t) piece(acc[t], wa, wb, xv[t]);
    }
    float* part = red[buf][warp] + 2 * tig * 16 + gid;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) part[(8 * t + (e & 1)) * 16 + 8 * (e >> 1)] = acc[t][0][e] + acc[t][1][e];
    asm volatile("bar.sync %0, %1;" ::"r"(1 + rw), "r"(32 * KW) : "memory");
    // The tile's tokens go to its warps in turn, and the next tile's to those after them.  A lane per weight row, its halves
    // take half of the parts each.
    const int row = lane & 15, n = (tile - u * tiles) * 16 + row;
    for (int t = (kw - turn) & (KW - 1); t < ps.z; t += KW) {
      float v[KW / 2];
#pragma unroll
      for (int i = 0; i < KW / 2; ++i) v[i] = red[buf][rw * KW + 2 * i + (lane >> 4)][t * 16 + row];
#pragma unroll
      for (int o = 1; o < KW / 2; o <<= 1)
#pragma unroll
        for (int i = 0; i < KW / 2; i += 2 * o) v[i] += v[i + o];
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
      const int idx = min(ps.y + t, kMaxPairs - 1);
      const float2 sc = scale_s[idx];
      const size_t ob = static_cast<size_t>(orow_s[idx]) * p.ldo;
      const float z = finish(p, x, v[0] * sc.x, ps.x, min(n, p.N - 1));
      if (p.flags & kGluFlags) {
        const float up = __shfl_down_sync(0xffffffffu, z, 1);   // the next weight row's
        if (lane < 16 && !(row & 1) && n < p.N) st_any(p.out, p.out_dtype, ob + n / 2, glu(z, up, p.flags, x) * sc.y);
      } else if (lane < 16 && n < p.N) {
        st_any(p.out, p.out_dtype, ob + n, z * sc.y);
      }
    }
    turn += ps.z;
    buf ^= 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---- token rows per group, or few weights -----------------------------------------------------------------------------
constexpr int kWarps = 8;
constexpr int kInFlight = 8;           // 16-byte pieces of weights a lane has requested

constexpr int kRowsOf(int kw) { return kWarps / kw * 16; }   // weight rows of a CTA

// NT * 8 token rows from m0 on (the first nr of them exist) times the CTA's weight rows from n_cta on.  KW warps share 16 weight
// rows, each with every KW-th piece of 32 columns.
template <int KW, int NT, bool AHEAD>
__device__ __forceinline__ void rows_pass(const vila_glinear_params& p, const vila_glinear_ext& x, int g, int n_cta, int m0, int nr, float* red) {
  constexpr int NP = kInFlight / 2, kRows = kRowsOf(KW), kPitch = kRows + 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int kw = warp % KW, rw = warp / KW, n0 = n_cta + rw * 16 + gid;
  const size_t a_col0 = p.mode == 0 ? static_cast<size_t>(g) * p.a_group_off : 0;
  const int k_first = 32 * kw + 8 * tig;
  const __nv_bfloat16* W = static_cast<const __nv_bfloat16*>(p.w) + static_cast<size_t>(g) * p.w_group_stride;
  const __nv_bfloat16 *w0 = W + static_cast<size_t>(min(n0, p.N - 1)) * p.ldw, *w1 = W + static_cast<size_t>(min(n0 + 8, p.N - 1)) * p.ldw;
  const __nv_bfloat16* xr[NT];
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const uint64_t policy = once_policy();
  uint4 w[NP][2];
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const int k = k_first + 32 * KW * q;
    w[q][0] = k < p.K ? ld_once(w0 + k, policy) : zero;
    w[q][1] = k < p.K ? ld_once(w1 + k, policy) : zero;
  }
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int i = m0 + min(8 * t + gid, nr - 1), row = p.a_rows ? p.a_rows[i] / p.a_row_div : i;
    xr[t] = static_cast<const __nv_bfloat16*>(p.a) + static_cast<size_t>(row) * p.lda + a_col0;
  }
  float sum[NT][4];
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[t][e] = 0.f;
  for (int k0 = k_first; k0 - 8 * tig < p.K; k0 += 32 * KW * NP) {
    float acc[NT][2][4];                                  // of the pieces in flight: short chains
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[t][e >> 2][e & 3] = 0.f;
    uint4 xv[NP][NT];
    const auto fetch = [&](int q) {
      const int k = k0 + 32 * KW * q;
#pragma unroll
      for (int t = 0; t < NT; ++t) xv[q][t] = k < p.K ? __ldg(reinterpret_cast<const uint4*>(xr[t] + k)) : zero;
    };
    if (AHEAD) {
#pragma unroll
      for (int q = 0; q < NP; ++q) fetch(q);
    }
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      const int k = k0 + 32 * KW * q;
      if (k - 8 * tig >= p.K) break;                      // uniform over the warp
      if (!AHEAD) fetch(q);
#pragma unroll
      for (int t = 0; t < NT; ++t) piece(acc[t], w[q][0], w[q][1], xv[q][t]);
      const int kn = k + 32 * KW * NP;
      w[q][0] = kn < p.K ? ld_once(w0 + kn, policy) : zero;
      w[q][1] = kn < p.K ? ld_once(w1 + kn, policy) : zero;
    }
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) sum[t][e] += acc[t][0][e] + acc[t][1][e];
  }
  // sums of the KW warps through shared memory: [kw][token][weight row]
  float* mine = red + (kw * 8 * NT + 2 * tig) * kPitch + rw * 16 + gid;
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) mine[(8 * t + (e & 1)) * kPitch + 8 * (e >> 1)] = sum[t][e];
  __syncthreads();
  const auto total = [&](int t, int row) {
    float v[KW];
#pragma unroll
    for (int k = 0; k < KW; ++k) v[k] = red[(k * 8 * NT + t) * kPitch + row];
#pragma unroll
    for (int o = 1; o < KW; o <<= 1)
#pragma unroll
      for (int k = 0; k < KW; k += 2 * o) v[k] += v[k + o];
    return v[0];
  };
  const bool pairs = (p.flags & kGluFlags) != 0;
  const int width = pairs ? kRows / 2 : kRows, outs = pairs ? p.N / 2 : p.N, c0 = pairs ? n_cta / 2 : n_cta;
  for (int i = threadIdx.x; i < nr * width; i += 32 * kWarps) {
    const int t = i / width, c = i - t * width;
    if (c0 + c >= outs) continue;
    const int idx = m0 + t, orow = p.o_rows ? p.o_rows[idx] : idx;
    const float is = in_scale_of(p, x, orow);
    const size_t ob = static_cast<size_t>(orow) * p.ldo + (p.mode == 0 ? static_cast<size_t>(g) * p.o_group_off : 0);
    float z;
    if (pairs) z = glu(finish(p, x, total(t, 2 * c) * is, g, n_cta + 2 * c), finish(p, x, total(t, 2 * c + 1) * is, g, n_cta + 2 * c + 1), p.flags, x);
    else z = finish(p, x, total(t, c) * is, g, n_cta + c);
    st_any(p.out, p.out_dtype, ob + c0 + c, z * (p.row_scale ? p.row_scale[orow] : 1.0f));
  }
}

// AHEAD: a pass's token rows are requested before its first weights are waited for.  For grids that the SMs hold at once and
// more than two pieces a warp, where a piece's way to L2 would otherwise follow the one before it (1024 x 1024 on one row 3.7 -> 3.3 us, a routed 512 x 2048
// on one pair 7.0 -> 4.9); larger ones hide it behind a fourth CTA on the SM, which the registers would cost them (2048 x 704
// on 32 pairs of 32 experts 19.0, 21.0 with it).
template <int KW, int NT, bool AHEAD>
__global__ void __launch_bounds__(32 * kWarps, NT == 1 ? (AHEAD ? 3 : 4) : 2) glinear_rows_kernel(const vila_glinear_params p, const vila_glinear_ext x) {
  __shared__ float red[KW * 8 * NT * (kRowsOf(KW) + 4)];
  const int g = blockIdx.y, n0 = blockIdx.x * kRowsOf(KW);
  const int begin = p.mode == 0 ? 0 : p.seg[g], end = p.mode == 0 ? p.M : p.seg[g + 1];
  for (int m0 = begin; m0 < end; m0 += 8 * NT) {
    if (m0 > begin) __syncthreads();                      // the pass before has been read
    rows_pass<KW, NT, AHEAD>(p, x, g, n0, m0, min(8 * NT, end - m0), red);
  }
}

template <int KW, int NT, int SLOTS, bool ROUTED>
int launch_stream(const vila_glinear_params& p, const vila_glinear_ext& x, cudaStream_t stream) {
  const long tiles = static_cast<long>((p.N + 15) / 16) * (ROUTED ? min(p.M, p.groups + p.M / 8) : 1), rw = kStay / KW, ctas = (tiles + rw - 1) / rw;
  constexpr int kTokens = kStreamSmem - kStay * SLOTS * 1024;
  const long rows = static_cast<long>(p.M) * ((2 * p.K + 127) / 128 * 128 + 64);
  const int tokens = static_cast<int>(rows < kTokens ? rows : kTokens);
  static PerDeviceOnce once;
  if (once.first()) VB_CUDA(cudaFuncSetAttribute(glinear_stream_kernel<KW, NT, SLOTS, ROUTED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem));
  VB_CUDA(launch_serial(glinear_stream_kernel<KW, NT, SLOTS, ROUTED>, dim3(static_cast<unsigned>(ctas < num_sms() ? ctas : num_sms())), dim3(32 * kStay),
                        kStay * SLOTS * 1024 + tokens, stream, p, x, tokens));
  return 0;
}
template <int KW>
int launch_stream(const vila_glinear_params& p, const vila_glinear_ext& x, cudaStream_t stream) {
  if (p.mode != 0) return launch_stream<KW, 1, 6, true>(p, x, stream);
  return p.M > 8 ? launch_stream<KW, 2, 6, false>(p, x, stream) : launch_stream<KW, 1, 6, false>(p, x, stream);
}
template <int KW, int NT>
int launch_rows(const vila_glinear_params& p, const vila_glinear_ext& x, cudaStream_t stream) {
  const dim3 grid((p.N + kRowsOf(KW) - 1) / kRowsOf(KW), p.groups);
  constexpr bool kAhead = NT == 1;
  if (kAhead && p.K > 64 * KW && static_cast<long>(grid.x) * grid.y <= 3L * num_sms()) VB_CUDA(launch_serial(glinear_rows_kernel<KW, NT, kAhead>, grid, dim3(32 * kWarps), 0, stream, p, x));
  else VB_CUDA(launch_serial(glinear_rows_kernel<KW, NT, false>, grid, dim3(32 * kWarps), 0, stream, p, x));
  return 0;
}
template <int KW>
int launch(const vila_glinear_params& p, const vila_glinear_ext& x, cudaStream_t stream) {
  return p.mode == 0 && p.M > 8 ? launch_rows<KW, 2>(p, x, stream) : launch_rows<KW, 1>(p, x, stream);
}

}  // namespace

// Few rows of bf16 operands, every row of both on a 16-byte boundary, at least 128 outputs.
bool glinear_rows_takes(const vila_glinear_params& p) {
  return p.a_dtype == VILA_DT_BF16 && p.w_dtype == VILA_DT_BF16 && p.M <= (p.mode == 0 ? 16 : 64) && p.N >= 128 && p.K % 8 == 0 &&
         p.lda % 8 == 0 && p.ldw % 8 == 0 && p.w_group_stride % 8 == 0 && p.a_group_off % 8 == 0 && p.groups <= 65535 &&
         reinterpret_cast<uintptr_t>(p.a) % 16 == 0 && reinterpret_cast<uintptr_t>(p.w) % 16 == 0;
}

// CTAs that stay take what streams long enough to pay for their start (token rows, pass list: 1 - 2 us): one layer of 2048
// columns and more (8 rows x 2048 x 4096: 7.2 us, 13 in the other form; 1024 x 1024: 4.1, 3.6) or of 16 M weights (4 x 32768 x
// 1024: 14.6, 19.5), routed passes of 1024 columns and 4 M weights (8 x 4 pairs x 1408 x 2048: 23.7, 28; one token's two
// pairs x 1024 x 1024: 5.7, 5.2; 704 columns: 21, 19.5) unless the SMs hold all tiles of all groups at once and a group has four
// pairs on average or fewer (1 - 16 pairs of 4 experts x 512 x 2048: 5.0 - 5.5 there, 5.8 - 7.5).  16 warps a tile where rows are long or tiles few, else 8 (16 x 32768
// x 2048: 34 and 29; 8 x 65536 x 4096: 86 and 89).  The other form: 8 warps a tile, 4 for rows of up to 128 columns,
// and of up to 256 where outputs are many (512 | 8192 outputs on one row 2.4 | 3.5 us with 8, 2.5 | 3.3 with 4, on 16 rows
// 2.4 | 5.1 and 2.9 | 3.9; 2048 x 128 on 4 rows 2.4 and 2.3).
int glinear_rows(const vila_glinear_params& p, cudaStream_t stream, const vila_glinear_ext& x) {
  const long weights = static_cast<long>(p.N) * p.K;
  const long tiles = static_cast<long>((p.N + 15) / 16) * p.groups;
  const bool few = tiles <= 3L * num_sms() && p.M <= 4 * p.groups;
  const bool stay = p.mode != 0 ? p.K >= 1024 && weights * min(p.M, p.groups) >= 4L << 20 && !few : p.groups == 1 && (p.K >= 2048 || weights >= 16L << 20);
  if (stay) return p.K >= 4096 || (p.mode == 0 && p.N <= 16 * num_sms()) ? launch_stream<16>(p, x, stream) : launch_stream<8>(p, x, stream);
  return p.K <= 128 || (p.K <= 256 && static_cast<long>(p.N) * p.groups >= 4096) ? launch<4>(p, x, stream) : launch<8>(p, x, stream);
}

}  // namespace vb
