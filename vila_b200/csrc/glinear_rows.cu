// vila_glinear of few rows (up to 16, or 64 routed pairs) for bf16 operands: weights streamed through registers, fp32
// multiply-adds on the CUDA cores.
//
// With a handful of rows the weight stream is the bound, and the tensor core buys nothing but its truncating sums: one
// accumulator over K = 2048 is 2.1e-6 off (5.6e-6 where all products are positive), four are 4.7e-7 (8.9e-7), where a
// lane's chain of 64 rounded multiply-adds and a tree over the lanes is 8e-8 (4e-8) off.  A warp owns R weight rows: each
// lane takes 8 of every 256 columns, keeps 16 pieces of 16 bytes in flight (a piece is requested again as soon as it has
// been used), multiplies them with up to 8 token rows from L1, two weight rows per instruction (fma.rn.f32x2), and reduces
// its R x 8 sums with one transposing tree.  More rows of a group take further passes over the same weights, which then
// come from L2.  A sum's order is that of glinear_small_kernel (which keeps fp32 operands, rows off 16-byte boundaries and
// fewer than 128 outputs), whatever R and the number of rows are.
//
// Measured, in brackets glinear_small_kernel and the tcgen05 tiles: 32768 x 2048 on 1 | 8 | 16 rows 28 | 40 | 71 us (8 rows:
// 166, 33), 128 x 8192 on one row 10 (32, 49), 1024 x 2048 on 8 rows 5.8 (28, 16), a routed 1408 x 2048 on 32 pairs of 32
// experts 28 (78, 28) and 2048 x 704 19 (54, 19).  Token rows staged in shared memory by the CTA were slower (the 8 rows 60), a ring
// of weights in shared memory won little there (38) and lost elsewhere (512 x 4096 on one row 9.0 against 6.6).
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "kernels.h"
#include "dtype_any.cuh"
#include "glinear_epi.cuh"

namespace vb {
namespace {

constexpr int kWarps = 4, kPass = 8;   // token rows of a pass
constexpr int kInFlight = 16;          // 16-byte pieces a lane has requested

using f2 = unsigned long long;         // two fp32 numbers in one register pair
__device__ __forceinline__ f2 pair(uint32_t x, uint32_t y) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(x), "r"(y));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float2 unpair(f2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint32_t word(const uint4& u, int i) { return i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w; }

// The sums of a warp's R x NT outputs over its lanes, their epilogue and stores.  v: this lane's share, token * R + weight row.
template <int R, int NT>
__device__ __forceinline__ void finish_rows(const vila_glinear_params& p, const vila_glinear_ext& x, int g, int n0, int m0, int nr,
                                            float (&v)[R * NT]) {
  constexpr int NV = R * NT;
  const int lane = threadIdx.x & 31;
  // every step of the tree halves the sums that a lane carries: value i of lane l ends up as sum (l / SPAN) * PER + i
  int n = NV;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool hi = (lane & off) != 0;
#pragma unroll
      for (int i = 0; i < NV / 2; ++i)
        if (i < n) {
          const float send = hi ? v[i] : v[i + n], keep = hi ? v[i + n] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    }
  }
  constexpr int PER = NV > 32 ? NV / 32 : 1, SPAN = NV > 32 ? 1 : 32 / NV;
  const int first = lane / SPAN * PER, t = first / R, row = first % R;   // PER sums of one token, weight rows next to each other
  const bool ok = t < nr && lane % SPAN == 0;
  const int i = m0 + min(t, nr - 1), orow = p.o_rows ? p.o_rows[i] : i;
  const float is = in_scale_of(p, x, orow), rs = p.row_scale ? p.row_scale[orow] : 1.0f;
  const size_t ob = static_cast<size_t>(orow) * p.ldo + (p.mode == 0 ? static_cast<size_t>(g) * p.o_group_off : 0);
  float z[PER];
#pragma unroll
  for (int c = 0; c < PER; ++c) z[c] = n0 + row + c < p.N ? finish(p, x, v[c] * is, g, n0 + row + c) : 0.f;
  if (p.flags & kGluFlags) {
    if (PER == 1) {
      const float up = __shfl_down_sync(0xffffffffu, z[0], SPAN);       // the next weight row's
      if (ok && !(row & 1) && n0 + row < p.N) st_any(p.out, p.out_dtype, ob + (n0 + row) / 2, glu(z[0], up, p.flags, x) * rs);
    } else {
#pragma unroll
      for (int c = 0; c < PER; c += 2)
        if (ok && n0 + row + c < p.N) st_any(p.out, p.out_dtype, ob + (n0 + row + c) / 2, glu(z[c], z[c + 1 < PER ? c + 1 : c], p.flags, x) * rs);
    }
  } else {
#pragma unroll
    for (int c = 0; c < PER; ++c)
      if (ok && n0 + row + c < p.N) st_any(p.out, p.out_dtype, ob + n0 + row + c, z[c] * rs);
  }
}

// NT token rows from m0 on (the first nr of them exist) times the weight rows n0 .. n0 + R - 1 of group g
template <int R, int NT>
__device__ __forceinline__ void rows_pass(const vila_glinear_params& p, const vila_glinear_ext& x, int g, int n0, int m0, int nr) {
  constexpr int NP = kInFlight / R, NV = R * NT;
  const int lane = threadIdx.x & 31;
  const size_t a_col0 = p.mode == 0 ? static_cast<size_t>(g) * p.a_group_off : 0;
  const __nv_bfloat16* W = static_cast<const __nv_bfloat16*>(p.w) + static_cast<size_t>(g) * p.w_group_stride + 8 * lane;
  const __nv_bfloat16* wr[R];
  const __nv_bfloat16* xr[NT];
#pragma unroll
  for (int r = 0; r < R; ++r) wr[r] = W + static_cast<size_t>(min(n0 + r, p.N - 1)) * p.ldw;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int i = m0 + min(t, nr - 1), row = p.a_rows ? p.a_rows[i] / p.a_row_div : i;
    xr[t] = static_cast<const __nv_bfloat16*>(p.a) + static_cast<size_t>(row) * p.lda + a_col0 + 8 * lane;
  }
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint4 w[NP][R];
#pragma unroll
  for (int q = 0; q < NP; ++q)
#pragma unroll
    for (int r = 0; r < R; ++r) w[q][r] = 256 * q + 8 * lane < p.K ? ldg_stream(wr[r] + 256 * q) : zero;
  f2 acc[NT][R / 2];
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int j = 0; j < R / 2; ++j) acc[t][j] = 0ull;
  for (int k0 = 0; k0 < p.K; k0 += 256 * NP) {
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      const int k = k0 + 256 * q;
      if (k >= p.K) break;                           // uniform over the warp
      uint4 xv[NT];
#pragma unroll
      for (int t = 0; t < NT; ++t) xv[t] = k + 8 * lane < p.K ? __ldg(reinterpret_cast<const uint4*>(xr[t] + k)) : zero;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        f2 wp[R / 2];
#pragma unroll
        for (int j = 0; j < R / 2; ++j) {
          const uint32_t a = word(w[q][2 * j], e >> 1), b = word(w[q][2 * j + 1], e >> 1);
          wp[j] = (e & 1) ? pair(a & 0xffff0000u, b & 0xffff0000u) : pair(a << 16, b << 16);
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const uint32_t u = word(xv[t], e >> 1), v = (e & 1) ? u & 0xffff0000u : u << 16;
          const f2 xx = pair(v, v);
#pragma unroll
          for (int j = 0; j < R / 2; ++j) acc[t][j] = fma2(xx, wp[j], acc[t][j]);
        }
      }
      const int kn = k + 256 * NP;
#pragma unroll
      for (int r = 0; r < R; ++r) w[q][r] = kn + 8 * lane < p.K ? ldg_stream(wr[r] + kn) : zero;
    }
  }
  float v[NV];
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int j = 0; j < R / 2; ++j) {
      const float2 s = unpair(acc[t][j]);
      v[t * R + 2 * j] = s.x;
      v[t * R + 2 * j + 1] = s.y;
    }
  finish_rows<R, NT>(p, x, g, n0, m0, nr, v);
}

template <int R>
__global__ void __launch_bounds__(32 * kWarps, 2) glinear_rows_kernel(const vila_glinear_params p, const vila_glinear_ext x) {
  const int g = blockIdx.y, n0 = (blockIdx.x * kWarps + (threadIdx.x >> 5)) * R;
  if (n0 >= p.N) return;
  const int begin = p.mode == 0 ? 0 : p.seg[g], end = p.mode == 0 ? p.M : p.seg[g + 1];
  for (int m0 = begin; m0 < end; m0 += kPass) {
    const int nr = min(kPass, end - m0);
    if (nr == 1) rows_pass<R, 1>(p, x, g, n0, m0, nr);
    else if (nr == 2) rows_pass<R, 2>(p, x, g, n0, m0, nr);
    else if (nr <= 4) rows_pass<R, 4>(p, x, g, n0, m0, nr);
    else rows_pass<R, 8>(p, x, g, n0, m0, nr);
  }
}

template <int R>
int launch(const vila_glinear_params& p, const vila_glinear_ext& x, cudaStream_t stream) {
  const dim3 grid((p.N + R * kWarps - 1) / (R * kWarps), p.groups);
  VB_CHECK(grid.y <= 65535, "glinear: too many groups (%d)", p.groups);
  VB_CUDA(launch_serial(glinear_rows_kernel<R>, grid, dim3(32 * kWarps), 0, stream, p, x));
  return 0;
}

}  // namespace

// Few rows of bf16 operands, every row of both on a 16-byte boundary, at least 128 outputs.
bool glinear_rows_takes(const vila_glinear_params& p) {
  return p.a_dtype == VILA_DT_BF16 && p.w_dtype == VILA_DT_BF16 && p.M <= (p.mode == 0 ? 16 : 64) && p.N >= 128 && p.K % 8 == 0 &&
         p.lda % 8 == 0 && p.ldw % 8 == 0 && p.w_group_stride % 8 == 0 && p.a_group_off % 8 == 0 && p.groups <= 65535 &&
         reinterpret_cast<uintptr_t>(p.a) % 16 == 0 && reinterpret_cast<uintptr_t>(p.w) % 16 == 0;
}

int glinear_rows(const vila_glinear_params& p, cudaStream_t stream, const vila_glinear_ext& x) {
  const long outputs = static_cast<long>(p.N) * p.groups;
  // Weight rows of a warp: more of them share the loads and conversions of the token rows, fewer of them are more warps.
  // 8192 outputs and up take eight (32768 x 2048 on 8 rows: 40 us, 44 with four, about 70 with two; 16 heads of 512 x 128
  // on one row 3.0, 4.1 and 6.3), 2400 - 7100 four (32 heads of 128 x 512 on one row: 3.1 against 3.4 and 4.3), fewer two
  // (2048 x 4096 on 8 rows: 10.1 against 12.4 and 18.6).
  if (outputs >= 48L * num_sms()) return launch<8>(p, x, stream);
  if (outputs > 16L * num_sms()) return launch<4>(p, x, stream);
  return launch<2>(p, x, stream);
}

}  // namespace vb
