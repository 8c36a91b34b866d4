// vila_ssd_scan of prompt portions (outer_scan.cu has the recurrence) in chunks of 64 tokens on the tensor cores, in fp32
// precision.  With c_i the sum of a chunk's log decays up to token i and S the state before the chunk:
//
//   y_i = exp(c_i) S^T C_i + sum_{j <= i} exp(c_i - c_j) dt_j (C_i . B_j) x_j + D x_i
//   S  <- exp(c_last) S + sum_j B_j (exp(c_last - c_j) dt_j x_j)^T
//
// x, B and C are bf16 numbers; what stands beside them (the state, the weights W_ij of the sum, the weighted x) is fp32 and is
// cut into three bf16 parts (8 + 8 + 8 bits) whose products with a bf16 number are exact.  The tensor core truncates as it
// accumulates: products of full size go into fresh sums of 16 terms (64 for the update), which join by rounded additions.
// c is summed in 64 bits and kept in two fp32 numbers, so that exp(c_i - c_j) has the rounding of the difference only.
// Relative error against float64, 2048 rows, 64 heads of 64 x 128: rows 8.3e-8, state 6.8e-8 (token by token 8.6e-8, 8.5e-8);
// where x, B, C and the state have one sign, so that truncations add up: 8.7e-8, 7.9e-8 (8.7e-8, 9.5e-8).
//
// Grid (sequence, head, 16 PT columns of P): a CTA walks the chunks of its sequence in order.
//   warps 0 - 7    hold the state in mma fragments (16 columns x N PT / 8 channels a warp: the accumulator layout of the update
//                  is the operand layout of the read-out): read-out of chunk c, then the state's update
//   warps 8 - 13   a chunk ahead, blocks of 16 rows x 16 tokens of the lower triangle: scores, weights in fragment order (the
//                  accumulator layout again), weights x x
//   warps 14, 15   the weighted x of the next chunk in fragment order; decays and weights of the one after it
//   warps 8 - 15   cp.async of chunk c + 2; rows of chunk c: read-out, weights x x and D x summed, gated, stored
// with one barrier per chunk for all, and one for the rows.
//
// Columns of a chunk that meet an infinite or NaN number are walked token by token by the same fragments, 16 of them at a time:
// zero weights and zero parts would meet the infinite number, which they do not in the recurrence.
//
// PT = 1 and 2 give the same bits (channels are summed by sixteens, then pairwise), so a sequence's numbers do not depend on
// how many others the launch has.
//
// 2048 rows of one sequence: 64 heads of 64 x 128 in 114 us (token by token, bound by instruction issue: 300), 32 heads 98
// (212), 128 heads 234 (593).  A chunk takes 5700 clocks: read-out 2400, update 1600, beside them scores and weights 4500,
// rows out 800.  The tensor pipe is busy for 2100 of them and shared memory's for 2700; what is left is latency of the
// chains load -> products -> parts -> products.  One set of eight warps that did all in turn took 8000 clocks.
#include <type_traits>
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "kernels.h"
#include "dtype_any.cuh"
#include "mma_bf16.cuh"

namespace vb {
namespace {

constexpr int kL = 64;                    // tokens of a chunk
constexpr int kOwners = 8;                // warps that hold the state
constexpr int kHelpers = 8;
constexpr int kThreads = 32 * (kOwners + kHelpers);

struct Scalars {                          // of a chunk's tokens
  float step[kL];                         // dt
  float lg[kL];                           // log decay
  float ch[kL], cl[kL];                   // c = ch + cl
  float ec[kL];                           // exp(c)
  float wj[kL];                           // exp(c_last - c) dt
  float ec_last;
  float pad[3];
};

template <int N, int PT>
struct Shape {
  static constexpr int PC = 16 * PT;                      // columns of a CTA
  static constexpr int NQ = kOwners / PT;                 // warps that share a 16-column tile
  static constexpr int NS = N / NQ;                       // channels of a warp
  static constexpr int kRow = 2 * (N + 8);                // bytes of a B / C row (an odd number of 16-byte pieces)
  static constexpr int kXRow = 2 * (PC + 8);
  static constexpr int kYRow = PC + 8;                    // floats of a partial row
  static constexpr int kCB = 2 * kL * kRow, kX = kL * kXRow;   // C | B and x of a chunk: three buffers each
  static constexpr int kXW = PT * 4 * 3 * 512;            // weighted x: two buffers
  static constexpr int kYO = NQ * kL * kYRow * 4, kYH = kL * 3 / 2 * kYRow * 4;   // partial rows: one and two buffers
  static constexpr int kSmem = 3 * (kCB + kX) + 2 * (kXW + kYH) + kYO + 4 * static_cast<int>(sizeof(Scalars)) + 16 * PT;
  static_assert(NS >= 16 && kSmem <= 227 * 1024, "ssd_chunk: shape");
};

__device__ __forceinline__ float softplus_f(float z) { return z > 20.0f ? z : log1pf(expf(z)); }
// loads that stay where they are written (the compiler moves others to their use, behind the chunk's products)
__device__ __forceinline__ uint32_t ld_now32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ld_now16(const unsigned short* p) {
  unsigned short v;
  asm volatile("ld.global.nc.b16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void add2(float& ax, float& ay, float cx, float cy) {
  asm("{.reg .b64 a, c;\nmov.b64 a, {%0, %1};\nmov.b64 c, {%2, %3};\nadd.rn.f32x2 a, a, c;\nmov.b64 {%0, %1}, a;}" : "+f"(ax), "+f"(ay) : "f"(cx), "f"(cy));
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

template <int N, int PT>
__global__ void __launch_bounds__(kThreads, 1) ssd_chunk_kernel(const __grid_constant__ vila_ssd_scan_params p, int min_rows) {
  using T = Shape<N, PT>;
  extern __shared__ __align__(128) uint8_t sm[];
  griddep_launch_dependents();   // the shorter sequences' launch may start
  uint8_t* x_s = sm + 3 * T::kCB;
  uint8_t* xw_s = x_s + 3 * T::kX;
  uint8_t* yo_s = xw_s + 2 * T::kXW;                      // read-outs of the state's warps
  uint8_t* yh_s = yo_s + T::kYO;                      // weights x x: rows 0 - 63, then rows 32 - 63 of a second warp
  Scalars* sc_s = reinterpret_cast<Scalars*>(yh_s + 2 * T::kYH);
  volatile int* odd_s = reinterpret_cast<int*>(sc_s + 4); // [chunk & 3][16-column tile]: goes token by token

  // this CTA's sequence: the blockIdx.x-th of those that are not outer_scan's
  const int* sq = p.seqs;
  {
    int want = blockIdx.x, s0 = 0;
    for (;; s0 += 32) {
      if (s0 >= p.nseq) return;
      const int s = s0 + (threadIdx.x & 31);
      unsigned hits = __ballot_sync(0xffffffffu, s < p.nseq && p.seqs[4 * s + 1] >= min_rows);
      if (want >= __popc(hits)) {
        want -= __popc(hits);
        continue;
      }
      for (; want > 0; --want) hits &= hits - 1;
      sq += 4 * (s0 + __ffs(hits) - 1);
      break;
    }
  }
  const int row0 = sq[0], n = sq[1], pos0 = sq[2], slot = sq[3];
  const int h = blockIdx.y, g = h / (p.H / p.G), col0 = blockIdx.z * T::PC;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const int nchunks = (n + kL - 1) / kL;
  const __nv_bfloat16* xbc = static_cast<const __nv_bfloat16*>(p.xbc);
  const size_t xoff = static_cast<size_t>(h) * p.P + col0;
  const uint32_t sm0 = smem_u32(sm), x0 = smem_u32(x_s);
  // ldmatrix addresses: rows lane & 15 with 8-column halves by lane >> 4, or rows by (lane & 7, lane >> 4) with halves by bit 3
  const int ra = lane & 15, ca = (lane >> 4) * 16;
  const int rt = (lane & 7) + ((lane >> 4) << 3), ct = ((lane >> 3) & 1) * 16;
  if (tid < 4 * PT) odd_s[tid] = 0;

  // Rows of a chunk: this thread's are columns ocol .. of row tid / 8.
  constexpr int OC = T::PC / 8;                           // 4 or 2
  const int orow = tid >> 3, ocol = (tid & 7) * OC;
  const float Dh = p.D[h];
  uint32_t zr[OC / 2];
  auto fetch_z = [&](int ch) {
#pragma unroll
    for (int q = 0; q < OC / 2; ++q) zr[q] = 0u;
    if (p.z && ch * kL + orow < n) {
      const __nv_bfloat16* z = static_cast<const __nv_bfloat16*>(p.z) + static_cast<size_t>(row0 + ch * kL + orow) * p.ld_z + xoff + ocol;
#pragma unroll
      for (int q = 0; q < OC / 2; ++q) zr[q] = ld_now32(reinterpret_cast<const uint32_t*>(z) + q);
    }
  };
  float gate[OC];
  auto gates = [&]() {
#pragma unroll
    for (int e = 0; e < OC; e += 2) {
      gate[e] = p.z ? silu_exact_f(bf_lo(zr[e / 2])) : 1.0f;
      gate[e + 1] = p.z ? silu_exact_f(bf_hi(zr[e / 2])) : 1.0f;
    }
  };
  auto rows_out = [&](int ch) {
    const int tok = ch * kL + orow;
    if (tok >= n) return;
    const bool walked = odd_s[(ch & 3) * PT + ocol / 16] != 0;   // the read-outs are whole rows then
    const float* yo = reinterpret_cast<const float*>(yo_s) + orow * T::kYRow + ocol;
    const float* yh = reinterpret_cast<const float*>(yh_s + (ch & 1) * T::kYH) + orow * T::kYRow + ocol;
    const uint8_t* xr = x_s + (ch % 3) * T::kX + orow * T::kXRow + 2 * ocol;
    float v[OC], y[T::NQ + 2][OC];
    auto get = [&](float (&d)[OC], const float* from, bool in) {
      if (OC == 4) *reinterpret_cast<float4*>(d) = in ? *reinterpret_cast<const float4*>(from) : make_float4(0.f, 0.f, 0.f, 0.f);
      else *reinterpret_cast<float2*>(d) = in ? *reinterpret_cast<const float2*>(from) : make_float2(0.f, 0.f);
    };
    get(y[0], yh, !walked);
    get(y[1], yh + 32 * T::kYRow, !walked && orow >= 32);
#pragma unroll
    for (int k = 0; k < T::NQ; ++k) get(y[2 + k], yo + k * kL * T::kYRow, true);
#pragma unroll
    for (int e = 0; e < OC; e += 2) {
      // pairwise
#pragma unroll
      for (int o = 1; o < T::NQ; o <<= 1)
#pragma unroll
        for (int k = 2; k < T::NQ + 2; k += 2 * o) add2(y[k][e], y[k][e + 1], y[k + o][e], y[k + o][e + 1]);
      add2(y[0][e], y[0][e + 1], y[1][e], y[1][e + 1]);
      add2(y[0][e], y[0][e + 1], y[2][e], y[2][e + 1]);
      v[e] = y[0][e];
      v[e + 1] = y[0][e + 1];
      const uint32_t x = *reinterpret_cast<const uint32_t*>(xr + 2 * e);
      v[e] = fmaf(Dh, bf_lo(x), v[e]) * gate[e];
      v[e + 1] = fmaf(Dh, bf_hi(x), v[e + 1]) * gate[e + 1];
    }
    const size_t at = static_cast<size_t>(row0 + tok) * p.ld_out + xoff + ocol;
    if (p.out_dtype == VILA_DT_F32) {
      if (OC == 4) *reinterpret_cast<float4*>(static_cast<float*>(p.out) + at) = *reinterpret_cast<const float4*>(v);
      else *reinterpret_cast<float2*>(static_cast<float*>(p.out) + at) = *reinterpret_cast<const float2*>(v);
    } else {
#pragma unroll
      for (int e = 0; e < OC; e += 2) *reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(p.out) + at + e) = pack_bf16(v[e], v[e + 1]);
    }
  };

  if (warp >= kOwners) {
    // ---------------- helpers ----------------
    const int hw = warp - kOwners, ht = tid - 32 * kOwners;
    const size_t boff = static_cast<size_t>(p.H) * p.P + static_cast<size_t>(g) * N, coff = boff + static_cast<size_t>(p.G) * N;
    const float neg_a = -expf(p.A_log[h]), bias = p.dt_bias[h];
    // C, B, x of a chunk: this thread's pieces are rows t, t + kStep, .. of one column
    constexpr int kPieces = N / 8, kXPieces = T::PC / 8, kStep = 32 * kHelpers / kPieces, kXStep = 32 * kHelpers / kXPieces;
    static_assert(kXStep >= kL, "ssd_chunk: a piece of x per thread");
    const int lt = ht / kPieces, lp = ht % kPieces, xt = ht / kXPieces, xp = ht % kXPieces;
    const __nv_bfloat16* src = xbc + static_cast<size_t>(row0 + lt) * p.ld_xbc + 8 * lp;
    const __nv_bfloat16* xsrc = xbc + static_cast<size_t>(row0 + xt) * p.ld_xbc + xoff + 8 * xp;
    const int64_t chunk_step = kL * p.ld_xbc, row_step = kStep * p.ld_xbc;
    int left = n, buf = 0;   // tokens from the next chunk on, its buffer
    auto load = [&]() {
      if (left <= 0) return;
      const uint32_t dst = sm0 + buf * T::kCB + lt * T::kRow + 16 * lp;
      const __nv_bfloat16* r = src;
#pragma unroll
      for (int k = 0; k < kL / kStep; ++k) {
        const bool in = lt + k * kStep < left;
        const __nv_bfloat16* from = in ? r : xbc;
        cp16(dst + k * kStep * T::kRow, from + coff, in);
        cp16(dst + (kL + k * kStep) * T::kRow, from + boff, in);
        r += row_step;
      }
      if (xt < kL) {
        const bool in = xt < left;
        cp16(x0 + buf * T::kX + xt * T::kXRow + 16 * xp, in ? xsrc : xbc, in);
      }
      src += chunk_step;
      xsrc += chunk_step;
      left -= kL;
      buf = buf == 2 ? 0 : buf + 1;
    };
    auto landed = [&]() { asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory"); };
    // decays and weights: tokens 2 lane, 2 lane + 1 of a chunk
    uint32_t raw[2];
    auto fetch_dt = [&](int ch) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int t = ch * kL + 2 * lane + k;
        raw[k] = t < n ? ld_now16(static_cast<const unsigned short*>(p.dt) + static_cast<size_t>(row0 + t) * p.ld_dt + h) : 0u;
      }
    };
    auto prepare = [&](int ch) {
      Scalars& s = sc_s[ch & 3];
      float step[2], lg[2];
      double c[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const bool in = ch * kL + 2 * lane + k < n;
        step[k] = in ? softplus_f(raw_to_float(raw[k], VILA_DT_BF16) + bias) : 0.f;
        lg[k] = in ? neg_a * step[k] : 0.f;
      }
      double sum = static_cast<double>(lg[0]) + static_cast<double>(lg[1]);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
      }
      const double before = __shfl_up_sync(0xffffffffu, sum, 1), last = __shfl_sync(0xffffffffu, sum, 31);
      c[0] = (lane ? before : 0.0) + static_cast<double>(lg[0]);
      c[1] = sum;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int t = 2 * lane + k;
        const float hi = static_cast<float>(c[k]);
        s.step[t] = step[k];
        s.lg[t] = lg[k];
        s.ch[t] = hi;
        s.cl[t] = static_cast<float>(c[k] - static_cast<double>(hi));
        s.ec[t] = expf(hi);
        s.wj[t] = expf(static_cast<float>(last - c[k])) * step[k];
      }
      if (lane == 0) s.ec_last = expf(static_cast<float>(last));
    };
    // this warp's blocks: rows 16 i .., tokens 16 j0 ..
    const int i = hw < 2 ? 3 : hw < 4 ? 2 : hw == 4 ? 1 : 0;
    const int j0 = hw == 1 || hw == 3 ? 2 : 0;
    const bool two = hw != 3 && hw != 5;
    load();
    if (hw == 7) {
      fetch_dt(0);
      prepare(0);
      if (nchunks > 1) fetch_dt(1);
    }
    landed();
    __syncthreads();
    for (int it = -1; it < nchunks; ++it) {
      load();
      if (ht < PT) odd_s[((it + 2) & 3) * PT + ht] = 0;
      if (it >= 0) fetch_z(it);
      const int ch = it + 1;
      if (ch < nchunks) {
        const Scalars& sc = sc_s[ch & 3];
        const uint32_t cb = sm0 + (ch % 3) * T::kCB, bb = cb + kL * T::kRow, xb = x0 + (ch % 3) * T::kX;
        if (hw >= 6) {
          // ---- weighted x: fragments of 16 columns x 16 tokens
          if (hw == 7 && ch + 1 < nchunks) prepare(ch + 1);
          if (hw == 7 && ch + 2 < nchunks) fetch_dt(ch + 2);
#pragma unroll
          for (int f = hw - 6; f < 4 * PT; f += 2) {
            const int ft = f % PT, k = f / PT;
            uint32_t xf[4], part[3][4];
            ldsm4_t(xb + (16 * k + rt) * T::kXRow + 32 * ft + ct, xf);
            const float2 w0 = *reinterpret_cast<const float2*>(sc.wj + 16 * k + 2 * tig), w1 = *reinterpret_cast<const float2*>(sc.wj + 16 * k + 8 + 2 * tig);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 w = e < 2 ? w0 : w1;
              split3(bf_lo(xf[e]) * w.x, bf_hi(xf[e]) * w.y, part[0][e], part[1][e], part[2][e]);
            }
#pragma unroll
            for (int q = 0; q < 3; ++q)
              *reinterpret_cast<uint4*>(xw_s + (ch & 1) * T::kXW + ((ft * 4 + k) * 3 + q) * 512 + 16 * lane) =
                  make_uint4(part[q][0], part[q][1], part[q][2], part[q][3]);
          }
        } else {
          // ---- scores, weights, weights x x
          float Y[2 * PT][4];
#pragma unroll
          for (int u = 0; u < 2 * PT; ++u)
#pragma unroll
            for (int e = 0; e < 4; ++e) Y[u][e] = 0.f;
          const int ri = 16 * i + gid;
          const float hi[2] = {sc.ch[ri], sc.ch[ri + 8]}, li[2] = {sc.cl[ri], sc.cl[ri + 8]};
          auto blocks = [&](auto count) {   // both of a warp's blocks in one go
            constexpr int NB = decltype(count)::value;
            float c[NB][2][2][4];   // sums of even and of odd steps
#pragma unroll
            for (int k = 0; k < N / 16; ++k) {
              uint32_t cf[4];
              ldsm4(cb + (16 * i + ra) * T::kRow + 32 * k + ca, cf);
#pragma unroll
              for (int b = 0; b < NB; ++b) {
                uint32_t bf[4];
                ldsm4(bb + (16 * (j0 + b) + rt) * T::kRow + 32 * k + ct, bf);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  if (k < 2) {
                    mma_bf16_first(c[b][k][u], cf, bf[2 * u], bf[2 * u + 1]);
                  } else {
                    float f[4];
                    mma_bf16_first(f, cf, bf[2 * u], bf[2 * u + 1]);
#pragma unroll
                    for (int e = 0; e < 4; e += 2) add2(c[b][k & 1][u][e], c[b][k & 1][u][e + 1], f[e], f[e + 1]);
                  }
                }
              }
            }
            uint32_t wf[NB][3][4];
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                const int j = 16 * (j0 + b) + 8 * u + 2 * tig;
                const float2 hj = *reinterpret_cast<const float2*>(sc.ch + j), lj = *reinterpret_cast<const float2*>(sc.cl + j), sj = *reinterpret_cast<const float2*>(sc.step + j);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                  add2(c[b][0][u][2 * r], c[b][0][u][2 * r + 1], c[b][1][u][2 * r], c[b][1][u][2 * r + 1]);
                  const float w0 = c[b][0][u][2 * r] * (expf((hi[r] - hj.x) + (li[r] - lj.x)) * sj.x);
                  const float w1 = c[b][0][u][2 * r + 1] * (expf((hi[r] - hj.y) + (li[r] - lj.y)) * sj.y);
                  split3(j <= ri + 8 * r ? w0 : 0.f, j < ri + 8 * r ? w1 : 0.f, wf[b][0][2 * u + r], wf[b][1][2 * u + r], wf[b][2][2 * u + r]);
                }
              }
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
              for (int q = 0; q < PT; ++q) {
                uint32_t xf[4];
                ldsm4_t(xb + (16 * (j0 + b) + ra) * T::kXRow + 32 * q + ca, xf);
                float f[2][4];
#pragma unroll
                for (int part = 2; part >= 0; --part)
#pragma unroll
                  for (int u = 0; u < 2; ++u) {
                    if (part == 2) mma_bf16_first(f[u], wf[b][part], xf[2 * u], xf[2 * u + 1]);
                    else mma_bf16(f[u], wf[b][part], xf[2 * u], xf[2 * u + 1]);
                  }
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                  for (int e = 0; e < 4; e += 2) add2(Y[2 * q + u][e], Y[2 * q + u][e + 1], f[u][e], f[u][e + 1]);
              }
          };
          if (two) blocks(std::integral_constant<int, 2>());
          else blocks(std::integral_constant<int, 1>());
          // rows 32 - 63 have a second warp, whose rows stand behind the others
          float* y = reinterpret_cast<float*>(yh_s + (ch & 1) * T::kYH) + (ri + (j0 ? 32 : 0)) * T::kYRow + 2 * tig;
#pragma unroll
          for (int q = 0; q < PT; ++q) {
            float odd = 0.f;
#pragma unroll
            for (int u = 2 * q; u < 2 * q + 2; ++u)
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                odd = fmaf(Y[u][2 * r], 0.f, fmaf(Y[u][2 * r + 1], 0.f, odd));
                *reinterpret_cast<float2*>(y + 8 * r * T::kYRow + 8 * u) = make_float2(Y[u][2 * r], Y[u][2 * r + 1]);
              }
            if (!(odd == 0.f)) odd_s[(ch & 3) * PT + q] = 1;
          }
        }
      }
      if (it >= 0) {
        gates();
        asm volatile("bar.sync 1, %0;" ::"r"(kThreads) : "memory");   // its read-outs
        rows_out(it);
      }
      landed();
      __syncthreads();
    }
    return;
  }

  // ---------------- the state's warps ----------------
  constexpr int NT = T::NS / 8, KS = T::NS / 16;          // 8- and 16-channel tiles of a warp
  static_assert(KS <= 2, "ssd_chunk: two partial rows at most");
  const int pt = warp % PT, nq = warp / PT, n0 = nq * T::NS;
  // S[t][e]: columns gid (e < 2) and gid + 8 of the warp's 16, channels n0 + 8 t + 2 tig + (e & 1)
  float S[NT][4];
  float* stp = p.state + ((static_cast<size_t>(slot) * p.H + h) * p.P + col0 + 16 * pt + gid) * N + n0 + 2 * tig;
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float2 v = make_float2(0.f, 0.f);
      if (pos0 > 0) v = *reinterpret_cast<const float2*>(stp + static_cast<size_t>(8 * r) * N + 8 * t);
      S[t][2 * r] = v.x;
      S[t][2 * r + 1] = v.y;
    }
  auto check = [&](int ch) {   // before chunk ch
    float odd = 0.f;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) odd = fmaf(S[t][e], 0.f, odd);
    if (!(odd == 0.f)) odd_s[(ch & 3) * PT + pt] = 1;
  };
  __syncthreads();
  check(0);
  __syncthreads();
  for (int ch = 0; ch < nchunks; ++ch) {
    const Scalars& sc = sc_s[ch & 3];
    const uint32_t cb = sm0 + (ch % 3) * T::kCB, bb = cb + kL * T::kRow;
    fetch_z(ch);
    float* yw = reinterpret_cast<float*>(yo_s) + (nq * kL + gid) * T::kYRow + 16 * pt + 2 * tig;
    if (odd_s[(ch & 3) * PT + pt] == 0) {
      // ---- read-out: the state in three parts against C, every 16 channels in sums of their own (the same in both widths)
      uint32_t sp[KS][2][3][2];
#pragma unroll
      for (int k = 0; k < KS; ++k)
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int hf = 0; hf < 2; ++hf)
            split3(S[2 * k + hf][2 * u], S[2 * k + hf][2 * u + 1], sp[k][u][0][hf], sp[k][u][1][hf], sp[k][u][2][hf]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t cf[KS][4];
#pragma unroll
        for (int k = 0; k < KS; ++k) ldsm4(cb + (16 * i + ra) * T::kRow + 2 * n0 + 32 * k + ca, cf[k]);
        float Y[KS][2][4], Yl[KS][2][4];
#pragma unroll
        for (int k = 0; k < KS; ++k)
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            mma_bf16_first(Y[k][u], cf[k], sp[k][u][0][0], sp[k][u][0][1]);
            mma_bf16_first(Yl[k][u], cf[k], sp[k][u][2][0], sp[k][u][2][1]);
          }
#pragma unroll
        for (int k = 0; k < KS; ++k)
#pragma unroll
          for (int u = 0; u < 2; ++u) mma_bf16(Yl[k][u], cf[k], sp[k][u][1][0], sp[k][u][1][1]);
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const float e = sc.ec[16 * i + gid + 8 * r];
            float a[KS], b[KS];
#pragma unroll
            for (int k = 0; k < KS; ++k) {
              a[k] = Yl[k][u][2 * r];
              b[k] = Yl[k][u][2 * r + 1];
              add2(a[k], b[k], Y[k][u][2 * r], Y[k][u][2 * r + 1]);
              a[k] *= e;
              b[k] *= e;
              if (k) add2(a[0], b[0], a[k], b[k]);        // two of rows_out's partial rows
            }
            *reinterpret_cast<float2*>(yw + (16 * i + 8 * r) * T::kYRow + 8 * u) = make_float2(a[0], b[0]);
          }
      }
      // ---- the state's update
      const float el = sc.ec_last;
      uint32_t wf[3][4][4];
#pragma unroll
      for (int part = 0; part < 3; ++part)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint4 w4 = *reinterpret_cast<const uint4*>(xw_s + (ch & 1) * T::kXW + ((pt * 4 + k) * 3 + part) * 512 + 16 * lane);
          wf[part][k][0] = w4.x;
          wf[part][k][1] = w4.y;
          wf[part][k][2] = w4.z;
          wf[part][k][3] = w4.w;
        }
#pragma unroll
      for (int t = 0; t < NT; t += 2) {
        uint32_t bf[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) ldsm4_t(bb + (16 * k + ra) * T::kRow + 2 * n0 + 16 * t + ca, bf[k]);
        float c[2][4];
#pragma unroll
        for (int part = 2; part >= 0; --part)
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              if (part == 2 && k == 0) mma_bf16_first(c[u], wf[part][k], bf[k][2 * u], bf[k][2 * u + 1]);
              else mma_bf16(c[u], wf[part][k], bf[k][2 * u], bf[k][2 * u + 1]);
            }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[t + u][e] = fmaf(el, S[t + u][e], c[u][e]);
      }
    } else {
      // token by token: fp32 multiply-adds in the order of the recurrence
      const __nv_bfloat16* cs = reinterpret_cast<const __nv_bfloat16*>(sm + (ch % 3) * T::kCB);
      const __nv_bfloat16 *bs = cs + kL * (N + 8), *xs = reinterpret_cast<const __nv_bfloat16*>(x_s + (ch % 3) * T::kX);
      const int nt = min(kL, n - ch * kL);
#pragma unroll 1
      for (int t = 0; t < nt; ++t) {
        const float gt = expf(sc.lg[t]), step = sc.step[t];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float w = step * __bfloat162float(xs[t * (T::PC + 8) + 16 * pt + gid + 8 * r]);
          float y[KS];
#pragma unroll
          for (int k = 0; k < NT; ++k)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int at = t * (N + 8) + n0 + 8 * k + 2 * tig + e;
              float& s = S[k][2 * r + e];
              s = fmaf(gt, s, __bfloat162float(bs[at]) * w);
              y[k / 2] = fmaf(s, __bfloat162float(cs[at]), k % 2 || e ? y[k / 2] : 0.f);
            }
#pragma unroll
          for (int k = 0; k < KS; ++k) y[k] = quad_sum(y[k]);
          if (tig == 0) yw[(t - gid) * T::kYRow + gid + 8 * r] = KS == 2 ? y[0] + y[KS - 1] : y[0];
        }
      }
    }
    check(ch + 1);
    gates();
    asm volatile("bar.sync 1, %0;" ::"r"(kThreads) : "memory");
    rows_out(ch);
    __syncthreads();
  }
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int r = 0; r < 2; ++r)
      *reinterpret_cast<float2*>(stp + static_cast<size_t>(8 * r) * N + 8 * t) = make_float2(S[t][2 * r], S[t][2 * r + 1]);
}

template <int N, int PT>
int launch(const vila_ssd_scan_params& p, int nseq, int min_rows, cudaStream_t stream) {
  auto kernel = ssd_chunk_kernel<N, PT>;
  static PerDeviceOnce once;
  if (once.first()) VB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<N, PT>::kSmem));
  VB_CUDA(launch_serial(kernel, dim3(nseq, p.H, p.P / (16 * PT)), dim3(kThreads), Shape<N, PT>::kSmem, stream, p, min_rows));
  return 0;
}

bool aligned(const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; }

}  // namespace

// bf16 operands with rows on 16-byte boundaries, 64 or 128 channels, heads of whole 16- (64 channels: 32-) column tiles
bool ssd_chunk_takes(const vila_ssd_scan_params& p) {
  return p.in_dtype == VILA_DT_BF16 && ((p.N == 64 && p.P % 32 == 0) || (p.N == 128 && p.P % 16 == 0)) && p.H <= 65535 && p.P / 16 <= 65535 &&
         p.ld_xbc % 8 == 0 && aligned(p.xbc, 16) && (p.z == nullptr || (p.ld_z % 4 == 0 && aligned(p.z, 8))) && p.ld_out % 4 == 0 &&
         aligned(p.out, 16) && aligned(p.state, 8);
}

// Sequences of at least min_rows rows (at most nseq of them).  A CTA of 32 columns takes 5/4 of the time of one of 16 (2048
// rows, one round: 114 and 95 us; the scores are the same in both): whichever takes less over the rounds of CTAs.
int ssd_chunk(const vila_ssd_scan_params& p, int nseq, int min_rows, cudaStream_t stream) {
  const long tiles = static_cast<long>(nseq) * p.H * (p.P / 16), sms = num_sms();
  const bool wide = p.P % 32 == 0 && (tiles / 2 + sms - 1) / sms * 5 <= (tiles + sms - 1) / sms * 4;
  if (p.N == 64) return launch<64, 2>(p, nseq, min_rows, stream);
  return wide ? launch<128, 2>(p, nseq, min_rows, stream) : launch<128, 1>(p, nseq, min_rows, stream);
}

}  // namespace vb
