// nn.Linear for up to 8 token rows (decoded tokens): weights streamed once through registers, fp32 FMA.
//
// With a handful of rows a projection is its weight stream plus the latency of one load and one reduction; the swap-AB
// tcgen05 kernel adds tensor maps, TMEM, a pipeline fill and a split-K exchange to that (9 us for 3 - 11 MB of weights).
// Here a warp owns four weight rows (two gate / up pairs): each lane takes 8 of every 256 columns, requests up to four
// such pieces of all four rows at once (16 x 16 bytes in flight per lane, before the dependency wait where the weights are
// parameters), multiplies them with the token rows from L1 and reduces the 4 x M sums with one transposing tree.  Narrow
// outputs of long rows give KS warps to the same rows, which take turns in the passes over K.  A sum's order depends on
// N and K only, not on M.  Rounding points as in the GEMM kernels.
// Measured against that kernel, weights from HBM, 1 | 4 | 8 rows: 1024 x 1024 2.1 | 2.5 | 4.2 us (6.0 there), 5440 x 1024
// 3.0 | 3.8 | 5.7 (7.7), 2048 x 5632 7.2 | 9.5 | 14.1 (11.9), 4608 x 3584 8.9 | 11.1 | 17.7 (12.5).
#include "common.cuh"
#include "kernels.h"

namespace vb {
namespace {

constexpr int kWarps = 4, kRows = 4, kPieces = 4;   // small CTAs: an SM holds three, so that the last wave is full

struct RowsArgs {
  const __nv_bfloat16 *x, *w;
  __nv_bfloat16* y;
  int ldx, ldw, ldy, M, N, K;
  GemmEpilogue epi;
};

__device__ __forceinline__ void widen(uint4 u, float (&f)[8]) {
  f[0] = bf_lo(u.x); f[1] = bf_hi(u.x); f[2] = bf_lo(u.y); f[3] = bf_hi(u.y);
  f[4] = bf_lo(u.z); f[5] = bf_hi(u.z); f[6] = bf_lo(u.w); f[7] = bf_hi(u.w);
}

template <int M, int KS>   // rows of the launch are M or fewer: the last ones repeat a row and are not written
__global__ void __launch_bounds__(32 * kWarps) gemm_rows_kernel(const RowsArgs a) {
  constexpr int NV = kRows * M;                       // sums of a warp: row * M + token
  __shared__ float part_s[kWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ks = warp % KS;
  const int n0 = (blockIdx.x * (kWarps / KS) + warp / KS) * kRows;
  griddep_launch_dependents();
  const __nv_bfloat16* wr[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) wr[r] = a.w + static_cast<size_t>(min(n0 + r, a.N - 1)) * a.ldw;
  uint4 w[kPieces][kRows];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < kPieces; ++q)
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        const int k = k0 + 256 * q + 8 * lane;
        w[q][r] = k < a.K ? ldg_stream(wr[r] + k) : make_uint4(0u, 0u, 0u, 0u);
      }
  };
  constexpr int kPass = 256 * kPieces;
  if (a.epi.static_w) fetch(ks * kPass);
  griddep_wait();
  if (!a.epi.static_w) fetch(ks * kPass);
  float s[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) s[i] = 0.f;
  for (int k0 = ks * kPass; k0 < a.K; k0 += KS * kPass) {
    if (k0 >= KS * kPass) fetch(k0);
#pragma unroll
    for (int q = 0; q < kPieces; ++q) {
      const int k = k0 + 256 * q + 8 * lane;
      if (k0 + 256 * q >= a.K) break;                 // uniform over the warp
      float wf[kRows][8];
#pragma unroll
      for (int r = 0; r < kRows; ++r) widen(w[q][r], wf[r]);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float xf[8];
        widen(k < a.K ? *reinterpret_cast<const uint4*>(a.x + static_cast<size_t>(min(m, a.M - 1)) * a.ldx + k) : make_uint4(0u, 0u, 0u, 0u), xf);
#pragma unroll
        for (int r = 0; r < kRows; ++r)
#pragma unroll
          for (int e = 0; e < 8; ++e) s[r * M + m] = fmaf(wf[r][e], xf[e], s[r * M + m]);
      }
    }
  }
  // transposing tree: every step halves the sums that a lane carries; lane l ends up with sum l * NV / 32
  int n = NV;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool hi = (lane & off) != 0;
#pragma unroll
      for (int i = 0; i < NV / 2; ++i)
        if (i < n) {
          const float send = hi ? s[i] : s[i + n], keep = hi ? s[i + n] : s[i];
          s[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    } else {
      s[0] += __shfl_xor_sync(0xffffffffu, s[0], off);
    }
  }
  if (KS > 1) {
    part_s[warp][lane] = s[0];
    __syncthreads();
    if (ks != 0) return;
#pragma unroll
    for (int q = 1; q < KS; ++q) s[0] += part_s[warp + q][lane];
  }
  constexpr int SPAN = 32 / NV;                       // lanes that hold the same sum
  const int own = lane / SPAN, row = own / M, m = own - row * M, nn = n0 + row;
  const GemmEpilogue& e = a.epi;
  const float z = s[0] + (e.bias && nn < a.N ? __bfloat162float(e.bias[nn]) : 0.f);
  const float up = __shfl_down_sync(0xffffffffu, z, M * SPAN);   // the next weight row's sum of this token
  if (lane % SPAN != 0 || m >= a.M || nn >= a.N) return;
  float y;
  int col = nn;
  if (e.swiglu) {
    if (row & 1) return;
    col = nn >> 1;
    if (e.swiglu == 2) y = glu_clamp_fast_f(z, up, e.act_pos, e.act_neg);
    else if (e.swiglu == 3) y = gelu_tanh_f(z) * up;
    else y = bf16_round(silu_f(bf16_round(z))) * bf16_round(up);
  } else if (e.act == ACT_NONE) {
    y = z;
  } else {
    const float b = bf16_round(z);
    y = e.act == ACT_GELU_TANH ? gelu_tanh_f(b) : e.act == ACT_GELU_ERF ? gelu_erf_f(b) : e.act == ACT_RELU2 ? fmaxf(b, 0.f) * fmaxf(b, 0.f)
        : e.act == ACT_XIELU ? xielu_fast_f(b, e.act_pos, e.act_neg) : silu_f(b);
  }
  if (e.residual) {
    const int rr = e.res_row_mod > 0 ? m % e.res_row_mod : m;
    y = bf16_round(y) + __bfloat162float(e.residual[static_cast<size_t>(rr) * e.ld_res + col]);
  }
  a.y[static_cast<size_t>(m) * a.ldy + col] = __float2bfloat16_rn(y);
}

template <int M>
int launch(const RowsArgs& a, cudaStream_t stream) {
  const int groups = (a.N + kRows - 1) / kRows, passes = (a.K + 256 * kPieces - 1) / (256 * kPieces), fit = 12 * num_sms();
  const int KS = passes >= 4 && 4 * groups <= fit ? 4 : passes >= 2 && 2 * groups <= fit ? 2 : 1;   // fit: warps the SMs hold
  const dim3 grid((groups + kWarps / KS - 1) / (kWarps / KS)), block(32 * kWarps);
  if (KS == 4) VB_CUDA(launch_pdl(gemm_rows_kernel<M, 4>, grid, block, 0, stream, a));
  else if (KS == 2) VB_CUDA(launch_pdl(gemm_rows_kernel<M, 2>, grid, block, 0, stream, a));
  else VB_CUDA(launch_pdl(gemm_rows_kernel<M, 1>, grid, block, 0, stream, a));
  return 0;
}

}  // namespace

// Rows of both operands on 16-byte boundaries; no fused rotation.  The multiply-adds grow with the rows while the tensor
// cores' time does not: up to 4 rows of 20 M weights and up to 8 of 6 M (37888 x 3584: 55 and 88 us against 50; eight rows
// of 4096 x 2048: 10.4 against 9.3).
bool gemm_rows_takes(const __nv_bfloat16* A, int lda, const __nv_bfloat16* W, int ldw, int M, int N, int K, const GemmEpilogue& epi) {
  const long long weights = static_cast<long long>(N) * K;
  return M >= 1 && weights <= (M <= 4 ? 20000000 : M <= 8 ? 6000000 : 0) && K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0 &&
         reinterpret_cast<uintptr_t>(W) % 16 == 0 && epi.rope_table == nullptr && (!epi.swiglu || N % 2 == 0);
}

int gemm_rows(const __nv_bfloat16* A, int lda, const __nv_bfloat16* W, int ldw, __nv_bfloat16* C, int ldc, int M, int N, int K,
              const GemmEpilogue& epi, cudaStream_t stream) {
  const RowsArgs a = {A, W, C, lda, ldw, ldc, M, N, K, epi};
  if (M == 1) return launch<1>(a, stream);
  if (M == 2) return launch<2>(a, stream);
  if (M <= 4) return launch<4>(a, stream);
  return launch<8>(a, stream);
}

}  // namespace vb
