// vila_glinear for bf16 operands on the tensor cores: swap-AB grouped GEMM.
//
// The weight rows are the 128 TMEM lanes of a tile and the token rows its accumulator columns, so that a tile's
// token count is free (a multiple of 16): a routed expert with 5 tokens costs 16 columns and one with 300 costs
// 128 + 128 + 48, where token-major 64- or 128-row tiles would compute padding, and decoded tokens stream every
// weight byte once through TMA with up to 200 KB in flight per SM.  The token rows are fetched through the row
// index (routed experts) by cp.async into the same 128-byte-swizzled layout that TMA gives the weights.
//
//   warps 0-3  token rows: cp.async, one stage ahead of the barrier they arrive on; afterwards the epilogue
//              (TMEM lane = weight row, column = token: bias, activation, gated units, scales, scatter)
//   warp 4     weight rows: TMA tiles of 128 x 64 out of a [K, N, groups] tensor map (rows past N read as zero)
//   warp 5     TMEM allocation and tcgen05.mma
//
// Measured against the CUDA-core and wmma forms it replaces for these operands: a head of 32768 x 2048 on 8 rows
// 166 -> 33 us (weights at 4.1 TB/s); a routed block of 32 experts (1408 | 704 x 2048, 4 per token) 849 -> 405 us on
// 2048 tokens and 167 -> 75 us on 8, routers and residual sums included.
//
// Two CTAs share an SM (<= 112 KB of stages each): one CTA's epilogue runs under the other's products.
// Every output is one sum over K in a fixed order, whatever tile, batch or group its row is in.
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "kernels.h"
#include "dtype_any.cuh"
#include "glinear_epi.cuh"

namespace vb {
namespace {

constexpr int kRowsW = 128, kDepth = 64;            // weight rows and K columns of a stage
constexpr int kThreads = 192, kTokenThreads = 128;
constexpr int kWBytes = kRowsW * kDepth * 2;

__device__ unsigned int g_gave_up;   // waits that ran out of tries (never in a correct run)

// An mbarrier wait that ends: a lost arrival must not leave the GPU spinning.
__device__ __forceinline__ bool mbar_wait_limited(uint64_t* bar, uint32_t parity) {
  for (int i = 0; i < (1 << 20); ++i)
    if (mbar_try_wait(bar, parity)) return true;
  atomicAdd(&g_gave_up, 1u);
  return false;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool ok) {
  const uint32_t n = ok ? 16u : 0u;   // 0: the 16 bytes are filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int BT> struct Shape {   // BT: most tokens of a tile
  static constexpr int kStages = BT <= 16 ? 6 : (BT <= 64 ? 4 : 3);
  static constexpr int kStage = kWBytes + BT * kDepth * 2;
  // K is summed in kAcc accumulators that the epilogue adds: the tensor core truncates as it accumulates, so the
  // error of one long sum grows with its length (K = 2048: 2.1e-6 in one accumulator, 5e-7 in four)
  static constexpr int kAcc = BT <= 64 ? 4 : 2;
  static constexpr int kCols = kAcc * BT;           // TMEM columns: two CTAs of an SM share 512
  static constexpr size_t kSmem = 1024 + static_cast<size_t>(kStages) * kStage + 256 + BT * 16;
};

// Which tokens does tile t of this launch hold?  -> group, first sorted position, count (0: none).
// Every warp finds out for itself: 32 groups per step, tiles counted with a warp scan.
__device__ __forceinline__ int find_tile(const vila_glinear_params& p, int BT, int t, int& g, int& m0) {
  if (p.mode == 0) {
    g = blockIdx.z;
    m0 = t * BT;
    return min(BT, p.M - m0);
  }
  const int lane = threadIdx.x & 31;
  for (int e0 = 0; e0 < p.groups; e0 += 32) {
    const int e = e0 + lane;
    int b = 0, n = 0;
    if (e < p.groups) {
      b = p.seg[e];
      n = p.seg[e + 1] - b;
    }
    const int nt = (n + BT - 1) / BT;
    int end = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, t < end);
    if (hit) {
      const int src = __ffs(hit) - 1;
      const int at = t - __shfl_sync(0xffffffffu, end - nt, src);
      g = e0 + src;
      m0 = __shfl_sync(0xffffffffu, b, src) + at * BT;
      return min(BT, __shfl_sync(0xffffffffu, n, src) - at * BT);
    }
    t -= __shfl_sync(0xffffffffu, end, 31);
  }
  return 0;
}

template <int BT>
__global__ void __launch_bounds__(kThreads) glinear_tc_kernel(const __grid_constant__ CUtensorMap tmap_w,
                                                              const vila_glinear_params p, const vila_glinear_ext x) {
  using S = Shape<BT>;
  constexpr int ST = S::kStages, LAG = ST - 1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + ST * S::kStage);
  uint64_t* empty_bar = full_bar + ST;
  uint64_t* acc_bar = empty_bar + ST;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_bar + 1);
  int* orow_s = reinterpret_cast<int*>(smem + ST * S::kStage + 256);   // [BT] output row (-1: none)
  float* rs_s = reinterpret_cast<float*>(orow_s + BT);                  // [BT] routing weight
  float* is_s = rs_s + BT;                                              // [BT] input scale

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int g = 0, m0 = 0;
  const int count = find_tile(p, BT, blockIdx.x, g, m0);
  if (count <= 0) return;                              // uniform over the CTA
  const int cols = (count + 15) & ~15;                 // accumulator columns in use
  const int n0 = blockIdx.y * kRowsW, nkb = (p.K + kDepth - 1) / kDepth;
  const int per_acc = (nkb + S::kAcc - 1) / S::kAcc, parts = (nkb + per_acc - 1) / per_acc;

  if (tid == 0) {
    tma_prefetch_desc(&tmap_w);
    for (int i = 0; i < ST; ++i) {
      mbar_init(&full_bar[i], kTokenThreads + 1);
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(acc_bar, 1);
    fence_barrier_init();
  }
  if (warp == 5) tmem_alloc<S::kCols>(tmem_ptr);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  bool ok = true;

  if (warp == 4) {
    if (lane == 0) {
      for (int kb = 0; kb < nkb && ok; ++kb) {
        const int s = kb % ST;
        if (kb >= ST) ok = mbar_wait_limited(&empty_bar[s], ((kb / ST) & 1) ^ 1);
        if (!ok) break;
        mbar_arrive_expect_tx(&full_bar[s], kWBytes);
        tma_load_3d(smem + s * S::kStage, &tmap_w, &full_bar[s], kb * kDepth, n0, g);
      }
      if (!ok) __nanosleep(1000000);   // requested tiles land before the CTA's memory is given back
    }
  } else if (warp == 5) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc_bf16(kRowsW, cols, 0, 0);
      int part = 0, left = per_acc;
      uint32_t more = 0;                                // 0: first product of an accumulator
      for (int kb = 0; kb < nkb && ok; ++kb) {
        const int s = kb % ST;
        ok = mbar_wait_limited(&full_bar[s], (kb / ST) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t wa = smem_u32(smem + s * S::kStage);
        const uint64_t ad = make_smem_desc(wa, 16, 1024, kLayoutSW128);
        const uint64_t bd = make_smem_desc(wa + kWBytes, 16, 1024, kLayoutSW128);
#pragma unroll
        for (int k = 0; k < kDepth / 16; ++k) {
          umma_f16(tmem + part * BT, ad + 2 * k, bd + 2 * k, idesc, more);
          more = 1;
        }
        umma_commit(&empty_bar[s]);
        if (--left == 0) {
          ++part;
          left = per_acc;
          more = 0;
        }
      }
      if (ok) umma_commit(acc_bar);
    }
  } else {
    // a thread fetches the 16-byte piece c of the rows r0, r0 + 16, .. of every stage
    const int r0 = tid >> 3, c = tid & 7;
    const __nv_bfloat16* src[BT / 16];
    const __nv_bfloat16* A = static_cast<const __nv_bfloat16*>(p.a) + (p.mode == 0 ? static_cast<size_t>(g) * p.a_group_off : 0);
#pragma unroll
    for (int j = 0; j < BT / 16; ++j) {
      const int i = m0 + r0 + 16 * j;
      const bool row = r0 + 16 * j < count;
      src[j] = row ? A + static_cast<size_t>(p.a_rows ? p.a_rows[i] / p.a_row_div : i) * p.lda + c * 8 : nullptr;
    }
    for (int m = tid; m < BT; m += kTokenThreads) {
      int o = -1;
      float rs = 1.f, is = 1.f;
      if (m < count) {
        const int i = m0 + m;
        o = p.o_rows ? p.o_rows[i] : i;
        if (p.row_scale) rs = p.row_scale[o];
        is = in_scale_of(p, x, o);
      }
      orow_s[m] = o;
      rs_s[m] = rs;
      is_s[m] = is;
    }
    const uint32_t base = smem_u32(smem) + kWBytes + r0 * 128 + ((c ^ (r0 & 7)) << 4);
    for (int kb = 0; kb < nkb && ok; ++kb) {
      const int s = kb % ST;
      if (kb >= ST) ok = mbar_wait_limited(&empty_bar[s], ((kb / ST) & 1) ^ 1);
      if (!ok) break;
      const bool in_k = kb * kDepth + c * 8 < p.K;
#pragma unroll
      for (int j = 0; j < BT / 16; ++j)
        if (16 * j < cols)
          cp_async16(base + s * S::kStage + j * 16 * 128, src[j] && in_k ? src[j] + kb * kDepth : A, src[j] && in_k);
      cp_async_commit();
      if (kb >= LAG) {
        cp_async_wait<LAG>();
        fence_proxy_async_smem();
        mbar_arrive(&full_bar[(kb - LAG) % ST]);
      }
    }
    cp_async_wait<0>();
    fence_proxy_async_smem();
    if (ok) {
      for (int kb = max(0, nkb - LAG); kb < nkb; ++kb) mbar_arrive(&full_bar[kb % ST]);
      ok = mbar_wait_limited(acc_bar, 0);
    }
    ok = __all_sync(0xffffffffu, ok);                // the warp's TMEM loads and shuffles need all lanes
    asm volatile("bar.sync 1, 128;" ::: "memory");   // orow_s, rs_s, is_s
    tc_fence_after();
    if (ok) {
      const int n = n0 + tid;                          // this thread's weight row
      const bool n_ok = n < p.N, gated = (p.flags & kGluFlags) != 0, odd = (n & 1) != 0;
      const float bias = p.bias && n_ok ? ld_any(p.bias, p.w_dtype, static_cast<size_t>(g) * p.bias_group_stride + n) : 0.f;
      const size_t o_col0 = p.mode == 0 ? static_cast<size_t>(g) * p.o_group_off : 0;
      for (int t0 = 0; t0 < cols; t0 += 16) {
        const uint32_t at = tmem + (static_cast<uint32_t>(warp * 32) << 16) + t0;
        float r[16];
        tmem_ld_32x32b_x16(at, reinterpret_cast<uint32_t*>(r));
        tmem_ld_wait();
        for (int q = 1; q < parts; ++q) {
          float more[16];
          tmem_ld_32x32b_x16(at + q * BT, reinterpret_cast<uint32_t*>(more));
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 16; ++k) r[k] += more[k];
        }
        if (gated) {
          // the lanes of a column pair hold gate and up: of two tokens each lane finishes one
#pragma unroll
          for (int k = 0; k < 16; k += 2) {
            const float za = fmaf(r[k], is_s[t0 + k], bias), zb = fmaf(r[k + 1], is_s[t0 + k + 1], bias);
            const float other = __shfl_xor_sync(0xffffffffu, odd ? za : zb, 1);
            const int t = t0 + k + (odd ? 1 : 0), orow = orow_s[t];
            if (orow >= 0 && n_ok)
              st_any(p.out, p.out_dtype, static_cast<size_t>(orow) * p.ldo + o_col0 + (n >> 1),
                     (odd ? glu(other, zb, p.flags, x) : glu(za, other, p.flags, x)) * rs_s[t]);
          }
        } else {
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const int orow = orow_s[t0 + k];
            const float z = fmaf(r[k], is_s[t0 + k], bias);
            if (orow >= 0 && n_ok)
              st_any(p.out, p.out_dtype, static_cast<size_t>(orow) * p.ldo + o_col0 + n, activate(z, p.act, x) * rs_s[t0 + k]);
          }
        }
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc<S::kCols>(tmem);
  }
}

template <int BT>
int launch(const CUtensorMap& tm, const vila_glinear_params& p, const vila_glinear_ext& x, cudaStream_t stream) {
  static PerDeviceOnce once;
  if (once.first())
    VB_CUDA(cudaFuncSetAttribute(glinear_tc_kernel<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Shape<BT>::kSmem)));
  const int tiles = (p.M + BT - 1) / BT + (p.mode == 1 ? p.groups : 0);   // mode 1: upper bound of sum_g ceil(rows_g / BT)
  const dim3 grid(tiles, (p.N + kRowsW - 1) / kRowsW, p.mode == 0 ? p.groups : 1);
  VB_CHECK(grid.y <= 65535 && grid.z <= 65535, "glinear: too many tiles (N=%d groups=%d)", p.N, p.groups);
  VB_CUDA(launch_serial(glinear_tc_kernel<BT>, grid, dim3(kThreads), Shape<BT>::kSmem, stream, tm, p, x));
  return 0;
}

}  // namespace

// 16-byte pieces of A rows, and a tensor map of W: every row of both starts on a 16-byte boundary.  Below 128 weight
// rows a tile would mostly multiply zeros.
bool glinear_tc_takes(const vila_glinear_params& p) {
  return p.a_dtype == VILA_DT_BF16 && p.w_dtype == VILA_DT_BF16 && p.N >= kRowsW && p.K % 8 == 0 && p.lda % 8 == 0 &&
         p.ldw % 8 == 0 && p.ldw >= p.K && p.w_group_stride % 8 == 0 && (p.groups == 1 || p.w_group_stride > 0) &&
         p.a_group_off % 8 == 0 && reinterpret_cast<uintptr_t>(p.a) % 16 == 0 && reinterpret_cast<uintptr_t>(p.w) % 16 == 0;
}

unsigned int stalled_waits() {
  unsigned int n = 0;
  return cudaMemcpyFromSymbol(&n, g_gave_up, sizeof n) == cudaSuccess ? n : ~0u;
}

int glinear_tc(const vila_glinear_params& p, cudaStream_t stream, const vila_glinear_ext& x) {
  CUtensorMap tm;
  const uint64_t gs = p.groups == 1 ? static_cast<uint64_t>(p.N) * p.ldw : p.w_group_stride;
  if (int rc = make_tmap_3d_bf16(&tm, p.w, p.K, p.N, p.groups, p.ldw, gs, kDepth, kRowsW, 1, 128)) return rc;
  // tokens of a tile: all of a plain layer's rows up to 128; of routed rows about twice the mean of a group.  Small
  // tiles leave room for more weight stages (6 of 18 KB), which is what decoded tokens are bound by.
  const int rows = p.mode == 0 ? p.M : 2 * ((p.M + p.groups - 1) / p.groups);
  if (rows <= 16) return launch<16>(tm, p, x, stream);
  if (rows <= 64) return launch<64>(tm, p, x, stream);
  return launch<128>(tm, p, x, stream);
}

}  // namespace vb
