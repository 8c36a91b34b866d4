// vila_glinear for bf16 operands on the tensor cores: persistent swap-AB grouped GEMM.
//
// The weight rows are the 128 TMEM lanes of a tile and the token rows its accumulator columns, so that a tile's
// token count is free (a multiple of 16): a routed expert with 5 tokens costs 16 columns and one with 300 costs
// two tiles of 150, where token-major tiles of fixed height would compute padding, and decoded tokens stream every
// weight byte once through TMA.
//
//   epilogue warps  (4 or 8) TMEM lane = weight row, column = token: bias, activation, gated units, scales, scatter
//   4 gather warps  token rows through the row index (routed experts): cp.async into the 128-byte-swizzled layout.
//                   The copies arrive on the stage's barrier by themselves, so all stages stay in flight; the
//                   consumer orders them before its products with a proxy fence.  (tile::gather4 was measured: 185 us
//                   where cp.async took 140 at the same depth, TMA issues too few rows per clock.)
//   TMA warp        weight tiles of 128 x 64 out of a [K, N, groups] tensor map (rows past N read as zero); token
//                   rows too where they are consecutive
//   MMA warp        TMEM allocation and tcgen05.mma into one of two accumulator sets: a tile's epilogue runs under
//                   the next tile's products
//
// Tiles are dealt round-robin, token tiles fastest, so that the tiles that share weights run together.  A tile size sums K
// in a fixed order, whatever tile or group a row is in, but the sizes cut K into different numbers of accumulators (kAcc):
// the rounding of a row changes where the number of rows changes the tile size.  Few rows are served by glinear_rows.cu,
// whose sums are rounded, not truncated.
//
// Measured against the wmma form it replaces for these operands: the two projections of a routed block of 32 experts
// (1408 | 704 x 2048, 4 per token) on 2048 tokens 720 -> 139 us (94 and 45: tiles of 128 - 256 tokens); the error
// is the wmma form's (2.1e-6 at K = 2048, one accumulator) or less.
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "kernels.h"
#include "dtype_any.cuh"
#include "glinear_epi.cuh"

#include <atomic>
#include <mutex>
#include <type_traits>

namespace vb {
// A word of pinned host memory that a launch which gave up sets: the host reads it without waiting for the device.
namespace {
std::atomic<volatile unsigned int*> g_failed{nullptr};
}
volatile unsigned int* failed_word() {
  static std::once_flag once;
  std::call_once(once, [] {
    void* w = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // the first call may be under capture
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (cudaHostAlloc(&w, sizeof(unsigned int), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
      *static_cast<volatile unsigned int*>(w) = 0u;
      g_failed = static_cast<volatile unsigned int*>(w);
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
  });
  return g_failed;
}

namespace {

constexpr int kRowsW = 128, kDepth = 64;            // weight rows and K columns of a stage
constexpr int kWBytes = kRowsW * kDepth * 2;
constexpr int kGatherWarps = 4, kBox = 64;          // token rows of one TMA box
constexpr int kMaxGroups = 1024;                    // groups whose tile offsets fit shared memory

__device__ unsigned int g_gave_up;   // CTAs that gave up (none in a correct run)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool ok) {
  const uint32_t n = ok ? 16u : 0u;   // 0: the 16 bytes are filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
// arrives (counted) when this thread's copies so far have landed
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int BT> struct Shape {   // BT: most tokens of a tile
  static constexpr int kStages = BT <= 16 ? 6 : 4;
  static constexpr int kEpi = BT <= 64 ? 4 : 8;     // epilogue warps
  static constexpr int kThreads = 32 * (kEpi + kGatherWarps + 2);
  static constexpr int kPerSm = BT <= 64 ? 2 : 1;   // CTAs an SM holds
  static constexpr int kStage = kWBytes + BT * kDepth * 2;
  // K is summed in kAcc accumulators that the epilogue adds: the tensor core truncates as it accumulates, so the
  // error of one long sum grows with its length (K = 2048: 2.1e-6 in one accumulator, 1.0e-6 in two, 4.7e-7 in four)
  static constexpr int kAcc = BT <= 16 ? 4 : (BT <= 64 ? 2 : 1);
  static constexpr int kCols = 2 * kAcc * BT;       // TMEM columns: the CTAs of an SM share 512
  static constexpr int kMeta = 2 * BT * 16;         // two tiles' output rows, routing weights, input scales
  static constexpr size_t smem(int groups) { return 1024 + static_cast<size_t>(kStages) * kStage + 256 + kMeta + 8 * (groups + 1); }
};

struct Tile { int g, m0, count, n0; };

// Token tiles of n rows: as few as possible, of nearly equal size, each a multiple of 16 rows but the last.
__device__ __forceinline__ int tiles_of(int n, int BT) { return (n + BT - 1) / BT; }
__device__ __forceinline__ void piece(int n, int BT, int j, int& off, int& count) {
  const int per = ((n + tiles_of(n, BT) - 1) / tiles_of(n, BT) + 15) & ~15;
  off = j * per;
  count = min(per, n - off);   // may be <= 0 for the last ones
}
// first: [groups + 1] token tiles before each group, then [groups + 1] its sorted positions (mode 1)
__device__ __forceinline__ Tile tile_at(const vila_glinear_params& p, int BT, int it, int n_blocks, const int* first) {
  Tile t;
  if (p.mode == 0) {
    const int per = tiles_of(p.M, BT), q = it / per;
    piece(p.M, BT, it - q * per, t.m0, t.count);
    t.g = q / n_blocks;
    t.n0 = (q - t.g * n_blocks) * kRowsW;
    return t;
  }
  const int total = first[p.groups], q = it / total, j = it - q * total;
  int lo = 0, hi = p.groups;           // first[lo] <= j < first[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (first[mid] <= j) lo = mid;
    else hi = mid;
  }
  const int *seg = first + p.groups + 1, b = seg[lo];
  int off;
  piece(seg[lo + 1] - b, BT, j - first[lo], off, t.count);
  t.g = lo;
  t.m0 = b + off;
  t.n0 = q * kRowsW;
  return t;
}

// EPI: an activation (VILA_ACT_*), or kGatedEpi + the flag of a gated unit.  It is a template parameter because the
// unrolled epilogue would otherwise hold every activation 16 times over: more code than the instruction cache, and the
// misses cost about 300 cycles per output (20 us for the epilogue of a 256-token tile).
constexpr int kGatedEpi = 64;

template <int BT, int EPI>
__global__ void __launch_bounds__(Shape<BT>::kThreads, Shape<BT>::kPerSm)
glinear_tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a,
                  const vila_glinear_params p, const vila_glinear_ext x, const WaitLimit limit, volatile unsigned int* failed) {
  using S = Shape<BT>;
  constexpr int ST = S::kStages, kGather = S::kEpi, kTma = kGather + kGatherWarps, kMma = kTma + 1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + ST * S::kStage);
  uint64_t* empty_bar = full_bar + ST;
  uint64_t* acc_full = empty_bar + ST;   // [2]
  uint64_t* acc_free = acc_full + 2;     // [2]
  uint64_t* meta_bar = acc_free + 2;     // a tile's output rows, weights and scales have been written
  uint64_t* drain_bar = meta_bar + 1;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(drain_bar + 1);
  volatile int* gave_up = reinterpret_cast<int*>(tmem_ptr + 1);
  long long* orow_s = reinterpret_cast<long long*>(smem + ST * S::kStage + 256);   // [2][BT] where the output row starts (-1: none)
  float* rs_s = reinterpret_cast<float*>(orow_s + 2 * BT);              // [2][BT] routing weight
  float* is_s = rs_s + 2 * BT;                                          // [2][BT] input scale
  int* first = reinterpret_cast<int*>(is_s + 2 * BT);                   // [2][groups + 1], see tile_at

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nkb = (p.K + kDepth - 1) / kDepth, n_blocks = (p.N + kRowsW - 1) / kRowsW;
  const int per_acc = (nkb + S::kAcc - 1) / S::kAcc, parts = (nkb + per_acc - 1) / per_acc;
  const bool gathered = p.a_rows != nullptr;

  if (tid == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_a);
    for (int i = 0; i < ST; ++i) {
      mbar_init(&full_bar[i], 1 + (gathered ? 32 * kGatherWarps : 0));
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_free[i], S::kEpi);
    }
    mbar_init(meta_bar, S::kEpi);
    mbar_init(drain_bar, 1);
    *gave_up = 0;
    fence_barrier_init();
  }
  if (warp == kMma) tmem_alloc<S::kCols>(tmem_ptr);
  if (warp == kTma && p.mode == 1) {   // token tiles before each group
    int sum = 0;
    for (int e0 = 0; e0 <= p.groups; e0 += 32) {
      const int e = e0 + lane;
      const int b = p.seg[min(e, p.groups)], b1 = p.seg[min(e + 1, p.groups)];
      if (e <= p.groups) first[p.groups + 1 + e] = b;
      int end = e < p.groups ? tiles_of(b1 - b, BT) : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += v;
      }
      if (e < p.groups) first[e + 1] = sum + end;
      sum += __shfl_sync(0xffffffffu, end, 31);
    }
    if (lane == 0) first[0] = 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  const int total = p.mode == 0 ? tiles_of(p.M, BT) * n_blocks * p.groups : first[p.groups] * n_blocks;
  bool ok = true;
  if (limit.quits >= 0) {
    ok = limit.quits != (warp == kTma ? 0 : warp == kMma ? 1 : warp >= kGather ? 2 : 3);
    if (!ok) *gave_up = 1;
  }

  if (warp == kTma) {
    if (lane == 0) {
      int s = 0, rounds = 0;              // rounds: through all the stages
      uint32_t ph = 1;                    // parity to wait for on an empty barrier: the first round passes
      for (int it = blockIdx.x; it < total && ok; it += gridDim.x) {
        const Tile t = tile_at(p, BT, it, n_blocks, first);
        if (t.count <= 0) continue;
        const int boxes = gathered ? 0 : (BT < kBox ? 1 : (t.count + kBox - 1) / kBox), box = BT < kBox ? BT : kBox;
        const int col0 = p.mode == 0 ? t.g * static_cast<int>(p.a_group_off) : 0;
        const uint32_t bytes = kWBytes + boxes * box * kDepth * 2;
        for (int kb = 0; kb < nkb; ++kb) {
          ok = mbar_wait_limited(&empty_bar[s], ph, gave_up, limit.tries);
          if (!ok) break;
          uint8_t* st = smem + s * S::kStage;
          mbar_arrive_expect_tx(&full_bar[s], bytes);
          tma_load_3d(st, &tmap_w, &full_bar[s], kb * kDepth, t.n0, t.g);
          for (int b = 0; b < boxes; ++b)
            tma_load_2d(st + kWBytes + b * box * kDepth * 2, &tmap_a, &full_bar[s], col0 + kb * kDepth, t.m0 + b * box);
          if (++s == ST) {
            s = 0;
            ph ^= 1;
            ++rounds;
          }
        }
      }
      // Requested tiles land before the CTA's memory is given back, whichever warp gave up (if none did they have long): stages below
      // s in this round, the others in the last.  Behind the CTA's last barrier instead this took 2 % of a large layer's time.
      for (int i = 0; i < ST; ++i) {
        const int round = i < s ? rounds : rounds - 1;
        if (round >= 0) mbar_drain(&full_bar[i], round & 1);
      }
    }
  } else if (warp == kMma) {
    if (lane == 0) {
      int s = 0, k = 0;
      uint32_t ph = 0;
      for (int it = blockIdx.x; it < total && ok; it += gridDim.x) {
        const Tile t = tile_at(p, BT, it, n_blocks, first);
        if (t.count <= 0) continue;
        const uint32_t idesc = make_idesc_bf16(kRowsW, (t.count + 15) & ~15, 0, 0), acc = tmem + (k & 1) * S::kAcc * BT;
        ok = mbar_wait_limited(&acc_free[k & 1], ((k >> 1) & 1) ^ 1, gave_up, limit.tries);
        tc_fence_after();
        int part = 0, left = per_acc;
        uint32_t more = 0;                                // 0: first product of an accumulator
        for (int kb = 0; kb < nkb && ok; ++kb) {
          ok = mbar_wait_limited(&full_bar[s], ph, gave_up, limit.tries);
          if (!ok) break;
          if (gathered) fence_proxy_async_smem();        // the copies that arrived here, before the products below
          tc_fence_after();
          const uint32_t wa = smem_u32(smem + s * S::kStage);
          const uint64_t ad = make_smem_desc(wa, 16, 1024, kLayoutSW128);
          const uint64_t bd = make_smem_desc(wa + kWBytes, 16, 1024, kLayoutSW128);
          const int steps = min(kDepth / 16, (p.K - kb * kDepth + 15) / 16);   // past K the token tile may hold other columns
#pragma unroll
          for (int q = 0; q < kDepth / 16; ++q) {
            if (q >= steps) break;
            umma_f16(acc + part * BT, ad + 2 * q, bd + 2 * q, idesc, more);
            more = 1;
          }
          umma_commit(&empty_bar[s]);
          if (--left == 0) {
            ++part;
            left = per_acc;
            more = 0;
          }
          if (++s == ST) {
            s = 0;
            ph ^= 1;
          }
        }
        if (ok) umma_commit(&acc_full[k & 1]);
        ++k;
      }
      umma_commit(drain_bar);             // products under way end before TMEM and the CTA's memory are given back, too
      mbar_drain(drain_bar, 0);
    }
  } else if (warp >= kGather) {
    if (gathered) {
      // a thread fetches the 16-byte piece c of the rows r0, r0 + 16, .. of every stage
      const int gt = tid - 32 * kGather, r0 = gt >> 3, c = gt & 7;
      const __nv_bfloat16* A = static_cast<const __nv_bfloat16*>(p.a);
      const uint32_t base = smem_u32(smem) + kWBytes + r0 * 128 + ((c ^ (r0 & 7)) << 4);
      int s = 0;
      uint32_t ph = 1;
      // the next tile's row indices are on their way while this tile's rows are fetched
      Tile t, next = {0, 0, 0, 0};
      int rows[BT / 16];
      auto look = [&](int it) {
        next.count = 0;
        if (it < total) next = tile_at(p, BT, it, n_blocks, first);
#pragma unroll
        for (int j = 0; j < BT / 16; ++j) rows[j] = r0 + 16 * j < next.count ? p.a_rows[next.m0 + r0 + 16 * j] : 0;
      };
      look(blockIdx.x);
      for (int it = blockIdx.x; it < total && ok; it += gridDim.x) {
        t = next;
        const __nv_bfloat16* src[BT / 16];
        const size_t col0 = p.mode == 0 ? static_cast<size_t>(t.g) * p.a_group_off : 0;
#pragma unroll
        for (int j = 0; j < BT / 16; ++j) src[j] = A + static_cast<size_t>(rows[j] / p.a_row_div) * p.lda + col0 + c * 8;
        look(it + gridDim.x);
        if (t.count <= 0) continue;
        for (int kb = 0; kb < nkb; ++kb) {
          ok = mbar_wait_limited(&empty_bar[s], ph, gave_up, limit.tries);
          if (!ok) break;
          const bool in_k = kb * kDepth + c * 8 < p.K;
#pragma unroll
          for (int j = 0; j < BT / 16; ++j)
            if (r0 + 16 * j < t.count)                   // later rows' columns are never read
              cp_async16(base + s * S::kStage + j * 16 * 128, in_k ? src[j] + kb * kDepth : A, in_k);
          cp_async_arrive(&full_bar[s]);
          if (++s == ST) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      cp_async_wait_all();
    }
  } else {
    const int quad = warp & 3, half = warp >> 2;
    static_assert(BT <= 32 * S::kEpi, "a thread looks up one token of a tile");
    // what the epilogue of a tile needs to know of token tid is looked up while the tile before it is written out
    Tile t, next = {0, 0, 0, 0};
    int o_next;
    float rs_next, is_next;
    auto look = [&](int it) {
      next.count = 0;
      if (it < total) next = tile_at(p, BT, it, n_blocks, first);
      o_next = -1;
      rs_next = is_next = 1.f;
      if (tid < next.count) {
        const int i = next.m0 + tid;
        o_next = p.o_rows ? p.o_rows[i] : i;
        if (p.row_scale) rs_next = p.row_scale[o_next];
        is_next = in_scale_of(p, x, o_next);
      }
    };
    look(blockIdx.x);
    int k = 0;
    for (int it = blockIdx.x; it < total && ok; it += gridDim.x) {
      t = next;
      if (t.count <= 0) {
        look(it + gridDim.x);
        continue;
      }
      const int cols = (t.count + 15) & ~15, buf = (k & 1) * BT;
      if (tid < cols) {
        orow_s[buf + tid] = o_next < 0 ? -1ll : static_cast<long long>(o_next) * p.ldo;
        rs_s[buf + tid] = rs_next;
        is_s[buf + tid] = is_next;
      }
      look(it + gridDim.x);
      __syncwarp();
      if (lane == 0) mbar_arrive(meta_bar);
      // all lanes or none: the TMEM loads need the whole warp
      ok = __all_sync(0xffffffffu, mbar_wait_limited(meta_bar, k & 1, gave_up, limit.tries) &&
                                       mbar_wait_limited(&acc_full[k & 1], (k >> 1) & 1, gave_up, limit.tries));
      if (!ok) break;
      tc_fence_after();
      const int n = t.n0 + quad * 32 + lane;             // this thread's weight row
      const bool n_ok = n < p.N, odd = (n & 1) != 0;
      const float bias = p.bias && n_ok ? ld_any(p.bias, p.w_dtype, static_cast<size_t>(t.g) * p.bias_group_stride + n) : 0.f;
      const size_t o_col0 = p.mode == 0 ? static_cast<size_t>(t.g) * p.o_group_off : 0;
      const uint32_t acc = tmem + (static_cast<uint32_t>(quad * 32) << 16) + (k & 1) * S::kAcc * BT;
      // The output's type is asked once a tile, a row's offset (which the thread that looked the row up multiplied) is added: with both per
      // output a tile of 128 x 256 took 10400 clocks, twice its products at K = 704.
      auto write = [&](auto* out) {
        using T = std::remove_pointer_t<decltype(out)>;
        auto store = [&](long long off, float v) {
          if (off >= 0 && n_ok) {
            if constexpr (sizeof(T) == 4) out[off] = v;
            else out[off] = __float2bfloat16_rn(v);
          }
        };
        out += EPI >= kGatedEpi ? o_col0 + (n >> 1) : o_col0 + n;
        for (int t0 = 16 * half; t0 < cols; t0 += 4 * S::kEpi) {
          float r[16];
          tmem_ld_32x32b_x16(acc + t0, reinterpret_cast<uint32_t*>(r));
          tmem_ld_wait();
          for (int q = 1; q < parts; ++q) {
            float more[16];
            tmem_ld_32x32b_x16(acc + t0 + q * BT, reinterpret_cast<uint32_t*>(more));
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) r[e] += more[e];
          }
#pragma unroll
          for (int e0 = 0; e0 < 16; e0 += 4) {
            longlong2 off[2];
            off[0] = *reinterpret_cast<const longlong2*>(orow_s + buf + t0 + e0);
            off[1] = *reinterpret_cast<const longlong2*>(orow_s + buf + t0 + e0 + 2);
            const float4 rs4 = *reinterpret_cast<const float4*>(rs_s + buf + t0 + e0), is4 = *reinterpret_cast<const float4*>(is_s + buf + t0 + e0);
            const float rs[4] = {rs4.x, rs4.y, rs4.z, rs4.w}, is[4] = {is4.x, is4.y, is4.z, is4.w};
            if (EPI >= kGatedEpi) {
              // the lanes of a column pair hold gate and up: of two tokens each lane finishes one
#pragma unroll
              for (int e = 0; e < 4; e += 2) {
                const float za = fmaf(r[e0 + e], is[e], bias), zb = fmaf(r[e0 + e + 1], is[e + 1], bias);
                const float other = __shfl_xor_sync(0xffffffffu, odd ? za : zb, 1);
                store(odd ? off[e / 2].y : off[e / 2].x,
                      glu(odd ? other : za, odd ? zb : other, EPI - kGatedEpi, x) * (odd ? rs[e + 1] : rs[e]));
              }
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                store(e & 1 ? off[e / 2].y : off[e / 2].x, activate(fmaf(r[e0 + e], is[e], bias), EPI, x) * rs[e]);
            }
          }
        }
      };
      if (p.out_dtype == VILA_DT_F32) write(static_cast<float*>(p.out));
      else write(static_cast<__nv_bfloat16*>(p.out));
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_free[k & 1]);
      ++k;
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == kMma) {
    tc_fence_after();
    tmem_dealloc<S::kCols>(tmem);
  }
  if (tid == 0 && *gave_up) {
    atomicAdd(&g_gave_up, 1u);
    *failed = 1u;
    __threadfence_system();
  }
}

template <int BT, int EPI>
int launch_epi(const CUtensorMap& tm, const CUtensorMap& ta, const vila_glinear_params& p, const vila_glinear_ext& x, int tries, cudaStream_t stream) {
  using S = Shape<BT>;
  static PerDeviceOnce once;
  if (once.first())
    VB_CUDA(cudaFuncSetAttribute(glinear_tc_kernel<BT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(S::smem(kMaxGroups))));
  const long long tok = (p.M + BT - 1) / BT + (p.mode == 1 ? p.groups : 0);   // mode 1: upper bound of sum_g ceil(rows_g / BT)
  const long long tiles = tok * ((p.N + kRowsW - 1) / kRowsW) * (p.mode == 0 ? p.groups : 1);
  VB_CHECK(tiles < (1LL << 31), "glinear: too many tiles (M=%d N=%d groups=%d)", p.M, p.N, p.groups);
  const int grid = static_cast<int>(tiles < S::kPerSm * num_sms() ? tiles : S::kPerSm * num_sms());
  VB_CUDA(launch_serial(glinear_tc_kernel<BT, EPI>, dim3(grid), dim3(S::kThreads), S::smem(p.mode == 1 ? p.groups : 0), stream, tm, ta, p, x, wait_limit(tries), failed_word()));
  return 0;
}
template <int BT>
int launch(const CUtensorMap& tm, const CUtensorMap& ta, const vila_glinear_params& p, const vila_glinear_ext& x, int tries, cudaStream_t stream) {
  if (p.flags & VILA_FLAG_GLU_CLAMP) return launch_epi<BT, kGatedEpi + VILA_FLAG_GLU_CLAMP>(tm, ta, p, x, tries, stream);
  if (p.flags & VILA_FLAG_GEGLU) return launch_epi<BT, kGatedEpi + VILA_FLAG_GEGLU>(tm, ta, p, x, tries, stream);
  if (p.flags & VILA_FLAG_SWIGLU) return launch_epi<BT, kGatedEpi + VILA_FLAG_SWIGLU>(tm, ta, p, x, tries, stream);
  switch (p.act) {
    case VILA_ACT_SILU: return launch_epi<BT, VILA_ACT_SILU>(tm, ta, p, x, tries, stream);
    case VILA_ACT_RELU2: return launch_epi<BT, VILA_ACT_RELU2>(tm, ta, p, x, tries, stream);
    case VILA_ACT_GELU_TANH: return launch_epi<BT, VILA_ACT_GELU_TANH>(tm, ta, p, x, tries, stream);
    case VILA_ACT_GELU_ERF: return launch_epi<BT, VILA_ACT_GELU_ERF>(tm, ta, p, x, tries, stream);
    case VILA_ACT_XIELU: return launch_epi<BT, VILA_ACT_XIELU>(tm, ta, p, x, tries, stream);
    case VILA_ACT_SOFTCAP: return launch_epi<BT, VILA_ACT_SOFTCAP>(tm, ta, p, x, tries, stream);
    default: return launch_epi<BT, VILA_ACT_NONE>(tm, ta, p, x, tries, stream);
  }
}

}  // namespace

// Tensor maps of A and W: every row of both starts on a 16-byte boundary.  Below 128 weight rows a tile would mostly
// multiply zeros.  Column groups of A follow one another without a gap of zeros, so that their K ends on a 16-column step.
bool glinear_tc_takes(const vila_glinear_params& p) {
  return p.a_dtype == VILA_DT_BF16 && p.w_dtype == VILA_DT_BF16 && p.N >= kRowsW && p.K % 8 == 0 && p.lda % 8 == 0 &&
         p.ldw % 8 == 0 && p.ldw >= p.K && p.w_group_stride % 8 == 0 && (p.groups == 1 || p.w_group_stride > 0) &&
         p.a_group_off % 8 == 0 && p.lda >= p.K && (p.mode == 1 ? p.groups <= kMaxGroups : p.groups == 1 || p.K % 16 == 0) &&
         reinterpret_cast<uintptr_t>(p.a) % 16 == 0 && reinterpret_cast<uintptr_t>(p.w) % 16 == 0;
}

unsigned int stalled_waits() {
  unsigned int n = 0;
  return cudaMemcpyFromSymbol(&n, g_gave_up, sizeof n) == cudaSuccess ? n : ~0u;
}

int wait_status() {
  volatile unsigned int* w = g_failed;
  if (w == nullptr || *w == 0u) return 0;
  *w = 0u;
  set_last_error("a wait of an earlier launch (linear layer or attention) ran out of tries; that launch's output is incomplete");
  return 1;
}

int glinear_tc(const vila_glinear_params& p, cudaStream_t stream, const vila_glinear_ext& x, int tries) {
  VB_CHECK(failed_word() != nullptr, "glinear: no pinned host memory for the status word");
  CUtensorMap tm, ta;
  const uint64_t gs = p.groups == 1 ? static_cast<uint64_t>(p.N) * p.ldw : p.w_group_stride;
  if (int rc = make_tmap_3d_bf16(&tm, p.w, p.K, p.N, p.groups, p.ldw, gs, kDepth, kRowsW, 1, 128)) return rc;
  // tokens of a tile: all of a plain layer's rows up to 256; of routed rows about twice the mean of a group.  Small
  // tiles leave room for two CTAs on an SM and more weight stages, which is what decoded tokens are bound by.
  const int mean2 = 2 * ((p.M + p.groups - 1) / p.groups), rows = p.mode == 0 || p.M < mean2 ? p.M : mean2;
  const int bt = rows <= 16 ? 16 : (rows <= 64 ? 64 : 256);
  // A (consecutive rows): plain and routed layers end at column K, column groups at the row's end; rows past M read as zero
  const bool grouped = p.mode == 0 && p.groups > 1;
  const uint64_t a_cols = grouped ? (p.groups - 1) * static_cast<uint64_t>(p.a_group_off) + p.K : p.K;
  if (int rc = make_tmap_2d_bf16(&ta, p.a, p.M, a_cols, p.lda, bt < kBox ? bt : kBox, kDepth, 128)) return rc;
  if (bt == 16) return launch<16>(tm, ta, p, x, tries, stream);
  if (bt == 64) return launch<64>(tm, ta, p, x, tries, stream);
  return launch<256>(tm, ta, p, x, tries, stream);
}

}  // namespace vb
