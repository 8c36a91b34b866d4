// Persistent warp-specialised bf16 GEMM for sm_100a:  C[M,N] = epi(A[M,K] · W[N,K]^T)
//
//   * operands staged global -> shared by TMA (cp.async.bulk.tensor, 128B swizzle, K-major)
//   * tcgen05.mma (cta_group::1, kind::f16, 128 x BLOCK_N x 16) issued by ONE thread
//   * fp32 accumulators live in TMEM, double-buffered so the epilogue of one work segment overlaps
//     the main loop of the next
//   * epilogue warps read TMEM with tcgen05.ld (lane == output row) and fuse
//     bias / GELU / SwiGLU / residual (+ broadcast "row modulo" residual for position embeddings).
//     For short K the epilogue is what a tile takes (K = 1152: 5 us of products in a 256 x 256 tile), and it was bound by
//     latency and by half-sector accesses: eight warps (four before), residual rows requested a chunk ahead and while the
//     products run, 32 bytes per lane and access.  13312 rows: 1152 x 592 with residual 61 -> 34 us, 1152 x 1152 70 -> 39,
//     3456 x 1152 92 -> 77, 4304 x 1152 with GELU 149 -> 113, 1152 x 4304 116 -> 109; 1024 rows 11.1 -> 9.4, 15.4 -> 12.7,
//     19.5 -> 16.6.  K of 3584 and more on 16470 rows: no change beyond what the power cap makes two runs differ by
//   * scheduling: data-parallel over output tiles, or STREAM-K when the tile count does not fill the
//     148 SMs evenly (skinny prefill GEMMs, M = 280): the (tile, k-block) iteration space is cut
//     into equal contiguous ranges, each partial tile is parked in its own fp32 workspace slot and
//     the last-arriving CTA sums the slots in a fixed order (deterministic) and applies the epilogue
//   * programmatic dependent launch: barrier init / TMEM alloc / descriptor prefetch and — for
//     parameter matrices — the first pipeline stages of W overlap the predecessor kernel's tail
//
// Replaces the cuBLAS calls behind nn.Linear on the reference hot path:
//   SigLIP q/k/v/out_proj, fc1/fc2      (modeling_siglip.py:384-387,707-715)
//   mm_projector Linear layers          (base_projector.py:145-162)
//   Qwen2 q/k/v/o, gate/up/down, lm_head (modeling_qwen2.py:164-176,223-226)
//   patch-embed conv as im2col GEMM     (modeling_siglip.py:269-275,322-328)
#include <math.h>

#include "common.cuh"
#include "kernels.h"

namespace vb {

namespace {

constexpr int BLOCK_M = 128;
constexpr int BLOCK_K = 64;  // 64 bf16 = 128 bytes = one 128B-swizzle row
constexpr int UMMA_K = 16;
constexpr int kEpiWarps = 8;      // two per TMEM lane quadrant, each with half of the 32-column chunks
constexpr int kNumThreads = 64 + 32 * kEpiWarps;  // warp0: TMA, warp1: MMA + TMEM alloc, warps 2..9: epilogue

// kPair: a 2-CTA cluster computes one (2*BLOCK_M) x BLOCK_N tile with tcgen05.mma.cta_group::2 —
// each CTA stages its own 128 rows of A and HALF of the W tile (BLOCK_N/2 rows); the tensor cores of
// both SMs read both halves, so the bytes each SM pulls through its L2 port per MAC drop by 1/3
// (128x256 tile: 48 KB -> 32 KB per k-block), which is what bounds the single-CTA kernel.
//
// kMode 2 (split-K pair): a 2-CTA cluster computes one 128 x BLOCK_N tile, each CTA half of the K
// range with ordinary cta_group::1 MMAs; the two fp32 partials are exchanged through distributed
// shared memory (each CTA parks the half of the columns it does NOT finalise, the peer pulls it),
// so under-filled GEMMs (N = 1152 ViT out_proj / fc2: 72 tiles) use all 148 SMs.  One tile per pair.
enum { kModeSingle = 0, kModePair = 1, kModeSplitK2 = 2 };

template <int BLOCK_N, int kStages, int kMode = kModeSingle>
struct GemmSmem {
  static constexpr bool kPair = kMode == kModePair;
  static constexpr int kABytes = BLOCK_M * BLOCK_K * 2;
  static constexpr int kBRows = kPair ? BLOCK_N / 2 : BLOCK_N;  // W rows staged by one CTA
  static constexpr int kBBytes = kBRows * BLOCK_K * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kBarrierBytes = (2 * kStages + 4) * 8 + 16;
  static constexpr int kTotal = kStages * kStageBytes + kBarrierBytes + 1024;  // + align slack
};


// 32 bytes (a whole sector of a row) per lane
__device__ __forceinline__ void ldg_v8(const void* p, uint4& a, uint4& b) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "l"(p) : "memory");
}
__device__ __forceinline__ void stg_v8(void* p, const uint4& a, const uint4& b) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
}

__device__ __forceinline__ float4 ld_cg_v4(const float* p) {
  float4 r;
  asm volatile("ld.global.cg.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
               : "l"(p));
  return r;
}

// Tile rasterisation: tiles are numbered so that the CTAs working at the same time share operand
// panels in L2.  Plain M-fastest numbering streams the whole A matrix once per N block (ncu, ViT qkv
// at M = 65536: 2.5 GB of DRAM traffic for 0.61 GB of operands + output).  Tiles are therefore grouped
// in bands of kBandM M-blocks; inside a band M runs fastest, then N: the ~74-148 concurrent tiles
// touch kBandM A panels and a sliding window of W panels.  With <= kBandM M-blocks (every prefill
// shape up to 2048 tokens) this IS the M-fastest order.
constexpr int kBandM = 8;
__device__ __forceinline__ void tile_coords(int t, int num_m_blocks, int num_n_blocks, int& m_blk, int& n_blk) {
  const int per_band = kBandM * num_n_blocks;
  const int band = t / per_band;
  const int r = t - band * per_band;
  const int m0 = band * kBandM;
  const int bm = min(kBandM, num_m_blocks - m0);
  n_blk = r / bm;
  m_blk = m0 + (r - n_blk * bm);
}

// Work decomposition shared by the three warp roles: a CTA walks a sequence of segments
// (tile, [kb0, kb1)).  Data-parallel: whole tiles blockIdx.x, +gridDim.x, ...  Stream-K: the
// contiguous iteration range [it0, it1) of the (tile, k-block) space.
struct Sched {
  int nkb, num_m_blocks, num_tiles;
  int stream_k;
  long it, it_end;  // stream-K
  int tile;         // data-parallel
  int stride;  // data-parallel: tiles between two visits of this CTA (or CTA pair)
  // tile_m: rows of one scheduling tile (128, or 256 for a CTA pair); worker/n_workers: index and
  // number of the units that walk the tile list (CTAs, or CTA pairs)
  __device__ __forceinline__ Sched(int M, int N, int K, int block_n, int stream_k_, int tile_m = BLOCK_M,
                                   int worker = blockIdx.x, int n_workers = gridDim.x) {
    nkb = (K + BLOCK_K - 1) / BLOCK_K;
    num_m_blocks = (M + tile_m - 1) / tile_m;
    num_tiles = num_m_blocks * ((N + block_n - 1) / block_n);
    stream_k = stream_k_;
    const long total = static_cast<long>(num_tiles) * nkb;
    it = total * worker / n_workers;
    it_end = total * (worker + 1) / n_workers;
    tile = worker;
    stride = n_workers;
  }
  // returns false when done; otherwise the next segment
  __device__ __forceinline__ bool next(int& t, int& kb0, int& kb1) {
    if (stream_k) {
      if (it >= it_end) return false;
      t = static_cast<int>(it / nkb);
      kb0 = static_cast<int>(it - static_cast<long>(t) * nkb);
      const long rem = it_end - it;
      kb1 = (nkb - kb0) < rem ? nkb : kb0 + static_cast<int>(rem);
      it += kb1 - kb0;
      return true;
    }
    if (tile >= num_tiles) return false;
    t = tile;
    kb0 = 0;
    kb1 = nkb;
    tile += stride;
    return true;
  }
};

template <int BLOCK_N, int kStages, int kMode>
__global__ void __launch_bounds__(kNumThreads, 1)
gemm_bf16_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a,
                         const __grid_constant__ CUtensorMap tmap_w, __nv_bfloat16* __restrict__ C,
                         int ldc, int M, int N, int K, GemmEpilogue epi) {
  using S = GemmSmem<BLOCK_N, kStages, kMode>;
  constexpr bool kPair = kMode == kModePair;
  constexpr bool kSplit2 = kMode == kModeSplitK2;
  constexpr bool kCluster = kPair || kSplit2;
  constexpr int TILE_M = kPair ? 2 * BLOCK_M : BLOCK_M;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + kStages * S::kABytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kStages * S::kStageBytes);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* tmem_full = empty_bar + kStages;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  uint32_t* last_flag = tmem_ptr + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_m_blocks = (M + TILE_M - 1) / TILE_M;
  const int num_n_blocks = (N + BLOCK_N - 1) / BLOCK_N;
  const int stream_k = (!kCluster && epi.split_k > 1) ? 1 : 0;
  const uint32_t rank = kCluster ? cluster_ctarank() : 0u;        // CTA within the pair
  const uint32_t mrank = kPair ? rank : 0u;                       // pair mode: which half of the operands
  const int worker = kCluster ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
  const int n_workers = kCluster ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);
  // split-K pair: this CTA's k-block range of every tile
  const int nkb_all = (K + BLOCK_K - 1) / BLOCK_K;
  const int sk_lo = (kSplit2 && rank == 1) ? (nkb_all + 1) / 2 : 0;
  const int sk_hi = (kSplit2 && rank == 0) ? (nkb_all + 1) / 2 : nkb_all;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_w);
#pragma unroll
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(&tmem_full[0], 1);
    mbar_init(&tmem_full[1], 1);
    // pair: one arrival per epilogue warp of BOTH CTAs, on the leader's barrier
    mbar_init(&tmem_empty[0], kPair ? 2 * kEpiWarps : 32 * kEpiWarps);
    mbar_init(&tmem_empty[1], kPair ? 2 * kEpiWarps : 32 * kEpiWarps);
    fence_barrier_init();
  }
  if (warp == 1) {
    if (kPair) tmem_alloc_pair<2 * BLOCK_N>(tmem_ptr);
    else tmem_alloc<2 * BLOCK_N>(tmem_ptr);
  }
  tc_fence_before();
  if (kCluster) cluster_sync_all();  // the peer's barriers exist before any remote signal
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  griddep_launch_dependents();

  if (warp == 0) {
    // ===================== TMA producer =====================
    if (lane == 0) {
      Sched sch(M, N, K, BLOCK_N, stream_k, TILE_M, worker, n_workers);
      // every load of a pair reports to the LEADER's full barrier, which expects both CTAs' bytes
      auto load = [&](void* dst, const CUtensorMap* tm, int i, int c0, int c1) {
        if (kPair) tma_load_2d_pair(dst, tm, mapa_u32(smem_u32(&full_bar[i]), 0), c0, c1);
        else tma_load_2d(dst, tm, &full_bar[i], c0, c1);
      };
      constexpr uint32_t kTxBytes = S::kStageBytes * (kPair ? 2 : 1);
      const int a_row_off = static_cast<int>(mrank) * BLOCK_M;
      const int w_row_off = static_cast<int>(mrank) * S::kBRows;
      int stage = 0;
      uint32_t phase = 0;
      int t, kb0, kb1;
      bool waited = false;
      // W is a parameter: fetch its first stages before the dependency wait (A comes after)
      int pre = 0;
      int pt = 0, pkb0 = 0, pkb1 = 0;
      Sched peek = sch;
      const bool have_first = peek.next(pt, pkb0, pkb1);
      if (kSplit2) {
        pkb0 = sk_lo;
        pkb1 = sk_hi;
      }
      if (epi.static_w && have_first) {
        pre = min(kStages, pkb1 - pkb0);
        int m_blk_unused, n_blk;
        tile_coords(pt, num_m_blocks, num_n_blocks, m_blk_unused, n_blk);
        for (int i = 0; i < pre; ++i) {
          if (mrank == 0) mbar_arrive_expect_tx(&full_bar[i], kTxBytes);
          load(smem_b + i * S::kBBytes, &tmap_w, i, (pkb0 + i) * BLOCK_K, n_blk * BLOCK_N + w_row_off);
        }
      }
      griddep_wait();
      waited = true;
      (void)waited;
      bool first = true;
      while (sch.next(t, kb0, kb1)) {
        int m_blk, n_blk;
        tile_coords(t, num_m_blocks, num_n_blocks, m_blk, n_blk);
        if (kSplit2) {
          kb0 = sk_lo;
          kb1 = sk_hi;
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (first && (kb - kb0) < pre) {
            // W already in flight for this stage: only A is missing
            load(smem_a + stage * S::kABytes, &tmap_a, stage, kb * BLOCK_K, m_blk * TILE_M + a_row_off);
          } else {
            mbar_wait(&empty_bar[stage], phase ^ 1);
            if (mrank == 0) mbar_arrive_expect_tx(&full_bar[stage], kTxBytes);
            load(smem_a + stage * S::kABytes, &tmap_a, stage, kb * BLOCK_K, m_blk * TILE_M + a_row_off);
            load(smem_b + stage * S::kBBytes, &tmap_w, stage, kb * BLOCK_K, n_blk * BLOCK_N + w_row_off);
          }
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        first = false;
      }
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (single thread) =====================
    if (lane == 0 && mrank == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(TILE_M, BLOCK_N, 0, 0);
      Sched sch(M, N, K, BLOCK_N, stream_k, TILE_M, worker, n_workers);
      int stage = 0;
      uint32_t phase = 0;
      int as = 0;
      uint32_t aphase = 0;
      int t, kb0, kb1;
      while (sch.next(t, kb0, kb1)) {
        if (kSplit2) {
          kb0 = sk_lo;
          kb1 = sk_hi;
        }
        mbar_wait(&tmem_empty[as], aphase ^ 1);
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + as * BLOCK_N;
        for (int kb = kb0; kb < kb1; ++kb) {
          mbar_wait(&full_bar[stage], phase);
          tc_fence_after();
          const uint64_t a_desc =
              make_smem_desc(smem_u32(smem_a + stage * S::kABytes), 16, 1024, kLayoutSW128);
          const uint64_t b_desc =
              make_smem_desc(smem_u32(smem_b + stage * S::kBBytes), 16, 1024, kLayoutSW128);
#pragma unroll
          for (int k = 0; k < BLOCK_K / UMMA_K; ++k) {
            // advance 32 bytes (16 bf16) along K inside the 128B swizzle atom: +2 in addr>>4 units
            const uint32_t acc = (kb != kb0 || k != 0) ? 1u : 0u;
            if (kPair) umma_f16_pair(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, acc);
            else umma_f16(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, acc);
          }
          // frees this smem stage (in both CTAs of a pair) when the MMAs retire
          if (kPair) umma_commit_pair(&empty_bar[stage]);
          else umma_commit(&empty_bar[stage]);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (kPair) umma_commit_pair(&tmem_full[as]);  // accumulator complete -> epilogue(s)
        else umma_commit(&tmem_full[as]);
        if (++as == 2) {
          as = 0;
          aphase ^= 1;
        }
      }
    }
  } else {
    // ===================== epilogue warps (TMEM -> regs -> global) =====================
    const int quad = warp & 3;  // TMEM lane quadrant this warp may access
    const int upper = (warp - 2) >> 2;  // which half of the quadrant's chunks this warp takes
    const bool wide_c = ldc % 16 == 0 && reinterpret_cast<uintptr_t>(C) % 32 == 0;
    const bool wide_res = epi.ld_res % 16 == 0 && reinterpret_cast<uintptr_t>(epi.residual) % 32 == 0;
    const int epi_tid = threadIdx.x - 64;
    Sched sch(M, N, K, BLOCK_N, stream_k, TILE_M, worker, n_workers);
    int as = 0;
    uint32_t aphase = 0;
    int t, kb0, kb1;
    griddep_wait();  // C / residual / workspace may still be in use by the predecessor
    while (sch.next(t, kb0, kb1)) {
      int m_blk, n_blk;
      tile_coords(t, num_m_blocks, num_n_blocks, m_blk, n_blk);
      const int row = m_blk * TILE_M + static_cast<int>(mrank) * BLOCK_M + quad * 32 + lane;
      const bool row_ok = row < M;
      constexpr int kHalfChunks = BLOCK_N / 64;  // 32-column chunks per half
      constexpr int kMine = (kSplit2 ? kHalfChunks : BLOCK_N / 32) / 2;
      static_assert(kMine >= 1, "gemm: a chunk for every epilogue warp");
      const int c_lo = (kSplit2 ? static_cast<int>(rank) * kHalfChunks : 0) + upper * kMine, c_hi = c_lo + kMine;
      // this row's residual, a chunk ahead: the first one while the accumulator is still being computed.  A gated unit adds
      // none here (its rows would have N / 2 columns, not the N that are read).
      const __nv_bfloat16* res_row = nullptr;
      if (epi.residual != nullptr && epi.swiglu == 0 && row_ok) {
        const int rr = epi.res_row_mod > 0 ? (row % epi.res_row_mod) : row;
        res_row = epi.residual + static_cast<size_t>(rr) * epi.ld_res;
      }
      uint4 res_next[4];
      auto fetch_residual = [&](int c) {
        const int n0 = n_blk * BLOCK_N + c * 32;
#pragma unroll
        for (int g = 0; g < 4; g += 2) {
          if (res_row == nullptr || c >= c_hi) continue;
          const __nv_bfloat16* src = res_row + n0 + g * 8;
          if (wide_res && n0 + g * 8 + 16 <= N) {
            ldg_v8(src, res_next[g], res_next[g + 1]);
          } else {
            if (n0 + g * 8 < N) res_next[g] = ldg_v4(src);
            if (n0 + g * 8 + 8 < N) res_next[g + 1] = ldg_v4(src + 8);
          }
        }
      };
      fetch_residual(c_lo);
      mbar_wait(&tmem_full[as], aphase);
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + as * BLOCK_N;
      const bool partial = !kSplit2 && ((kb0 != 0) || (kb1 != sch.nkb));
      // split-K pair: park the column half the PEER finalises ([col/4][row] float4 -> conflict-free
      // for the writer here and for the peer's DSMEM reads), then meet the peer at the cluster barrier
      float4* xchg = reinterpret_cast<float4*>(smem_a);  // the pipeline stages are dead by now
      if (kSplit2) {
        const int c_peer = static_cast<int>(1u - rank) * kHalfChunks;
#pragma unroll 1
        for (int c = upper * kMine; c < (upper + 1) * kMine; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(t_row + (c_peer + c) * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int g = 0; g < 8; ++g)
            xchg[(c * 8 + g) * BLOCK_M + quad * 32 + lane] =
                make_float4(__uint_as_float(r[4 * g]), __uint_as_float(r[4 * g + 1]),
                            __uint_as_float(r[4 * g + 2]), __uint_as_float(r[4 * g + 3]));
        }
        cluster_sync_all();  // (warps 0/1 execute the matching barrier after their loops)
      }
      const uint32_t xchg_peer = kSplit2 ? mapa_u32(smem_u32(xchg), 1u - rank) : 0u;
      bool finalize = true;       // apply the epilogue and write C
      bool from_ws = false;       // accumulator comes from the fp32 workspace
      int n_slots = 0;
      const float* slot0 = nullptr;  // first partial slot of this tile, this thread's row
      if (partial) {
        // ---- stream-K partial tile: park the fp32 partial in this segment's own workspace slot
        // (slots are summed later in a fixed order -> deterministic, no atomics on data) ----
        const long total = static_cast<long>(sch.num_tiles) * sch.nkb;
        const long i0 = static_cast<long>(t) * sch.nkb;
        auto cta_of = [&](long i) {
          long g = i * gridDim.x / total;
          while (g + 1 < static_cast<long>(gridDim.x) && total * (g + 1) / gridDim.x <= i) ++g;
          return static_cast<int>(g);
        };
        const int c_first = cta_of(i0);
        n_slots = cta_of(i0 + sch.nkb - 1) - c_first + 1;
        const int my_slot = static_cast<int>(blockIdx.x) - c_first;
        const size_t tile_base = static_cast<size_t>(t) * epi.split_k * (BLOCK_M * BLOCK_N);
        const size_t row_off = static_cast<size_t>(quad * 32 + lane) * BLOCK_N;
        slot0 = epi.splitk_ws + tile_base + row_off;
        float* mine = epi.splitk_ws + tile_base + static_cast<size_t>(my_slot) * (BLOCK_M * BLOCK_N) + row_off;
#pragma unroll 1
        for (int c = c_lo; c < c_hi; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(t_row + c * 32, r);
          tmem_ld_wait();
          if (row_ok) {
#pragma unroll
            for (int g = 0; g < 8; ++g)
              *reinterpret_cast<uint4*>(mine + c * 32 + g * 4) =
                  make_uint4(r[g * 4 + 0], r[g * 4 + 1], r[g * 4 + 2], r[g * 4 + 3]);
          }
        }
        tc_fence_before();
        mbar_arrive(&tmem_empty[as]);  // TMEM stage is free again
        __threadfence();
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");
        if (epi_tid == 0) {
          const int add = kb1 - kb0;
          const int prev = atomicAdd(&epi.splitk_counters[t], add);
          const int last = (prev + add == sch.nkb) ? 1 : 0;
          if (last) epi.splitk_counters[t] = 0;  // self-cleaning
          *last_flag = last;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");
        finalize = (*last_flag != 0);
        from_ws = true;
        if (finalize) __threadfence();
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");  // everyone has read last_flag
      }
      if (finalize) {
#pragma unroll 1
        for (int c = c_lo; c < c_hi; ++c) {
          float v[32];
          uint4 res[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) res[g] = res_next[g];
          fetch_residual(c + 1);
          const int n0 = n_blk * BLOCK_N + c * 32;
          if (!from_ws) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(t_row + c * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
            if (kSplit2) {
              // + the peer's partial of the same columns (two operands: order-independent)
#pragma unroll
              for (int g = 0; g < 8; ++g) {
                const float4 q = ld_dsmem_v4f(
                    xchg_peer + static_cast<uint32_t>(((c - static_cast<int>(rank) * kHalfChunks) * 8 + g) * BLOCK_M + quad * 32 + lane) * 16u);
                v[4 * g + 0] += q.x; v[4 * g + 1] += q.y; v[4 * g + 2] += q.z; v[4 * g + 3] += q.w;
              }
            }
          } else {
            if (n0 >= N) continue;
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0.f;
            if (row_ok) {
              for (int s = 0; s < n_slots; ++s) {  // fixed order: slot 0 (lowest k) first
                const float* wsp = slot0 + static_cast<size_t>(s) * (BLOCK_M * BLOCK_N) + c * 32;
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                  const float4 q = ld_cg_v4(wsp + g * 4);
                  v[g * 4 + 0] += q.x; v[g * 4 + 1] += q.y; v[g * 4 + 2] += q.z; v[g * 4 + 3] += q.w;
                }
              }
            }
          }
          if (n0 >= N) continue;
          if (epi.bias != nullptr) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              if (n0 + g * 8 < N) {
                const uint4 b = ldg_v4(epi.bias + n0 + g * 8);
                v[g * 8 + 0] += bf_lo(b.x);
                v[g * 8 + 1] += bf_hi(b.x);
                v[g * 8 + 2] += bf_lo(b.y);
                v[g * 8 + 3] += bf_hi(b.y);
                v[g * 8 + 4] += bf_lo(b.z);
                v[g * 8 + 5] += bf_hi(b.z);
                v[g * 8 + 6] += bf_lo(b.w);
                v[g * 8 + 7] += bf_hi(b.w);
              }
            }
          }
          if (epi.swiglu == 2) {
            // interleaved (gate, up) column pairs -> 16 outputs of the clamped gated unit, rounded once
            if (row_ok) {
              uint32_t o[8];
#pragma unroll
              for (int j = 0; j < 8; ++j)
                o[j] = pack_bf16(glu_clamp_fast_f(v[4 * j + 0], v[4 * j + 1], epi.act_pos, epi.act_neg),
                                 glu_clamp_fast_f(v[4 * j + 2], v[4 * j + 3], epi.act_pos, epi.act_neg));
              __nv_bfloat16* dst = C + static_cast<size_t>(row) * ldc + (n0 >> 1);
              if (n0 + 16 <= N) stg_v4(dst, make_uint4(o[0], o[1], o[2], o[3]));
              if (n0 + 32 <= N) stg_v4(dst + 8, make_uint4(o[4], o[5], o[6], o[7]));
            }
            continue;
          }
          if (epi.swiglu == 3) {   // gelu_tanh(gate) * up, rounded once
            if (row_ok) {
              uint32_t o[8];
#pragma unroll
              for (int j = 0; j < 8; ++j)
                o[j] = pack_bf16(gelu_tanh_f(v[4 * j + 0]) * v[4 * j + 1], gelu_tanh_f(v[4 * j + 2]) * v[4 * j + 3]);
              __nv_bfloat16* dst = C + static_cast<size_t>(row) * ldc + (n0 >> 1);
              if (n0 + 16 <= N) stg_v4(dst, make_uint4(o[0], o[1], o[2], o[3]));
              if (n0 + 32 <= N) stg_v4(dst + 8, make_uint4(o[4], o[5], o[6], o[7]));
            }
            continue;
          }
          if (epi.swiglu) {
            // interleaved (gate, up) column pairs -> 16 outputs: silu(gate) * up,
            // rounding to bf16 at the points the reference's unfused ops do.
            if (row_ok) {
              uint32_t o[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                float g0 = bf16_round(v[4 * j + 0]), u0 = bf16_round(v[4 * j + 1]);
                float g1 = bf16_round(v[4 * j + 2]), u1 = bf16_round(v[4 * j + 3]);
                float a0 = bf16_round(silu_f(g0)) * u0;
                float a1 = bf16_round(silu_f(g1)) * u1;
                o[j] = pack_bf16(a0, a1);
              }
              __nv_bfloat16* dst = C + static_cast<size_t>(row) * ldc + (n0 >> 1);
              if (n0 + 16 <= N) stg_v4(dst, make_uint4(o[0], o[1], o[2], o[3]));
              if (n0 + 32 <= N) stg_v4(dst + 8, make_uint4(o[4], o[5], o[6], o[7]));
            }
            continue;
          }
          // one loop per activation: its instructions lie together (chosen inside one loop, 32 bodies of all activations
          // did not fit the instruction cache: 13312 x 4304 x 1152 with GELU 317 us)
          auto activate = [&](auto f) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = f(bf16_round(v[j]));
          };
          switch (epi.act) {
            case ACT_NONE: break;
            case ACT_GELU_TANH: activate([](float x) { return gelu_tanh_f(x); }); break;
            case ACT_GELU_ERF: activate([](float x) { return gelu_erf_f(x); }); break;
            case ACT_RELU2: activate([](float x) { return fmaxf(x, 0.f) * fmaxf(x, 0.f); }); break;
            case ACT_XIELU: activate([&](float x) { return xielu_fast_f(x, epi.act_pos, epi.act_neg); }); break;
            default: activate([](float x) { return silu_f(x); });
          }
          if (row_ok) {
            uint4 o[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              float* w = v + g * 8;
              if (res_row != nullptr) {
                const uint4 b = res[g];
                w[0] = bf16_round(w[0]) + bf_lo(b.x);
                w[1] = bf16_round(w[1]) + bf_hi(b.x);
                w[2] = bf16_round(w[2]) + bf_lo(b.y);
                w[3] = bf16_round(w[3]) + bf_hi(b.y);
                w[4] = bf16_round(w[4]) + bf_lo(b.z);
                w[5] = bf16_round(w[5]) + bf_hi(b.z);
                w[6] = bf16_round(w[6]) + bf_lo(b.w);
                w[7] = bf16_round(w[7]) + bf_hi(b.w);
              }
              o[g] = make_uint4(pack_bf16(w[0], w[1]), pack_bf16(w[2], w[3]), pack_bf16(w[4], w[5]), pack_bf16(w[6], w[7]));
            }
            __nv_bfloat16* dst = C + static_cast<size_t>(row) * ldc + n0;
#pragma unroll
            for (int g = 0; g < 4; g += 2) {
              if (wide_c && n0 + g * 8 + 16 <= N) {
                stg_v8(dst + g * 8, o[g], o[g + 1]);
              } else {
                if (n0 + g * 8 < N) stg_v4(dst + g * 8, o[g]);
                if (n0 + g * 8 + 8 < N) stg_v4(dst + g * 8 + 8, o[g + 1]);
              }
            }
          }
        }
      }
      if (!partial) {
        tc_fence_before();
        if (kPair) {
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&tmem_empty[as]), 0));
        } else {
          mbar_arrive(&tmem_empty[as]);
        }
      }
      if (++as == 2) {
        as = 0;
        aphase ^= 1;
      }
    }
  }

  tc_fence_before();
  if (kSplit2 && warp < 2) cluster_sync_all();  // matches the epilogue warps' exchange barrier
  // pair: the leader's MMAs read the peer's shared memory until the end; split-K pair: the peer
  // pulls this CTA's parked partial
  if (kCluster) cluster_sync_all();
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if (kPair) tmem_dealloc_pair<2 * BLOCK_N>(tmem_base);
    else tmem_dealloc<2 * BLOCK_N>(tmem_base);
  }
}

// caller-registered scratch for stream-K partial sums (vila_set_workspace)
struct Workspace {
  void* ptr = nullptr;
  size_t bytes = 0;
};
// one registration per DEVICE (a process may drive several GPUs; the scratch is device memory)
Workspace g_ws_dev[64];
inline Workspace& cur_ws() {
  int d = 0;
  cudaGetDevice(&d);
  return g_ws_dev[(d < 0 || d >= 64) ? 0 : d];
}
#define g_ws cur_ws()
constexpr size_t kCounterBytes = 64 * 1024;  // 16384 tile counters

template <int BLOCK_N, int kStages, int kMode = kModeSingle>
int launch_gemm(const __nv_bfloat16* A, int lda, const __nv_bfloat16* W, int ldw, __nv_bfloat16* C,
                int ldc, int M, int N, int K, GemmEpilogue epi, int force_stream_k,
                cudaStream_t stream) {
  using S = GemmSmem<BLOCK_N, kStages, kMode>;
  constexpr bool kPair = kMode == kModePair;
  constexpr int TILE_M = kPair ? 2 * BLOCK_M : BLOCK_M;
  CUtensorMap ta, tw;
  if (make_tmap_2d_bf16(&ta, A, M, K, lda, BLOCK_M, BLOCK_K, 128)) return 1;
  if (make_tmap_2d_bf16(&tw, W, N, K, ldw, S::kBRows, BLOCK_K, 128)) return 1;
  auto kern = gemm_bf16_tcgen05_kernel<BLOCK_N, kStages, kMode>;
  static PerDeviceOnce attr_once;
  if (attr_once.first()) {
    VB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal));
  }
  const int sms = num_sms();
  const int tiles = ((M + TILE_M - 1) / TILE_M) * ((N + BLOCK_N - 1) / BLOCK_N);
  if (kMode == kModeSplitK2) {
    // one 128 x BLOCK_N tile per CTA pair, half of K each
    if (tiles > sms / 2 || (K + BLOCK_K - 1) / BLOCK_K < 2) {
      set_last_error("gemm: split-K pairs need <= %d tiles and >= 2 k-blocks (tiles=%d)", sms / 2, tiles);
      return 1;
    }
    epi.split_k = 1;
    VB_CUDA(launch_pdl_cluster(kern, dim3(2 * tiles), dim3(kNumThreads), S::kTotal, stream,
                               dim3(2, 1, 1), ta, tw, C, ldc, M, N, K, epi));
    return 0;
  }
  if (kPair) {
    // data-parallel over 256 x BLOCK_N tiles, one tile at a time per CTA pair
    const int pairs = tiles < sms / 2 ? tiles : sms / 2;
    epi.split_k = 1;
    VB_CUDA(launch_pdl_cluster(kern, dim3(2 * pairs), dim3(kNumThreads), S::kTotal, stream,
                               dim3(2, 1, 1), ta, tw, C, ldc, M, N, K, epi));
    return 0;
  }
  const int nkb = (K + BLOCK_K - 1) / BLOCK_K;
  // stream-K when whole tiles would leave SMs idle or produce a ragged last wave
  bool sk = false;
  const long total_it = static_cast<long>(tiles) * nkb;
  const int sk_grid = total_it < sms ? static_cast<int>(total_it) : sms;
  const long ipc = total_it / sk_grid;  // k-iterations per CTA (floor)
  const int max_slots = static_cast<int>((nkb + ipc - 1) / ipc) + 1;
  const size_t need = kCounterBytes + static_cast<size_t>(tiles) * max_slots * BLOCK_M * BLOCK_N * 4;
  const bool ws_ok = g_ws.ptr != nullptr && g_ws.bytes >= need && tiles <= 16384;
  if (force_stream_k >= 0) {
    sk = force_stream_k != 0;
  }
  // (stream-K stays opt-in: on the NVILA shapes the partial-tile fix-up costs more than the SM
  //  under-fill it removes — see profiles/r01_gemm_configs.md)
  if (sk && !ws_ok) {
    set_last_error("gemm: stream-K needs a registered workspace of >= %zu bytes (vila_set_workspace)",
                   need);
    return 1;
  }
  int grid = tiles < sms ? tiles : sms;
  epi.split_k = 1;
  if (sk) {
    grid = sk_grid;
    epi.split_k = max_slots;  // > 1 selects the stream-K schedule; = workspace slots per tile
    epi.splitk_counters = static_cast<int*>(g_ws.ptr);
    epi.splitk_ws = reinterpret_cast<float*>(static_cast<char*>(g_ws.ptr) + kCounterBytes);
  }
  VB_CUDA(launch_pdl(kern, dim3(grid), dim3(kNumThreads), S::kTotal, stream, ta, tw, C, ldc, M, N,
                     K, epi));
  return 0;
}

int check_args(const __nv_bfloat16* A, int lda, const __nv_bfloat16* W, int ldw, __nv_bfloat16* C,
               int ldc, int M, int N, int K, const GemmEpilogue& epi) {
  VB_CHECK(M > 0 && N > 0 && K > 0, "gemm: empty problem M=%d N=%d K=%d", M, N, K);
  VB_CHECK(K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0,
           "gemm: K, lda, ldw must be multiples of 8 (TMA 16-byte strides): K=%d lda=%d ldw=%d", K,
           lda, ldw);
  VB_CHECK(N % 8 == 0 && ldc % 8 == 0, "gemm: N and ldc must be multiples of 8: N=%d ldc=%d", N,
           ldc);
  VB_CHECK((reinterpret_cast<uintptr_t>(A) & 15) == 0 && (reinterpret_cast<uintptr_t>(W) & 15) == 0 &&
               (reinterpret_cast<uintptr_t>(C) & 15) == 0,
           "gemm: pointers must be 16-byte aligned");
  if (epi.swiglu) VB_CHECK(N % 32 == 0, "gemm: swiglu epilogue needs N %% 32 == 0 (N=%d)", N);
  return 0;
}

}  // namespace

// q/k/v projection with RoPE + KV-cache append fused into the epilogue (swap-AB kernel, M <= 384,
// head_dim 128).  Returns -1 when the shape is not covered (caller: plain GEMM + rope_kv_append).
int gemm_qkv_rope_bf16(const __nv_bfloat16* A, int lda, const __nv_bfloat16* W, int ldw, __nv_bfloat16* C,
                       int ldc, int M, int N, int K, const GemmEpilogue& epi, cudaStream_t stream) {
  if (check_args(A, lda, W, ldw, C, ldc, M, N, K, epi)) return 1;
  if (M > 384) return -1;
  return gemm_skinny_bf16(A, lda, W, ldw, C, ldc, M, N, K, epi, 0, stream);
}

void get_workspace(void** ptr, size_t* bytes) {
  *ptr = g_ws.ptr;
  *bytes = g_ws.bytes;
}

int set_workspace(void* ptr, size_t bytes) {
  VB_CHECK(ptr == nullptr || bytes >= kCounterBytes + 1024, "workspace too small (%zu bytes)", bytes);
  VB_CHECK((reinterpret_cast<uintptr_t>(ptr) & 255) == 0, "workspace must be 256-byte aligned");
  g_ws.ptr = ptr;
  g_ws.bytes = ptr ? bytes : 0;
  return 0;
}

int gemm_bf16(const __nv_bfloat16* A, int lda, const __nv_bfloat16* W, int ldw, __nv_bfloat16* C,
              int ldc, int M, int N, int K, const GemmEpilogue& epi, cudaStream_t stream) {
  if (check_args(A, lda, W, ldw, C, ldc, M, N, K, epi)) return 1;
  VB_CHECK(epi.rope_table == nullptr, "gemm: the fused RoPE epilogue is only available through gemm_qkv_rope_bf16");
  // decoded tokens: the weight stream alone
  if (gemm_rows_takes(A, lda, W, ldw, M, N, K, epi)) return gemm_rows(A, lda, W, ldw, C, ldc, M, N, K, epi, stream);
  // The forms of the kernel by what they would take: a start and so much per round of tiles and element of K.  Fitted to one
  // to sixteen rounds of K = 592 .. 18944 (rows 17 .. 2000, outputs 1024 .. 37888).
  //   128 x 128 tiles, K halved over a CTA pair (one round of up to 74)  4.6 + 2.45e-3 K     K = 1024: 7.1   3584: 15
  //   128 x 128 tiles of one CTA                                         3.6 + 4.55e-3 K               8.5         20.5
  //   128 x 256 tiles of one CTA                                         3.4 + 5.80e-3 K               9.4         25
  //   256 x 256 tiles of a CTA pair                                      4.4 + 5.00e-3 K               9.6         22
  // e.g. (us; before: 256-wide tiles from 70 % of the SMs on, pairs from 85 %, halves only for rows that fill their tiles)
  //   800 x 3088 x 1024 11.2 (14.0), 800 x 1024 x 2688 12 (17), 1000 x 2560 x 2048 16 (23), 400 x 2048 x 11008 32 (53)
  const long sms = num_sms(), mb = (M + 127) / 128, mb2 = (M + 255) / 256, nb = (N + 127) / 128, nb2 = (N + 255) / 256;
  const auto rounds = [](long tiles, long at_once) { return static_cast<double>((tiles + at_once - 1) / at_once); };
  const double mbytes = 2e-6 * N * K;
  const double t_half = mb * nb <= sms / 2 && K >= 512 ? 4.6 + 2.45e-3 * K : 1e30;
  const double t_128 = 3.6 + 4.55e-3 * K * rounds(mb * nb, sms);
  const double t_256 = 3.4 + 5.80e-3 * K * rounds(mb * nb2, sms);
  const double t_pair = 4.4 + 5.00e-3 * K * rounds(mb2 * nb2, sms / 2);
  const double t_tiles = fmin(fmin(t_half, t_128), fmin(t_256, t_pair));
  if (M <= 384) {
    // Few tokens: the swap-AB kernel (every weight byte enters an SM once, K split over a cluster) where the weight stream is
    // what counts: 6 us + 0.027 a row + 0.20 a MB, 0.0003 more per row.  With an activation its epilogue counts as well and
    // tiles are ahead: any form up to 16 MB of weights (4304 x 1152 with GELU on 100 rows 8.1, there 14.0), the halves of K
    // always where they are by the two estimates (3584 x 4608 with GELU on 100 | 256 rows 16.4 | 17.5, there
    // 19.8 | 23.2), the others from 0.7 of that estimate on (22016 gated outputs x 2048 on 40 | 279 rows 24 | 34,
    // there 33 | 50).  Theirs is too low for large weights on partly filled row blocks: 37888 x 3584 on 279 rows, the third
    // block with 23 of 128, should be 66 and is 81, there 82 (behind other kernels 90 and 82).
    // Without an activation, where they fill one round (no faster than the weights at 4.8 TB/s): 279 rows x
    // 3088 x 1024 7.9 and 14.2, 200 x 2048 x 2048 9.3 and 14.0, but 3584 x 18944 90 and 46; up to 56 rows (40 rows x 4608 x 3584
    // 12.9 and 10.2, 2560 x 2048 8.7 and 6.8) and for more than 8192 outputs never.
    // Weights of a round of CTA pairs and more (18944 outputs) go to the swap-AB kernel's pairs, whole blocks of 256 in turn: 6 us +
    // 0.04 a row + 0.118 a MB, 0.0002 more per row.  40 / 100 / 279 / 384 rows x 37888 x 3584 gated 43 / 46 / 64 / 81 (one CTA a
    // block 43 / 47 / 71 / 92, tiles 46 / 48 / 82 / 92), 22016 x 2048 20.5 / 21 / 32 / 45 (22 / 24 / 35 / 47 and 22 / 23 / 33 / 34).
    // An activation of every output is more of an epilogue than that estimate knows: with one the tiles stay where they were ahead
    // (GELU, 279 rows x 22016 x 2048 37 and 70, 384 x 27392 x 2048 48 and 90), and up to 256 rows one round of single CTAs too (40 x
    // 18944 x 2048 18 and 23); the others take pairs (279 x 20480 x 3584 80, one CTA a block 111).
    // A projection with a bias and no more onto whole 128-column heads may be the other half of vila_linear_qkv_rope: it
    // stays where that has the same bits (rows that fill their tiles: K halved, as ever).  Without a bias it goes by the
    // time, and the header says so (1024 x 1024 on 279 rows 6.4, there 13.0).
    const bool plain = epi.act == ACT_NONE && epi.swiglu == 0;
    const bool heads = plain && epi.residual == nullptr && epi.bias != nullptr && N % 128 == 0;
    const bool one_round = mb * nb <= sms || mb2 * nb2 <= sms / 2;
    const double t_swap = 6.0 + 0.027 * M + (0.20 + 0.0003 * M) * mbytes;
    const bool whole = (nb + 1) / 2 >= sms / 2 && (epi.act == ACT_NONE || nb > sms || M > 256);
    const double t_whole = 6.0 + 0.04 * M + (0.118 + 0.0002 * M) * mbytes;
    const bool ahead = M > 56 && N <= 8192 && (t_half < 1.05 * t_swap || (one_round && fmax(t_tiles, 4.0 + 0.21 * mbytes) < 0.95 * t_swap));
    const bool tiles = M <= 16 ? false : heads ? t_half < 1e30 && M * 10 >= mb * 128 * 9 : plain ? ahead : whole && epi.swiglu != 0 ? fmax(1.25 * t_tiles, 4.0 + 0.18 * mbytes) < t_whole : mbytes < 16 || t_half < t_swap || t_tiles < 0.7 * t_swap;
    if (!tiles) {
      const int rc = gemm_skinny_bf16(A, lda, W, ldw, C, ldc, M, N, K, epi, whole && M > 16 ? 1 : 0, stream);
      if (rc >= 0) return rc;
    }
    if (heads && t_half < 1e30) return launch_gemm<128, 6, kModeSplitK2>(A, lda, W, ldw, C, ldc, M, N, K, epi, -1, stream);
  }
  if (t_half <= t_tiles) return launch_gemm<128, 6, kModeSplitK2>(A, lda, W, ldw, C, ldc, M, N, K, epi, -1, stream);
  if (N < 128) return launch_gemm<64, 8>(A, lda, W, ldw, C, ldc, M, N, K, epi, -1, stream);
  if (t_pair <= t_tiles) return launch_gemm<256, 6, kModePair>(A, lda, W, ldw, C, ldc, M, N, K, epi, -1, stream);
  if (t_256 <= t_tiles) return launch_gemm<256, 4>(A, lda, W, ldw, C, ldc, M, N, K, epi, -1, stream);
  return launch_gemm<128, 6>(A, lda, W, ldw, C, ldc, M, N, K, epi, -1, stream);
}

// test hook: force a tile configuration (block_n in {64,128,256}; +1000 forces stream-K, +2000 off;
// 3000 / 3001: swap-AB skinny kernel, single CTA / CTA pair; 4128 / 4256: CTA-pair 256 x BLOCK_N
// tiles; 5128: split-K CTA pairs on 128 x 128 tiles)
int gemm_bf16_cfg(int block_n, const __nv_bfloat16* A, int lda, const __nv_bfloat16* W, int ldw,
                  __nv_bfloat16* C, int ldc, int M, int N, int K, const GemmEpilogue& epi,
                  cudaStream_t stream) {
  if (check_args(A, lda, W, ldw, C, ldc, M, N, K, epi)) return 1;
  if (block_n == 4256) return launch_gemm<256, 6, kModePair>(A, lda, W, ldw, C, ldc, M, N, K, epi, -1, stream);
  if (block_n == 4128) return launch_gemm<128, 8, kModePair>(A, lda, W, ldw, C, ldc, M, N, K, epi, -1, stream);
  if (block_n == 5128) return launch_gemm<128, 6, kModeSplitK2>(A, lda, W, ldw, C, ldc, M, N, K, epi, -1, stream);
  if (block_n == 3000 || block_n == 3001) {
    const int rc = gemm_skinny_bf16(A, lda, W, ldw, C, ldc, M, N, K, epi, block_n - 3000, stream);
    if (rc < 0) set_last_error("gemm_bf16_cfg: skinny kernel does not handle M=%d", M);
    return rc < 0 ? 1 : rc;
  }
  int fsk = -1;
  if (block_n >= 2000) {
    fsk = 0;
    block_n -= 2000;
  } else if (block_n >= 1000) {
    fsk = 1;
    block_n -= 1000;
  }
  switch (block_n) {
    case 64: return launch_gemm<64, 8>(A, lda, W, ldw, C, ldc, M, N, K, epi, fsk, stream);
    case 128: return launch_gemm<128, 6>(A, lda, W, ldw, C, ldc, M, N, K, epi, fsk, stream);
    case 256: return launch_gemm<256, 4>(A, lda, W, ldw, C, ldc, M, N, K, epi, fsk, stream);
    default: set_last_error("gemm_bf16_cfg: unsupported block_n %d", block_n); return 1;
  }
}

}  // namespace vb
