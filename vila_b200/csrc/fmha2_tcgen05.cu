// Flash-attention forward for sm_100a: one persistent CTA per SM walks units of one or two 128-row query tiles.
//
//   warps 0 - 7 (and 8 - 15)  softmax of query tile 0 (and 1): eight warps a tile, two threads a row (keys 0 - 63 and 64 - 127
//                             of a block), so that four warps per scheduler hide the latency of the loads, the row maxima and
//                             the exponentials; with one thread a row the exponential unit was busy for 40 % of the time
//   next two warps            TMA: Q tiles, and ONE ring over the sequence K0, V0, K1, V1, ...; rows of O
//   last one or two warps     a tile's tcgen05.mma issuer (one issuer for both tiles was what the kernel waited for)
//   TMEM: scores at 0 and 128 (fp32 128 x 128 each); at 256 / 384 O of tile 0 / 1, or (one tile) the sums of two key
//   blocks and of the next two
//
// The weights go back to TMEM as bf16 over the scores that they come from and are the A operand of the PV product from
// there: in shared memory they cost its port 48 KB a block beside the 64 KB of the operands and the 32 KB that arrive.
//   two tiles: each PV(j) S(j+1) in turn: the tensor pipe works on one tile under the other's softmax
//   one tile:  S(j+1) PV(j): two score buffers, taken in turn; the sums of two blocks join the row's in registers, under the next PV
// The products of one thread execute in order, so scores may follow the weights that a product issued before still reads.
// Descriptors are a base plus constants: made anew for every instruction, the issue alone took 85 clocks of the 64 that a
// product of 128 x 128 x 16 needs.
//
// Bound by the chain of a tile (two tiles: scores 500 clocks at 128 columns, maxima and exponentials 1500, product 500) and by
// the exponential unit (1024 a tile and block).  Before (four softmax warps a tile, weights through shared memory, one CTA a
// pair of tiles): 16 heads of 72 columns, 1024 x 1024, 1 / 4 / 13 images 20.4 / 46.8 / 136.8 us, now 17.0 / 42.1 / 107; causal,
// 28 heads of 128 over 4, 279 / 1024 / 2500 / 8000 / 16470 rows 9.8 / 33 / 91 / 550 / 1955, now 7.8 / 15.0 / 49.7 / 385 / 1530 (1270 TFLOP/s).
// Registers: two tiles have 96 a thread and spill 44 - 68 bytes of their softmax, one tile (168) up to 72, at 128 columns.
//
// S = QK^T in fp32, online softmax in fp32 with exp2, P rounded to bf16 for PV, a lazy (exact) rescale when a row maximum moves
// by more than 2^8.  The tensor core truncates as it accumulates: one tile adds the sums of two blocks, 16 products, by rounded
// additions; two tiles, which have no registers for them, let O grow in TMEM.  Mean signed error of values of one sign, 1024 / 4096 /
// 16384 keys, against the exact result rounded to bf16: -2.9 / -3.5 / -2.2e-6 (-2.7 / -3.3 / -2.1e-6 a block at a time) and -4.3 / -16 /
// -78e-6.  With O in TMEM one tile was 5 % faster at 128 columns (1024 rows 14.2; a block at a time 15.2), 3 % at 72.  D = 65 .. 96 zero-padded by TMA fill (SW64
// chunks of 32 columns; up to 80 columns products stop there), D = 64 and 128 as SW128 chunks, V the MN-major B operand.
//
// Replaces flash_attn_func in SiglipFlashAttention2 (modeling_siglip.py:583-585, non-causal, scale 72^-0.5) and HF
// _flash_attention_forward for Qwen2 (modeling_qwen2.py:191-310; causal GQA).
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace vb {
namespace {

constexpr int BQ = 128;
constexpr int BKV = 128;

template <int DP, int CW, int TILES>
struct Shape {
  static constexpr int kChunks = (DP + CW - 1) / CW;
  static constexpr int kChunkBytes = 128 * CW * 2;
  static constexpr int kTileBytes = kChunks * kChunkBytes;  // one 128-row Q / K / V tile
  static constexpr uint32_t kLayout = CW == 64 ? kLayoutSW128 : kLayoutSW64;
  static constexpr int kSwizzleBytes = CW * 2;
  static constexpr int kSBO = 8 * CW * 2;
  static constexpr int kQ = TILES == 2 && DP == 128 ? 1 : 2;   // Q buffers of a tile: the next unit's arrives under this one's products
  static constexpr int kRing = DP == 128 ? 4 : 5;           // K / V slots
  static constexpr int kSoftmaxWarps = 8 * TILES;
  static constexpr int kProducer = kSoftmaxWarps, kStore = kProducer + 1, kMma = kStore + 1;   // warps
  static constexpr int kThreads = 32 * (kMma + TILES);
  static constexpr int kHalf = DP / 2;                      // O columns of a thread
  static constexpr int kNumBars = 2 * kRing + 6 * kQ + 10;
  static constexpr int kSmem = (TILES * kQ + kRing) * kTileBytes + TILES * 2 * 2 * BQ * 4 + kNumBars * 8 + 16 + 1024;
};

__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 3-input maximum: half the instructions
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// a chunk of O from shared memory; the tensor's ends are not written past
__device__ __forceinline__ void store_chunk(const CUtensorMap* m, uint32_t src, int c0, int h, int row, int b) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(src), "r"(c0), "r"(h), "r"(row), "r"(b)
               : "memory");
}

struct Args {
  const int32_t* page_table;
  int page_table_stride;
  int Sq, Sk, Hq, Hkv, D, causal, paged, B;
  int units;                  // query units (of TILES tiles) of a sequence and head
  float scale_log2;
};

// ADD: one tile whose rows have more than two key blocks; what two blocks sum to stays in TMEM otherwise
template <int DP, int CW, int TILES, bool ADD>
__global__ void __launch_bounds__(Shape<DP, CW, TILES>::kThreads, 1)
fmha_pipe_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o, const Args a, const WaitLimit limit, volatile unsigned int* failed) {
  using C = Shape<DP, CW, TILES>;
  constexpr int R = C::kRing;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* q_s = smem;                                  // [tile][buffer]
  uint8_t* ring_s = q_s + TILES * C::kQ * C::kTileBytes;
  float* xm = reinterpret_cast<float*>(ring_s + R * C::kTileBytes);   // [tile][half][row] maxima, then sums
  float* xl = xm + TILES * 2 * BQ;
  uint64_t* r_full = reinterpret_cast<uint64_t*>(xl + TILES * 2 * BQ);   // [R]
  uint64_t* r_empty = r_full + R;                       // [R]
  uint64_t* q_full = r_empty + R;                       // [tile][buffer]
  uint64_t* q_empty = q_full + 2 * C::kQ;               // [tile][buffer]
  uint64_t* s_full = q_empty + 2 * C::kQ;               // [2]: by score buffer
  uint64_t* p_full = s_full + 2;                        // [2]
  uint64_t* o_full = p_full + 2;                        // [2]: by tile, or (one tile) of even and odd blocks
  uint64_t* o_free = o_full + 2;                        // [2]
  uint64_t* o_ready = o_free + 2;                       // [tile][buffer]: rows stand in the Q buffer
  uint64_t* fin = o_ready + 2 * C::kQ;                  // [2]
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(fin + 2);
  volatile int* gave_up = reinterpret_cast<int*>(tmem_ptr + 1);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x) >> 5, 0);   // known to be the same for a warp
  const int lane = threadIdx.x & 31;
  const int off = a.Sk - a.Sq;
  const int heads = a.Hq * a.B;
  const int total = a.units * heads;

  if (threadIdx.x == 0) {
    for (int i = 0; i < R; ++i) {
      mbar_init(&r_full[i], 1);
      mbar_init(&r_empty[i], TILES);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 8);
      mbar_init(&o_full[i], 1);
      mbar_init(&o_free[i], 8);
    }
    for (int i = 0; i < 2 * C::kQ; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&o_ready[i], 8);
    }
    mbar_init(&fin[0], 1);
    mbar_init(&fin[1], 1);
    *gave_up = 0;
    fence_barrier_init();
  }
  if (warp == C::kMma) tmem_alloc<512>(tmem_ptr);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  griddep_launch_dependents();
  griddep_wait();

  // The CTA's units in turn.  Causal: the longest first, and back and forth over the CTAs from round to round, so that each
  // gets about the same; otherwise the units of a head next to each other.
  struct Unit {
    int u, h, b, n[2], nmax;
  };
  auto unit = [&](int round, Unit& w) {
    const int g = static_cast<int>(gridDim.x), c = static_cast<int>(blockIdx.x);
    const int i = round * g + ((round & 1) ? g - 1 - c : c);
    if (i >= total) return false;
    int hb;
    if (a.causal) {
      w.u = a.units - 1 - i / heads;
      hb = i % heads;
    } else {
      w.u = i % a.units;
      hb = i / a.units;
    }
    w.b = hb / a.Hq;
    w.h = hb - w.b * a.Hq;
    w.nmax = 0;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int q0 = (w.u * TILES + t) * BQ;
      int n = 0;
      if (t < TILES && q0 < a.Sq) {
        int kv_end = a.Sk;
        if (a.causal) kv_end = min(a.Sk, min(q0 + BQ, a.Sq) + off);
        n = (kv_end + BKV - 1) / BKV;
      }
      w.n[t] = n;
      w.nmax = max(w.nmax, n);
    }
    return true;
  };
  const int rounds = (total + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  int items = 0, qn[2] = {0, 0};   // producer: tiles asked for, of the ring and of the queries

  // The producer and the issuers run as whole warps whose values are the same in all lanes (they stay in uniform registers) and
  // elect a lane for what is issued.
  if (limit.quits == (warp == C::kProducer ? 0 : warp == C::kStore ? 1 : warp >= C::kMma ? 2 : 3)) *gave_up = 1;
  auto wait = [&](uint64_t* bar, int phase) { return __all_sync(0xffffffffu, mbar_wait_limited(bar, phase & 1, gave_up, limit.tries)); };
  if (warp == C::kProducer) {
    // ===================== TMA producer =====================
    if (elect_one()) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
    }
    int slot = 0, ph = 1;
    bool ok = limit.quits != 0;
    Unit w;
    for (int r = 0; ok && r < rounds; ++r) {
      if (!unit(r, w)) continue;
      const int hk = w.h / (a.Hq / a.Hkv);
      auto load = [&](const CUtensorMap* tm, int tok, int page) {
        ok = wait(&r_empty[slot], ph);
        if (!ok) return;
        if (elect_one()) {
          mbar_arrive_expect_tx(&r_full[slot], C::kTileBytes);
#pragma unroll
          for (int c = 0; c < C::kChunks; ++c)
            tma_load_4d(ring_s + slot * C::kTileBytes + c * C::kChunkBytes, tm, &r_full[slot], c * CW, hk, tok, page);
        }
        ++items;
        if (++slot == R) {
          slot = 0;
          ph ^= 1;
        }
      };
      for (int j = 0; ok && j < w.nmax; ++j) {
        int tok = 0, page = 0;
        if (a.paged) page = a.page_table ? a.page_table[w.b * a.page_table_stride + j] : j;
        else tok = w.b * a.Sk + j * BKV;
        load(&tm_k, tok, page);
        if (j == 0) {   // behind the first keys: those wait for a slot only, the queries for the last unit's scores
#pragma unroll
          for (int t = 0; t < TILES; ++t) {
            if (w.n[t] == 0 || !ok) continue;
            const int qb = qn[t] % C::kQ, at = t * C::kQ + qb;
            ok = wait(&q_empty[at], qn[t] / C::kQ + 1);
            if (!ok) continue;
            if (elect_one()) {
              mbar_arrive_expect_tx(&q_full[at], C::kTileBytes);
#pragma unroll
              for (int c = 0; c < C::kChunks; ++c)
                tma_load_4d(q_s + at * C::kTileBytes + c * C::kChunkBytes, &tm_q, &q_full[at], c * CW, w.h,
                            w.b * a.Sq + (w.u * TILES + t) * BQ, 0);
            }
            ++qn[t];
          }
        }
        if (ok) load(&tm_v, tok, page);
      }
    }
  } else if (warp == C::kStore) {
    // ===================== rows of O =====================
    int un[2] = {0, 0};
    bool ok = limit.quits != 1;
    Unit w;
    for (int r = 0; ok && r < rounds; ++r) {
      if (!unit(r, w)) continue;
#pragma unroll
      for (int t = 0; t < TILES; ++t) {
        if (w.n[t] == 0 || !ok) continue;
        const int at = t * C::kQ + un[t] % C::kQ;
        ok = wait(&o_ready[at], un[t] / C::kQ);
        if (!ok) continue;
        if (elect_one()) {
#pragma unroll
          for (int c = 0; c < C::kChunks; ++c)
            if (c * CW < a.D) store_chunk(&tm_o, smem_u32(q_s) + at * C::kTileBytes + c * C::kChunkBytes, c * CW, w.h, (w.u * TILES + t) * BQ, w.b);
          asm volatile("cp.async.bulk.commit_group;\ncp.async.bulk.wait_group.read 0;" ::: "memory");
          mbar_arrive(&q_empty[at]);
        }
        __syncwarp();
        ++un[t];
      }
    }
  } else if (warp >= C::kMma) {
    // ===================== MMA issuer of tile t =====================
    const int t = TILES == 2 ? warp - C::kMma : 0;
    constexpr uint32_t idesc_s = make_idesc_bf16(BQ, BKV, 0, 0);
    constexpr uint32_t idesc_o = make_idesc_bf16(BQ, DP, 0, 1);
    constexpr int kSteps = CW / 16, kTile16 = C::kTileBytes >> 4;
    const uint64_t qd0 = make_smem_desc(smem_u32(q_s) + t * C::kQ * C::kTileBytes, 16, C::kSBO, C::kLayout);
    const uint64_t kd0 = make_smem_desc(smem_u32(ring_s), 16, C::kSBO, C::kLayout);
    const uint64_t vd0 = make_smem_desc(smem_u32(ring_s), C::kChunkBytes, C::kSBO, C::kLayout);
    const uint32_t o_tmem = tmem_base + 256 + t * 128;
    bool ok = limit.quits != 2;
    int slot = 0, ph = 0, g = 0, units = 0, pairs = 0;   // ring; blocks, units and (one tile) pairs of blocks of the tile so far
    auto advance = [&]() {
      if (++slot == R) {
        slot = 0;
        ph ^= 1;
      }
    };
    // scores of block n against the K in `slot`
    auto issue_s = [&](int n, int slot_k) {
      tc_fence_after();
      const int sb = TILES == 2 ? t : n & 1, qb = units % C::kQ;
      if (elect_one()) {
        const uint64_t qd = qd0 + static_cast<uint32_t>(qb * kTile16), kd = kd0 + static_cast<uint32_t>(slot_k * kTile16);
        const uint32_t d = tmem_base + sb * BKV;
#pragma unroll
        for (int k = 0; k < DP / 16; ++k) {
          const int o = (k / kSteps) * (C::kChunkBytes >> 4) + (k % kSteps) * 2;
          umma_f16(d, qd + o, kd + o, idesc_s, k != 0 ? 1u : 0u);
        }
        umma_commit(&s_full[sb]);
        umma_commit(&r_empty[slot_k]);
      }
      __syncwarp();
    };
    auto issue_pv = [&](int n, int slot_v, bool first) {
      tc_fence_after();
      const int sb = TILES == 2 ? t : n & 1;
      if (elect_one()) {
        const uint64_t vd = vd0 + static_cast<uint32_t>(slot_v * kTile16);
        const uint32_t p = tmem_base + sb * BKV;
#pragma unroll
        for (int k = 0; k < BKV / 16; ++k)   // weights of keys 16 k ..: 8 columns, each half's from its own scores' first on
          umma_f16_ts(o_tmem + (TILES == 2 ? 0 : (pairs & 1) * 128), p + (k >> 2) * 64 + (k & 3) * 8, vd + k * (16 * CW * 2 >> 4), idesc_o,
                      k != 0 || !first ? 1u : 0u);
        umma_commit(&o_full[sb]);
        umma_commit(&r_empty[slot_v]);
      }
      __syncwarp();
    };
    Unit w;
    for (int r = 0; ok && r < rounds; ++r) {
      if (!unit(r, w)) continue;
      const int n = TILES == 2 && t == 1 ? w.n[1] : w.n[0];
      ok = wait(&r_full[slot], ph);
      if (ok && n > 0) {
        ok = wait(&q_full[t * C::kQ + units % C::kQ], units / C::kQ);
        if (ok) issue_s(g, slot);
      }
      if (!ok) break;
      if (n == 0 && elect_one()) mbar_arrive(&r_empty[slot]);
      advance();
      for (int j = 0; j < n; ++j, ++g) {
        const int slot_v = slot, ph_v = ph;
        advance();
        const int slot_k = slot, ph_k = ph;
        const bool more = j + 1 < n;
        if (TILES == 1 && more) {
          ok = wait(&r_full[slot_k], ph_k);
          if (!ok) break;
          issue_s(g + 1, slot_k);
        }
        // the weights: also orders this PV after any rescale of block j and (one tile) after the sums that were here have been taken in
        ok = wait(&r_full[slot_v], ph_v) && (TILES == 1 || ((!more || wait(&r_full[slot_k], ph_k)) && (j > 0 || wait(&o_free[t], units + 1)))) &&
             wait(&p_full[TILES == 2 ? t : g & 1], TILES == 2 ? g : g >> 1);
        if (!ok) break;
        issue_pv(g, slot_v, TILES == 1 ? (j & 1) == 0 : j == 0);
        if (TILES == 1 && ((j & 1) != 0 || !more)) ++pairs;
        if (TILES == 2 && more) issue_s(g + 1, slot_k);
        if (more) advance();
      }
      // blocks that only the other tile sees: K and V from block n on (the first K is counted above)
      for (int i = n == 0 ? 1 : 2 * n; ok && i < 2 * w.nmax; ++i) {
        ok = wait(&r_full[slot], ph);
        if (ok && elect_one()) mbar_arrive(&r_empty[slot]);
        advance();
      }
      if (!ok) break;
      units += n > 0;
    }
  } else {
    // ===================== softmax =====================
    const int t = TILES == 2 ? warp >> 3 : 0, half = (warp >> 2) & 1, quad = warp & 3;
    const int row = quad * 32 + lane, id = 1 + t * 4 + quad;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t o_addr = lane_addr + 256 + t * 128 + half * C::kHalf;
    float *xm_t = xm + t * 2 * BQ + row, *xl_t = xl + t * 2 * BQ + row;
    int g = 0, units = 0;   // blocks and units of the tile so far
    // One tile: a row's sums, to which those of two blocks, up to block b, are added from TMEM under the next block's product
    uint32_t o[C::kHalf];
    int pairs = 0;          // that have been taken in, or (one tile, not ADD) units before this one
    auto take = [&](int b, auto columns) {   // of so many at a time
      constexpr int N = decltype(columns)::value;
      wait(&o_full[b & 1], b >> 1);
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < C::kHalf; c += N) {
        uint32_t x[N];
        const uint32_t from = o_addr + (pairs & 1) * 128 + c;
#pragma unroll
        for (int i = 0; i + 32 <= N; i += 32) tmem_ld_32x32b_x32(from + i, x + i);
#pragma unroll
        for (int i = N / 32 * 32; i < N; i += 8) tmem_ld_32x32b_x8(from + i, x + i);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < N; i += 2) {
          float y0 = __uint_as_float(o[c + i]), y1 = __uint_as_float(o[c + i + 1]);
          fadd2(y0, y1, __uint_as_float(x[i]), __uint_as_float(x[i + 1]));
          o[c + i] = __float_as_uint(y0);
          o[c + i + 1] = __float_as_uint(y1);
        }
      }
      ++pairs;
    };
    using Few = std::integral_constant<int, 8>;
    using All = std::integral_constant<int, C::kHalf>;
    Unit w;
    for (int r = 0; r < rounds; ++r) {
      if (!unit(r, w) || w.n[t] == 0) continue;
      if (ADD) {
#pragma unroll
        for (int i = 0; i < C::kHalf; ++i) o[i] = 0u;
      }
      const int n = w.n[t], q0 = (w.u * TILES + t) * BQ;
      const int kv_lim = a.causal ? min(a.Sk - 1, q0 + row + off) : a.Sk - 1;
      // Two tiles: O accumulates in TMEM across KV blocks.  Each row keeps a reference maximum m_ref; the accumulator is rescaled
      // only when a row's maximum exceeds m_ref by more than 2^8 (exact: P, l and O all use the same m_ref, the final division
      // by l cancels it).  The two warps of a row decide together.
      float m_ref = 0.f, l = 0.f;
      for (int j = 0; j < n; ++j, ++g) {
        const int sb = TILES == 2 ? t : g & 1;
        const uint32_t s_addr = lane_addr + sb * BKV + half * 64;
        wait(&s_full[sb], TILES == 2 ? g : g >> 1);
        tc_fence_after();
        const int kv0 = j * BKV + half * 64;
        const bool need_mask = (kv0 + 64 > a.Sk) || (a.causal && (kv0 + 63 > q0 + off));
        uint32_t s[64];
        tmem_ld_32x32b_x32(s_addr, s);
        tmem_ld_32x32b_x32(s_addr + 32, s + 32);
        tmem_ld_wait();
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (kv0 + i > kv_lim) s[i] = 0xff800000u;
        }
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};   // short chains
#pragma unroll
        for (int i = 0; i < 64; i += 8)
#pragma unroll
          for (int q = 0; q < 4; ++q) m4[q] = fmax3(m4[q], __uint_as_float(s[i + 2 * q]), __uint_as_float(s[i + 2 * q + 1]));
        float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * a.scale_log2;
        bool taken = !ADD || j == 0 || (j & 1) != 0;   // no two blocks' sums are complete and still in TMEM
        if (pair_any(id, j == 0 || mx > m_ref + 8.0f)) {
          xm_t[half * BQ] = mx;
          pair_sync(id);
          mx = fmaxf(mx, xm_t[(half ^ 1) * BQ]);
          if (j == 0) {
            m_ref = mx == -INFINITY ? 0.f : mx;
          } else {
            const float m_new = mx > m_ref + 8.0f ? mx : m_ref;
            const float alpha = ex2f(m_ref - m_new);                      // 1 for rows that keep their reference
            // rare: few registers rather than few round trips
            if (ADD && !taken) {
              take(g - 1, Few());
              taken = true;
            } else {
              // PV(j - 1) has landed
              if (TILES == 1) wait(&o_full[(g - 1) & 1], (g - 1) >> 1);
              else wait(&o_full[t], g - 1);
              tc_fence_after();
              const uint32_t sums = o_addr + (TILES == 1 ? (pairs & 1) * 128 : 0);
#pragma unroll 1
              for (int c = 0; c < C::kHalf / 8; ++c) {
                uint32_t o8[8];
                tmem_ld_32x32b_x8(sums + c * 8, o8);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; ++i) o8[i] = __float_as_uint(__uint_as_float(o8[i]) * alpha);
                tmem_st_32x32b_x8(sums + c * 8, o8);
              }
            }
            if (ADD) {
#pragma unroll
              for (int i = 0; i < C::kHalf; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            }
            l *= alpha;
            m_ref = m_new;
          }
        }
        float l4[4] = {0.f, 0.f, 0.f, 0.f};
        const float neg_m = -m_ref;
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
          float e[4];
          ffma2(e[0], e[1], __uint_as_float(s[i]), __uint_as_float(s[i + 1]), a.scale_log2, neg_m);
          ffma2(e[2], e[3], __uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]), a.scale_log2, neg_m);
#pragma unroll
          for (int q = 0; q < 4; ++q) e[q] = ex2f(e[q]);
          fadd2(l4[0], l4[1], e[0], e[1]);
          fadd2(l4[2], l4[3], e[2], e[3]);
          s[i / 2] = pack_bf16(e[0], e[1]);
          s[i / 2 + 1] = pack_bf16(e[2], e[3]);
        }
        tmem_st_32x32b_x32(s_addr, s);
        l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[sb]);
        if constexpr (ADD) {
          if (!taken) take(g - 1, All());
        }
      }
      // ---- O / l
      xl_t[half * BQ] = l;
      pair_sync(id);
      l += xl_t[(half ^ 1) * BQ];
      if constexpr (ADD) {
        take(g - 1, All());
      } else {
        if (TILES == 1) wait(&o_full[(g - 1) & 1], (g - 1) >> 1);
        else wait(&o_full[t], g - 1);
        tc_fence_after();
        const uint32_t sums = o_addr + (TILES == 1 ? (pairs++ & 1) * 128 : 0);
#pragma unroll
        for (int c = 0; c < C::kHalf / 8; ++c) tmem_ld_32x32b_x8(sums + c * 8, o + c * 8);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (TILES == 2 && lane == 0) mbar_arrive(&o_free[t]);
      }
      // Rows go out by TMA from the unit's Q tile, which its last scores have left: 16-byte stores of a row per lane held the
      // load / store unit for 2500 clocks a unit, and the softmax warps that issued the copies waited as long for TMA's queue.
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const int qb = t * C::kQ + units % C::kQ;
      const uint32_t out = smem_u32(q_s) + qb * C::kTileBytes + row * (CW * 2);
      const int swz = CW == 64 ? row & 7 : (row >> 1) & 3;
#pragma unroll
      for (int c = 0; c < C::kHalf / 8; ++c) {
        const int col = half * C::kHalf + c * 8, piece = (col % CW) / 8;
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(out + (col / CW) * C::kChunkBytes + ((piece ^ swz) << 4)),
                     "r"(pack_bf16(__uint_as_float(o[c * 8 + 0]) * inv, __uint_as_float(o[c * 8 + 1]) * inv)),
                     "r"(pack_bf16(__uint_as_float(o[c * 8 + 2]) * inv, __uint_as_float(o[c * 8 + 3]) * inv)),
                     "r"(pack_bf16(__uint_as_float(o[c * 8 + 4]) * inv, __uint_as_float(o[c * 8 + 5]) * inv)),
                     "r"(pack_bf16(__uint_as_float(o[c * 8 + 6]) * inv, __uint_as_float(o[c * 8 + 7]) * inv))
                     : "memory");
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&o_ready[qb]);
      ++units;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*gave_up) {
    // Copies and products in flight end before shared memory and TMEM go, also those of warps whose own waits all held: a
    // producer or an issuer that was through with its work before another warp gave up.
    if (warp == C::kProducer) {
      for (int k = max(0, items - R); k < items; ++k) mbar_drain(&r_full[k % R], (k / R) & 1);
#pragma unroll
      for (int t = 0; t < TILES; ++t)
        for (int k = max(0, qn[t] - C::kQ); k < qn[t]; ++k) mbar_drain(&q_full[t * C::kQ + k % C::kQ], (k / C::kQ) & 1);
    } else if (warp >= C::kMma) {
      uint64_t* done = &fin[warp - C::kMma];
      if (elect_one()) umma_commit(done);
      mbar_drain(done, 0);
    }
    __syncthreads();
  }
  if (warp == C::kMma) {
    tc_fence_after();
    tmem_dealloc<512>(tmem_base);
  }
  if (threadIdx.x == 0 && *gave_up) {
    *failed = 1u;
    __threadfence_system();
  }
}

template <int DP, int CW, int TILES, bool ADD>
int launch(const FmhaParams& p, cudaStream_t stream, int tries) {
  using C = Shape<DP, CW, TILES>;
  static_assert(C::kSmem <= 227 * 1024, "fmha: shared memory");
  volatile unsigned int* failed = failed_word();
  VB_CHECK(failed != nullptr, "fmha: no pinned host memory for the status word");
  CUtensorMap tq, tk, tv, to;
  {
    uint64_t dims[4] = {(uint64_t)p.D, (uint64_t)p.Hq, (uint64_t)p.B * p.Sq, 1};
    uint64_t str[3] = {(uint64_t)p.q_head_stride, (uint64_t)p.q_tok_stride,
                       (uint64_t)p.q_tok_stride * p.B * p.Sq};
    uint32_t box[4] = {CW, 1, BQ, 1};
    if (make_tmap_nd_bf16(&tq, p.q, 4, dims, str, box, C::kSwizzleBytes)) return 1;
  }
  {
    uint64_t dims[4] = {(uint64_t)p.D, (uint64_t)p.Hq, (uint64_t)p.Sq, (uint64_t)p.B};
    uint64_t str[3] = {(uint64_t)p.o_head_stride, (uint64_t)p.o_tok_stride, (uint64_t)p.o_tok_stride * p.Sq};
    uint32_t box[4] = {CW, 1, BQ, 1};
    if (make_tmap_nd_bf16(&to, p.o, 4, dims, str, box, C::kSwizzleBytes)) return 1;
  }
  const bool paged = p.kv_page_stride != 0;
  {
    uint64_t dims[4], str[3];
    if (paged) {
      dims[0] = p.D; dims[1] = p.Hkv; dims[2] = BKV; dims[3] = p.kv_num_pages;
      str[0] = p.kv_head_stride; str[1] = p.kv_tok_stride; str[2] = p.kv_page_stride;
    } else {
      dims[0] = p.D; dims[1] = p.Hkv; dims[2] = (uint64_t)p.B * p.Sk; dims[3] = 1;
      str[0] = p.kv_head_stride; str[1] = p.kv_tok_stride;
      str[2] = (uint64_t)p.kv_tok_stride * p.B * p.Sk;
    }
    uint32_t box[4] = {CW, 1, BKV, 1};
    if (make_tmap_nd_bf16(&tk, p.k, 4, dims, str, box, C::kSwizzleBytes)) return 1;
    if (make_tmap_nd_bf16(&tv, p.v, 4, dims, str, box, C::kSwizzleBytes)) return 1;
  }
  Args a;
  a.page_table = p.page_table;
  a.page_table_stride = p.page_table_stride;
  a.Sq = p.Sq; a.Sk = p.Sk; a.Hq = p.Hq; a.Hkv = p.Hkv; a.D = p.D; a.B = p.B;
  a.causal = p.causal;
  a.paged = paged ? 1 : 0;
  a.units = (p.Sq + TILES * BQ - 1) / (TILES * BQ);
  a.scale_log2 = p.scale * 1.4426950408889634f;
  auto kern = fmha_pipe_kernel<DP, CW, TILES, ADD>;
  static PerDeviceOnce attr_once;
  if (attr_once.first()) {
    VB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem));
  }
  const long total = static_cast<long>(a.units) * p.Hq * p.B;
  VB_CHECK(total < (1L << 30), "fmha: too many query tiles");
  const int grid = static_cast<int>(total < num_sms() ? total : num_sms());
  VB_CUDA(launch_pdl(kern, dim3(grid), dim3(C::kThreads), C::kSmem, stream, tq, tk, tv, to, a, wait_limit(tries), failed));
  return 0;
}

template <int DP, int CW>
int launch_tiles(const FmhaParams& p, int tiles, cudaStream_t stream, int tries) {
  if (tiles == 2) return launch<DP, CW, 2, false>(p, stream, tries);
  // up to two key blocks there is nothing to add, and the registers for it cost 0.4 of 5.8 us (64 rows, 128 columns); the same bits
  return p.Sk > 2 * BKV ? launch<DP, CW, 1, true>(p, stream, tries) : launch<DP, CW, 1, false>(p, stream, tries);
}

}  // namespace

int fmha_prefill(const FmhaParams& p, cudaStream_t stream) { return fmha_prefill_cfg(0, p, stream); }

// variant: 0 by size, 1 one query tile at a time, 2 (3, 4) two; tries: of every wait (tests, see wait_limit), -1 the kernel's limit
int fmha_prefill_cfg(int variant, const FmhaParams& p, cudaStream_t stream, int tries) {
  VB_CHECK(variant >= 0 && variant <= 4, "fmha: unknown variant %d", variant);
  VB_CHECK(p.B > 0 && p.Sq > 0 && p.Sk > 0, "fmha: empty problem");
  VB_CHECK(p.Hq % p.Hkv == 0, "fmha: Hq (%d) must be a multiple of Hkv (%d)", p.Hq, p.Hkv);
  VB_CHECK(p.D % 8 == 0, "fmha: head dim must be a multiple of 8 (got %d)", p.D);
  VB_CHECK(p.q_tok_stride % 8 == 0 && p.q_head_stride % 8 == 0 && p.kv_tok_stride % 8 == 0 &&
               p.kv_head_stride % 8 == 0 && p.o_tok_stride % 8 == 0 && p.o_head_stride % 8 == 0,
           "fmha: strides must be multiples of 8 elements (16 bytes)");
  VB_CHECK(!p.causal || p.Sk >= p.Sq, "fmha: causal needs Sk >= Sq");
  if (wait_status()) return 1;   // an earlier launch gave up: nothing is built on its output
  // Two tiles at a time take 1.6 times as long per key block as one (13 x 16 heads of 1024 keys, head size 72: 23.5 and 14.5
  // us a round of units).  Key blocks per CTA: whole rounds of equal units, or (causal, dealt evenly) the mean, but no less
  // than the longest unit.  1 / 2 / 3 / 4 / 7 / 13 images: one 17, 31, 39, 56, 84, 167 us, two 25, 26, 46, 46, 76, 121; causal,
  // 28 heads of 128, 600 / 1024 / 1500 / 2500 / 8000 rows: 10.8, 15.0, 27, 55, 445 and 14, 21, 29, 50, 385.
  // More than 2560 keys keep rounded sums (see above) where two tiles would not fill the SMs once, and at 64 columns; up to there
  // the two forms' errors are the same (rms 1.7958e-3 at 1024 keys, both; 1.7676e-3 and 1.7694e-3 at 16384).
  const int q_tiles = (p.Sq + BQ - 1) / BQ;
  auto blocks = [&](int per) {
    const int units = (q_tiles + per - 1) / per;
    const long heads = static_cast<long>(p.Hq) * p.B, sms = num_sms();
    if (!p.causal) return (units * heads + sms - 1) / sms * ((p.Sk + BKV - 1) / BKV);
    long sum = 0, most = 0;
    for (int u = 1; u <= units; ++u) {
      most = (min(p.Sk, min(u * per * BQ, p.Sq) + p.Sk - p.Sq) + BKV - 1) / BKV;
      sum += most;
    }
    return max(most, (sum * heads + sms - 1) / sms);
  };
  const bool grow = p.Sk <= 2560 || (p.D > 64 && static_cast<long>((q_tiles + 1) / 2) * p.Hq * p.B >= num_sms());
  const int tiles = variant == 0 ? (grow && 8 * blocks(2) < 5 * blocks(1) ? 2 : 1) : variant == 1 || q_tiles == 1 ? 1 : 2;
  if (p.D == 128) return launch_tiles<128, 64>(p, tiles, stream, tries);
  if (p.D > 80 && p.D <= 96) return launch_tiles<96, 32>(p, tiles, stream, tries);
  if (p.D > 64 && p.D <= 80) return launch_tiles<80, 32>(p, tiles, stream, tries);
  VB_CHECK(variant < 2 || p.D == 64, "fmha: the two-tile kernel does not cover head dim %d", p.D);
  if (p.D == 64) return launch_tiles<64, 64>(p, tiles, stream, tries);
  set_last_error("fmha: unsupported head dim %d (supported: 64, 65..96, 128)", p.D);
  return 1;
}

}  // namespace vb
