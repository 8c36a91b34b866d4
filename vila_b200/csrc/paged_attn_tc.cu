// vila_paged_attention for prompt portions over a bf16 pool, 128 key and value columns, on tcgen05 in fp32 precision.
//
// What is computed is paged_attn_mma.cu's: queries and weights in three bf16 parts, whose products with bf16 keys and values are
// exact; a score in two sums, of the first 64 columns' first parts and of the rest, small parts first; a block's 64 keys in fresh
// sums of a value column, the parts in ascending size, which join the row's by rounded additions (the tensor core truncates, tcgen05
// as mma.sync does), in registers for up to four blocks, which then join those before them in TMEM (a quarter of the roundings
// of a long sum); rows that come out infinite or NaN again, key by key.  A row's numbers depend on its own keys only, by blocks at
// multiples of 64.
//
// A CTA: 128 rows = 8 groups of a 16-row tile and one of the query heads that share the key / value head.
//   warps 0 - 7    queries; softmax, two threads a row (keys 0 - 31 and 32 - 63 of a block); the row's sums in their registers (64
//                  columns each).  Those whose 32 rows belong to no tile only count the blocks.
//   warps 8, 9     keys and values by cp.async into a ring of 64-key blocks (K-major and MN-major operands, 128-byte swizzle); the
//                  first ones come while the queries do
//   warp 10        tcgen05.mma issuer, TMEM
// (three warps a scheduler: the softmax needs 168 registers a thread)
// TMEM: two score buffers of 128 columns (the two sums of 64 keys), over which the weights' parts come back as the A operand; 128
// columns for a block's sums and 128 for the rows'.  S(j + 1) is computed under block j's softmax, PV(j) under block j + 1's, whose
// end takes it in before PV(j + 1) may begin.
//
// A block takes 2800 clocks without the cap: scores 1200 (24 products of 64 keys, 50 clocks each), sums 800, the issuer's turns; 3400
// with it (maxima, cap, exponentials and parts 2800, taking in the last block's sums 450); a launch of one block 8 - 9 us.  2048
// causal rows of 16 heads over 4: 60 us, capped 71 (mma.sync: 171, 187); 700 rows on 300 keys of 32 heads over 32, capped / chunks of
// 512 with a bias 121 / 80 -> 55 / 47; 2 / 33 / 200 rows of 16 over 4 8.4 / 9.2 / 15.8 -> 8.3 / 8.7 / 14.2.  When a warp after the
// other brought its queries, before the first keys and for rows of no tile too: 9.8 / 12.8 / 15.5.
//
// As in fmha2_tcgen05.cu a row's reference maximum moves only when a score exceeds it by 5.5 (a weight of 2^8): exact, since
// weights, sums and l use the same.
//
// Relative error against float64 (2-norm, fp32 out, rows on 64 / 512 / 2048 / 3072 keys; mma.sync in brackets), values of both signs:
// 1.2 / 2.0 / 2.1 / 2.15e-7 (1.5 / 2.8 / 3.0 / 3.05e-7); of one sign: 0.88 / 1.02 / 1.05 / 1.08e-7 (0.92 / 1.04 / 1.14 / 1.21e-7).  With
// one sum of all first parts and one of all blocks (l compensated as below): 1.5 / 2.8 / 3.0 / 3.05e-7 and 0.92 / 1.06 / 1.27 /
// 1.40e-7; the two sums of a score cost nothing, a row's groups of four blocks 2 % (2048 capped rows 74.1 -> 75.7 us).
#include "../../include/vila_b200.h"
#include "common.cuh"
#include "kernels.h"
#include "dtype_any.cuh"
#include "paged_attn_common.cuh"
#include "mma_bf16.cuh"

namespace vb {
namespace {

constexpr int D = 128, kBK = 64, kM = 128;
constexpr int kLoaders = 2, kMma = 8 + kLoaders, kThreads = 32 * (kMma + 1);
constexpr int kQPart = kM * D * 2;                 // bytes of a part of the queries
constexpr int kStage = 2 * kBK * D * 2;            // keys, then values
constexpr int kStages = 3;
constexpr int kNumBars = 2 * kStages + 6;
constexpr int kSmem = 3 * kQPart + kStages * kStage + 3 * 2 * kM * 4 + kNumBars * 8 + 16 + 1024;
constexpr int kBiasBytes = (227 * 1024 - kSmem) / 16 * 16;
static_assert(kBiasBytes >= 16 * 1024, "paged_attn_tc: shared memory");
constexpr float kLead = 5.5f;

// A row's sums join those in TMEM behind every fourth block of its sequence, and behind the second and the last kept one of a window:
// by position, so that a row's numbers do not depend on its launch.
__device__ __forceinline__ bool joins(int block, int kept_blocks) { return (block & 3) == 3 || block == 1 || block == kept_blocks - 1; }

template <bool CAP>
__global__ void __launch_bounds__(kThreads, 1)
paged_attn_tc_kernel(const __grid_constant__ vila_paged_attn_params p, int tiles_per_cta, int bias_rows, const WaitLimit limit, volatile unsigned int* failed) {
  extern __shared__ uint8_t raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* q_s = smem;                             // [part][64-column chunk][128 rows]
  uint8_t* ring = q_s + 3 * kQPart;                // [stage]: keys [chunk][64], values [chunk][64]
  float* xm = reinterpret_cast<float*>(ring + kStages * kStage);   // [half][row]: maxima, sums, rows that are not finite
  float* xl = xm + 2 * kM;
  int* xodd = reinterpret_cast<int*>(xl + 2 * kM);
  uint64_t* kv_full = reinterpret_cast<uint64_t*>(xodd + 2 * kM);
  uint64_t* kv_empty = kv_full + kStages;
  uint64_t* s_full = kv_empty + kStages;           // [2]
  uint64_t* p_full = s_full + 2;                   // [2]
  uint64_t* o_full = p_full + 2;
  uint64_t* fin = o_full + 1;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(fin + 1);
  volatile int* gave_up = reinterpret_cast<int*>(tmem_ptr + 1);
  float* bias_s = reinterpret_cast<float*>(tmem_ptr + 4);   // [head][bias_rows]: the heads' biases by distance, if there is room

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  // CTAs of late positions, which see most keys, start first, those of all heads
  const int rep = p.H / p.G, g = blockIdx.x % p.G;
  const int tile0 = (static_cast<int>(gridDim.x) / p.G - 1 - static_cast<int>(blockIdx.x) / p.G) * tiles_per_cta, ntile = min(tiles_per_cta, p.ntiles - tile0);
  if (warp == kMma && lane == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&kv_full[i], 32 * kLoaders);
      mbar_init(&kv_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 8);
    }
    mbar_init(o_full, 1);
    mbar_init(fin, 1);
    *gave_up = 0;
    fence_barrier_init();
  }
  if (warp == kMma) tmem_alloc<512>(tmem_ptr);
  tc_fence_before();
  __syncthreads();   // the loaders go ahead, the others meet again behind the queries
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  if (warp < 8) {
    // queries, scaled, in three parts: row r is row r & 15 of tile (r >> 4) / rep, head (r >> 4) % rep.  A warp brings a row at a time
    // and asks for eight before it writes: one after the other their latency was 5 us.  Whole 32 rows of no
    // tile hold what was there: their warps leave them alone.
    constexpr int kAhead = 8;
    for (int r0 = warp; r0 < (16 * rep * ntile + 31) / 32 * 32; r0 += 8 * kAhead) {
      float4 v[kAhead];
      float sc[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int r = r0 + 8 * u, mt = (r >> 4) / rep, h = g * rep + (r >> 4) % rep;
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        sc[u] = 0.f;
        if (mt < ntile) {
          const int* t = p.tiles + 4 * (tile0 + mt);
          if ((r & 15) < t[1]) v[u] = *reinterpret_cast<const float4*>(p.q + (static_cast<size_t>(t[0] + (r & 15)) * p.H + h) * D + 4 * lane);
          sc[u] = head_scale(p, h);
        }
      }
      uint8_t* at = q_s + (lane >> 4) * (kM * 128) + (lane & 1) * 8;
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int r = r0 + 8 * u;
        uint2 part[3];
        split3(v[u].x * sc[u], v[u].y * sc[u], part[0].x, part[1].x, part[2].x);
        split3(v[u].z * sc[u], v[u].w * sc[u], part[0].y, part[1].y, part[2].y);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint2*>(at + k * kQPart + r * 128 + ((((lane & 15) >> 1) ^ (r & 7)) << 4)) = part[k];
      }
    }
    fence_proxy_async_smem();
  }
  if (warp < 8 || warp == kMma) asm volatile("bar.sync 5, 288;" ::: "memory");

  // the CTA's tiles in runs of one sequence (nearly always a single run)
  struct Run {
    int begin, end, slot, nkeys;
    BlockList bl;
  };
  auto next_run = [&](Run& r, int begin) {
    if (begin >= ntile) return false;
    r.begin = begin;
    r.slot = p.tiles[4 * (tile0 + begin) + 3];
    int first_pos = 0x7fffffff;
    r.nkeys = 0;
    for (r.end = begin; r.end < ntile && p.tiles[4 * (tile0 + r.end) + 3] == r.slot; ++r.end) {
      const int* t = p.tiles + 4 * (tile0 + r.end);
      first_pos = min(first_pos, t[2]);
      r.nkeys = max(r.nkeys, t[2] + t[1]);
    }
    r.bl = visible_blocks(p, first_pos, r.nkeys, kBK);
    return true;
  };
  if (limit.quits == (warp < 8 ? 2 : warp == kMma ? 1 : 0)) *gave_up = 1;
  auto wait = [&](uint64_t* bar, int phase) { return __all_sync(0xffffffffu, mbar_wait_limited(bar, phase & 1, gave_up, limit.tries)); };
  Run run;

  if (warp >= 8 && warp < kMma) {
    // ===================== keys and values =====================
    const size_t prow = static_cast<size_t>(p.G) * 2 * D;
    const __nv_bfloat16* pool = static_cast<const __nv_bfloat16*>(p.pool);
    // lane: a 16-byte piece of the keys' (0 - 15) or the values' rows
    constexpr int kKeys = kBK / kLoaders;   // of a warp, one to a lane
    static_assert(kKeys == 32, "paged_attn_tc: loaders");
    const int c = lane & 15, k0 = (warp - 8) * kKeys;
    const size_t off = (static_cast<size_t>(lane < 16 ? 0 : p.G) + g) * D + 8 * c;
    const uint32_t dst = smem_u32(ring) + (lane < 16 ? 0 : kBK * D * 2) + (c >> 3) * (kBK * 128) + k0 * 128;
    int stage = 0, ph = 1;
    bool ok = limit.quits != 0;
    for (int b = 0; ok && next_run(run, b); b = run.end) {
      const int32_t* pt = p.page_tables + static_cast<size_t>(run.slot) * p.pt_stride;
      auto look = [&](int v) {   // rows of this warp's keys of block v, -1 behind the last
        if (v >= run.bl.count) return -1;
        const int j = run.bl.block(v) * kBK + k0 + lane;
        return j < run.nkeys ? static_cast<int>(pool_row(pt, p.page, j)) : -1;
      };
      int rows = look(0);
      for (int v = 0; v < run.bl.count; ++v) {
        const int next = look(v + 1);
        ok = wait(&kv_empty[stage], ph);
        if (!ok) break;
#pragma unroll 8
        for (int jj = 0; jj < kKeys; ++jj) {
          const int row = __shfl_sync(0xffffffffu, rows, jj);
          cp16(dst + stage * kStage + jj * 128 + (((c & 7) ^ (jj & 7)) << 4), pool + static_cast<size_t>(max(row, 0)) * prow + off, row >= 0);
        }
        // shown to the tensor core by who wrote it: the issuer would take 300 clocks a block for it
        asm volatile("cp.async.wait_all;" ::: "memory");
        fence_proxy_async_smem();
        mbar_arrive(&kv_full[stage]);
        rows = next;
        if (++stage == kStages) {
          stage = 0;
          ph ^= 1;
        }
      }
    }
  } else if (warp == kMma) {
    // ===================== products =====================
    int total = 0;
    for (int b = 0; next_run(run, b); b = run.end) total += run.bl.count;
    constexpr uint32_t idesc_s = make_idesc_bf16(kM, kBK, 0, 0);
    constexpr uint32_t idesc_o = make_idesc_bf16(kM, D, 0, 1);
    const uint64_t qd = make_smem_desc(smem_u32(q_s), 16, 1024, kLayoutSW128);
    const uint64_t kd0 = make_smem_desc(smem_u32(ring), 16, 1024, kLayoutSW128);
    const uint64_t vd0 = make_smem_desc(smem_u32(ring) + kBK * D * 2, kBK * 128, 1024, kLayoutSW128);
    bool ok = limit.quits != 1;
    auto issue_s = [&](int n, int stage) {
      tc_fence_after();
      if (elect_one()) {
        const uint64_t kd = kd0 + static_cast<uint32_t>(stage * (kStage >> 4));
        const uint32_t d = tmem + (n & 1) * 128;
#pragma unroll
        for (int part = 2; part >= 0; --part)
#pragma unroll
          for (int k = 0; k < D / 16; ++k)
            umma_f16(d + (part || k >= D / 32 ? 64 : 0), qd + ((part * kQPart + (k >> 2) * (kM * 128) + (k & 3) * 32) >> 4),
                     kd + (((k >> 2) * (kBK * 128) + (k & 3) * 32) >> 4), idesc_s, k != 0 || part == 1 ? 1u : 0u);
        umma_commit(&s_full[n & 1]);
      }
      __syncwarp();
    };
    if (ok && total > 0) {
      ok = wait(&kv_full[0], 0);
      if (ok) issue_s(0, 0);
    }
    int st = 0, st1 = 1, ph1 = 0;   // stages of blocks n and n + 1, whose turn
    for (int n = 0; ok && n < total; ++n) {
      if (n + 1 < total) {
        ok = wait(&kv_full[st1], ph1);
        if (!ok) break;
        issue_s(n + 1, st1);
      }
      ok = wait(&p_full[n & 1], n >> 1);   // behind it the sums of block n - 1 have been taken in, too
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint64_t vd = vd0 + static_cast<uint32_t>(st * (kStage >> 4));
        const uint32_t a = tmem + (n & 1) * 128, d = tmem + 256;
#pragma unroll
        for (int part = 2; part >= 0; --part)
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)   // keys 16 k ..: of half k / 2, whose parts stand over its own scores
            umma_f16_ts(d, a + (k >> 1) * 32 + (part == 2 ? 64 : 16 * part) + (k & 1) * 8, vd + k * (16 * 128 >> 4), idesc_o,
                        part != 2 || k != 0 ? 1u : 0u);
        umma_commit(o_full);
        umma_commit(&kv_empty[st]);
      }
      __syncwarp();
      st = st1;
      if (++st1 == kStages) {
        st1 = 0;
        ph1 ^= 1;
      }
    }
    // products in flight end before their operands and TMEM go, whichever warp gave up (the loaders' copies have landed)
    if (elect_one()) umma_commit(fin);
    mbar_drain(fin, 0);
  } else if ((warp & 3) * 32 >= 16 * rep * ntile) {
    // no rows: the weights that stand there reach sums that nobody reads
    int n = 0;
    for (int b = 0; next_run(run, b); b = run.end)
      for (int v = 0; v < run.bl.count; ++v, ++n) {
        wait(&s_full[n & 1], n >> 1);
        if (lane == 0) mbar_arrive(&p_full[n & 1]);
      }
  } else {
    // ===================== softmax =====================
    const int half = warp >> 2, quad = warp & 3, r = quad * 32 + lane, id = 1 + quad;
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    const int my_tile = (r >> 4) / rep, h = g * rep + (r >> 4) % rep;
    const bool active = my_tile < ntile;
    const int* tile = p.tiles + 4 * (tile0 + (active ? my_tile : 0));
    const int i = r & 15, row0 = tile[0], nrows = active ? tile[1] : 0;
    const int pos = i < nrows ? tile[2] + i : -1;
    const int lo = first_key(p, max(pos, 0)), wlo = p.window > 0 ? pos - p.window + 1 : 0, keep = p.window > 0 ? p.keep_first : 0;
    const float cap_inv = cap_inverse(p);
    if (bias_rows > 0) {   // under the first block's scores
      // the heads' biases, neighbours in global memory, by the distances that occur
      int far = 0;
      for (int mt = 0; mt < ntile; ++mt) far = max(far, p.tiles[4 * (tile0 + mt) + 2] + p.tiles[4 * (tile0 + mt) + 1]);
      if (p.chunk > 0) far = min(far, p.chunk);
      const int nbias = rep * min(far, bias_rows), nq = (16 * rep * ntile + 31) / 32;   // pairs of warps that have rows
      for (int x0 = half * 32 * nq + quad * 32 + lane; x0 < nbias; x0 += 4 * 64 * nq) {
        float b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int x = x0 + u * 64 * nq;
          if (x < nbias) b[u] = p.dist_bias[static_cast<size_t>(x / rep) * p.H + g * rep + x % rep];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int x = x0 + u * 64 * nq;
          if (x < nbias) bias_s[(x % rep) * bias_rows + x / rep] = b[u];
        }
      }
      asm volatile("bar.sync 6, %0;" ::"r"(64 * nq) : "memory");
    }
    float m = kNegBig, l = 0.f;
    float l_lost = 0.f;   // what l's additions rounded away: one sum over all keys of a row weighs on every column
    if (p.sink != nullptr) {
      const float z = p.sink[h];
      if (z >= kNegBig) {   // a sink below every score (-inf: switched off) weighs nothing
        m = z;
        l = half == 0 ? ex2(fmaf(z, kLog2e, -log2_units(z))) : 0.f;
      }
    }
    float o[64];
#pragma unroll
    for (int c = 0; c < 64; ++c) o[c] = 0.f;
    int n = 0;            // blocks so far
    bool pending = false; // the sums of block n - 1 have not been taken in
    int last = 0;         // that block's place in its sequence
    const uint32_t sums = lanes + 384 + half * 64;
    bool kept = false;    // there are sums in TMEM
    // o joins the row's sums in TMEM.  With nothing in o it changes nothing, so that it does not matter whether a row's CTA goes on
    // over blocks that the row does not see.
    auto keep_sums = [&]() {
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        uint32_t t[32];
        if (kept) {
          tmem_ld_32x32b_x32(sums + c, t);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 2) add2(o[c + e], o[c + e + 1], __uint_as_float(t[e]), __uint_as_float(t[e + 1]));
        }
        tmem_st_32x32b_x32(sums + c, reinterpret_cast<uint32_t*>(o + c));
#pragma unroll
        for (int e = 0; e < 32; ++e) o[c + e] = 0.f;
      }
      tmem_st_wait();
      kept = true;
    };
    auto take = [&](int b) {
      wait(o_full, b);
      tc_fence_after();
      const uint32_t at = lanes + 256 + half * 64;
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        uint32_t t[32];
        tmem_ld_32x32b_x32(at + c, t);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; e += 2) add2(o[c + e], o[c + e + 1], __uint_as_float(t[e]), __uint_as_float(t[e + 1]));
      }
    };
    for (int b = 0; next_run(run, b); b = run.end) {
      const bool mine = active && my_tile >= run.begin && my_tile < run.end && pos >= 0;
      for (int v = 0; v < run.bl.count; ++v, ++n) {
        const int j0 = run.bl.block(v) * kBK + half * 32;
        const uint32_t at = lanes + (n & 1) * 128 + half * 32;
        wait(&s_full[n & 1], n >> 1);
        tc_fence_after();
        float s[32];
        {
          uint32_t t0[32], t1[32];
          tmem_ld_32x32b_x32(at, t0);
          tmem_ld_32x32b_x32(at + 64, t1);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            s[e] = __uint_as_float(t0[e]);
            s[e + 1] = __uint_as_float(t0[e + 1]);
            add2(s[e], s[e + 1], __uint_as_float(t1[e]), __uint_as_float(t1[e + 1]));
          }
        }
        if (CAP) {
          float top[4] = {0.f, 0.f, 0.f, 0.f};   // NaN is NaN in either form
#pragma unroll
          for (int e = 0; e < 32; ++e) top[e & 3] = fmaxf(top[e & 3], fabsf(s[e]));
          if (__any_sync(0xffffffffu, fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])) > p.softcap)) {
            const float inv_over = cap_inverse_over(cap_inv);
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
              const float x = s[e], y = s[e + 1];
              cap2(s[e], s[e + 1], cap_inv);
              if (over_cap(p, x)) s[e] = capped_over(p.softcap, inv_over, x);
              if (over_cap(p, y)) s[e + 1] = capped_over(p.softcap, inv_over, y);
            }
          } else {
#pragma unroll
            for (int e = 0; e < 32; e += 2) cap2(s[e], s[e + 1], cap_inv);
          }
        }
        if (bias_rows > 0) {
          const float* bias = bias_s + (h - g * rep) * bias_rows;
#pragma unroll
          for (int e = 0; e < 32; ++e) s[e] += bias[min(max(pos - (j0 + e), 0), bias_rows - 1)];
        } else if (p.dist_bias) {
#pragma unroll
          for (int e = 0; e < 32; ++e) s[e] += dist_bias(p, max(pos - (j0 + e), 0), h);
        }
        // does the row see all of its thread's keys
        const bool all = mine && j0 + 31 <= pos && j0 >= lo && (j0 >= wlo || j0 + 31 < keep);
        const bool every = __all_sync(0xffffffffu, all);
        if (!every) {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const int j = j0 + e;
            if (!(mine && j <= pos && j >= lo && (j >= wlo || j < keep))) s[e] = kNegBig;
          }
        }
        float m4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
        for (int e = 4; e < 32; ++e) m4[e & 3] = fmaxf(m4[e & 3], s[e]);
        float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
        if (pair_any(id, mx > m + kLead)) {
          xm[half * kM + r] = mx;
          pair_sync(id);
          mx = fmaxf(mx, xm[(half ^ 1) * kM + r]);
          if (pending) take(n - 1);
          pending = false;
          const float mn = mx > m + kLead ? mx : m;
          const float alpha = ex2(__fsub_rn(log2_units(m), log2_units(mn)));
          l *= alpha;
          l_lost *= alpha;
#pragma unroll
          for (int c = 0; c < 64; ++c) o[c] *= alpha;
          if (kept) {
#pragma unroll 1
            for (int c = 0; c < 64; c += 8) {   // rare: few registers
              uint32_t t[8];
              tmem_ld_32x32b_x8(sums + c, t);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 8; ++e) t[e] = __float_as_uint(__uint_as_float(t[e]) * alpha);
              tmem_st_32x32b_x8(sums + c, t);
            }
            tmem_st_wait();
          }
          m = mn;
        }
        const float ml = log2_units(m);
        float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 2; ++k) {   // 16 keys: 8 columns of each part
          uint32_t part[3][8];
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            float* w = s + 16 * k + e;
            const float w0 = ex2(fmaf(w[0], kLog2e, -ml)), w1 = ex2(fmaf(w[1], kLog2e, -ml));
            // a hidden key weighs nothing, also while its row has seen no key at all (m still kNegBig)
            const float x = every || w[0] != kNegBig ? w0 : 0.f, y = every || w[1] != kNegBig ? w1 : 0.f;
            add2(l4[e & 2], l4[(e & 2) + 1], x, y);
            split3(x, y, part[0][e / 2], part[1][e / 2], part[2][e / 2]);
          }
          tmem_st_32x32b_x8(at + 8 * k, part[0]);
          tmem_st_32x32b_x8(at + 16 + 8 * k, part[1]);
          tmem_st_32x32b_x8(at + 64 + 8 * k, part[2]);
        }
        const float lb = (l4[0] + l4[1]) + (l4[2] + l4[3]), ls = __fadd_rn(l, lb), lt = __fsub_rn(ls, l);
        l_lost += __fadd_rn(__fsub_rn(l, __fsub_rn(ls, lt)), __fsub_rn(lb, lt));
        l = ls;
        tmem_st_wait();
        if (pending) take(n - 1);   // before this block's product, which goes where these sums are
        if (n > 0 && joins(last, (keep + kBK - 1) / kBK)) keep_sums();
        pending = true;
        last = run.bl.block(v);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[n & 1]);
      }
    }
    if (pending) take(n - 1);
    if (kept) {
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        uint32_t t[32];
        tmem_ld_32x32b_x32(sums + c, t);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; e += 2) add2(o[c + e], o[c + e + 1], __uint_as_float(t[e]), __uint_as_float(t[e + 1]));
      }
    }
    // ---- rows
    l += l_lost;
    float z = l * 0.f;
#pragma unroll
    for (int c = 0; c < 64; ++c) z = fmaf(o[c], 0.f, z);
    const bool valid = i < nrows;
    xl[half * kM + r] = l;
    xodd[half * kM + r] = valid && !(z == 0.f);
    pair_sync(id);
    l += xl[(half ^ 1) * kM + r];
    const bool odd = (xodd[r] | xodd[kM + r]) != 0;
    unsigned again = __ballot_sync(0xffffffffu, odd);
    if (again) {   // the ring is free: every block has been multiplied
      float* rows = reinterpret_cast<float*>(ring);
      for (int k = half; again; k ^= 1) {
        const int src = __ffs(again) - 1, ri = __shfl_sync(0xffffffffu, i, src);
        again &= again - 1;
        const int rr0 = __shfl_sync(0xffffffffu, row0, src), rpos = __shfl_sync(0xffffffffu, pos, src), rh = __shfl_sync(0xffffffffu, h, src);
        const int slot = __shfl_sync(0xffffffffu, tile[3], src);
        if (k == 0) row_again<D, 1, D>(p, rr0 + ri, rpos, slot, rh, 0, rows + (quad * 32 + src) * D);
      }
      pair_sync(id);
      if (odd) {
        l = 1.f;
#pragma unroll
        for (int c = 0; c < 64; c += 4) {
          const float4 x = *reinterpret_cast<const float4*>(rows + r * D + half * 64 + c);
          o[c] = x.x;
          o[c + 1] = x.y;
          o[c + 2] = x.z;
          o[c + 3] = x.w;
        }
      }
    }
    if (valid) {
      const float inv = out_gate(p, row0 + i, h) / l;
      const size_t ob = (static_cast<size_t>(row0 + i) * p.H + h) * D + half * 64;
      if (p.out_dtype == VILA_DT_F32) {
#pragma unroll
        for (int c = 0; c < 64; c += 4)
          *reinterpret_cast<float4*>(static_cast<float*>(p.out) + ob + c) = make_float4(o[c] * inv, o[c + 1] * inv, o[c + 2] * inv, o[c + 3] * inv);
      } else {
#pragma unroll
        for (int c = 0; c < 64; c += 8)
          *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.out) + ob + c) =
              make_uint4(pack_bf16(o[c] * inv, o[c + 1] * inv), pack_bf16(o[c + 2] * inv, o[c + 3] * inv),
                         pack_bf16(o[c + 4] * inv, o[c + 5] * inv), pack_bf16(o[c + 6] * inv, o[c + 7] * inv));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMma) {
    tc_fence_after();
    tmem_dealloc<512>(tmem);
  }
  if (tid == 0 && *gave_up) {
    *failed = 1u;
    __threadfence_system();
  }
}

template <bool CAP>
int launch(const vila_paged_attn_params& p, cudaStream_t stream, int tries) {
  volatile unsigned int* failed = failed_word();
  VB_CHECK(failed != nullptr, "paged_attention: no pinned host memory for the status word");
  auto kernel = paged_attn_tc_kernel<CAP>;
  static PerDeviceOnce once;
  if (once.first()) VB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem + kBiasBytes));
  // Tiles of a CTA: as few as leave no CTA without an SM, otherwise as many as its 128 rows hold.  A CTA of one tile takes as long
  // as one of several tiles of a sequence, and tiles of other sequences wait for each other there: 8 sequences of 16 rows on 100 keys,
  // capped, 16 heads over 4 / over 16 / 32 over 32 19.8 / 48 / 49 us as full as they get and 11.2 / 11.6 / 16.9 so (mma.sync 12.1 / 29 /
  // 29); 16 of 3 rows on 900 74 / 274 / 274 and 40 / 77 / 145 (50 / 171 / 172).
  const int rep = p.H / p.G;
  int tpc = 1;
  while (tpc < 8 / rep && static_cast<long>((p.ntiles + tpc - 1) / tpc) * p.G > num_sms()) ++tpc;
  // a lookup of every score in global memory, a line apart from row to row, cost more than the rest of a block's softmax
  const long bias_bytes = p.dist_bias ? 4L * rep * p.dist_rows : 0;
  const bool staged = bias_bytes > 0 && bias_bytes <= kBiasBytes;
  const long ctas = static_cast<long>((p.ntiles + tpc - 1) / tpc) * p.G;
  VB_CHECK(ctas < (1L << 31), "paged_attention: too many tiles");
  VB_CUDA(launch_serial(kernel, dim3(static_cast<unsigned>(ctas)), dim3(kThreads), kSmem + (staged ? bias_bytes : 0), stream, p, tpc, staged ? p.dist_rows : 0, wait_limit(tries), failed));
  return 0;
}

bool aligned(const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; }

}  // namespace

bool paged_attention_tc_takes(const vila_paged_attn_params& p) {
  return p.max_rows > 1 && p.nsplit == 1 && p.pool_dtype == VILA_DT_BF16 && p.talk == nullptr && maps_of(p.maps) == 1 && p.dim == D && p.vdim == D &&
         p.H / p.G <= 8 && aligned(p.pool, 16) && aligned(p.q, 16) && aligned(p.out, 16);
}

int paged_attention_tc(const vila_paged_attn_params& p, cudaStream_t stream, int tries) {
  if (wait_status()) return 1;   // an earlier launch gave up: nothing is built on its output
  return p.softcap > 0.f ? launch<true>(p, stream, tries) : launch<false>(p, stream, tries);
}

}  // namespace vb
