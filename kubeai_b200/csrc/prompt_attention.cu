// Softmax attention of whole prompts on the 5th-generation tensor cores (mixers.h PromptAttnArgs): every sequence of the step
// starts at its first token, so its keys and values are the step's own rows and lie densely in memory.  Causal, with an
// optional window, sink, cap and per-head gate; 128 dimensions a head, or 128 of its own and 64 more against a key part that
// all heads share (latent attention, whose per-head keys and values one product rebuilds from the latents: that and 192 + 256
// dimensions a pair are 0.4 of the work of scores and sums in 576 + 512 latent dimensions).  There a value is two bf16 terms, the
// rounded sum and what the rounding left: the absorbed form it stands for keeps the weighted latents in fp32 up to W_uv.
//
// A CTA owns 256 query tokens of one head as two 128-row tiles that share every 64-key tile.  One thread loads (TMA, 128-byte
// swizzle, keys and values in rings of their own), one issues every tcgen05.mma:
//   S_i = Q_i K^T    M = 128, N = 64; two buffers per tile in TMEM, so that the next scores are formed under this softmax
//   O_i += P_i V     M = 128, N = 128; P_i in TMEM, where the softmax warps wrote it over its scores, V in place as an MN-major operand
// Two groups of four softmax warps (thread = row) work in fp32 with base-2 exponentials and rescale O_i in TMEM only when a row
// of the warp moved its maximum.  Key tiles outside a row tile's triangle or window are skipped for that tile.  Rows behind a
// sequence's end belong to the next one: their keys are masked and their values cleared, so that nothing of another sequence
// can reach a result.  A masked key has weight 0, which a product turns into NaN where its value is infinite or NaN: a row that
// comes out not finite looks for such a key and is then formed again, key by key.  Every wait has a limit; a CTA that gives up sets an error mark and still meets at the end.
//
// With keys and values per head (window_prompt_prep gathers them from the cache): sequences of 455, 1365 and 2275 tokens, 16 query
// and 4 key heads, cap: 291 us on mma.sync -> 101.
//
// What bounds it, in cycles of a key tile (of both row tiles): the products with 192 dimensions a head and two terms, 2100 of 3200 (scores of 64
// columns are held up by their operands in shared memory); under a cap the exponentials' unit, three a score, 3100 of 3500; else
// half and half, with what the barriers between them cost.  The longest CTA has 36 of the tiles.  16 heads, 192 + 128 dimensions with
// values in two terms, sequences of 455, 1365 and 2275 tokens: 77 us (52 GFLOP); the latent-space kernel on mma.sync took 883, with its two
// per-head products 1109.  With P in shared memory, one buffer of second terms and one product a time it
// took 90 (under a cap, 4096 tokens in eight sequences, 60 for 55 now).
//
// Weights are relative to the row's largest score so far, so the largest weight is exactly 1 and its rounding to bf16 costs nothing.  Relative to 2^8 times an
// older maximum, which saves most of the rescaling (75 us for 77, under the cap 53.6 for 55.3, 39.0 for 42.4 in windows), outputs were off by 2 to 10 % more.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdlib.h>

#include <atomic>

#include "gemm.h"
#include "launch.h"
#include "mixers.h"
#include "ptx.cuh"

namespace b200 {
namespace {

typedef __nv_bfloat16 bf16;
constexpr int kRows = 128, kKeys = 64, kD = 128;     // rows of a query tile, keys of a tile, value dimensions
constexpr int kQSlab = kRows * 128, kKSlab = kKeys * 128;   // bytes of 64 columns
constexpr int kVTile = 2 * kKSlab;
constexpr int kThreads = 320;                        // warp 0: loads, warps 1-4 and 5-8: rows of tile 0 and 1, warp 9: products
constexpr int kWaitLimit = 1 << 22;
template <int NS>
constexpr int smem_bytes() { return 1024 + 2 * NS * kQSlab + 2 * NS * kKSlab + 2 * (NS == 3 ? 2 : 1) * kVTile + 256; }
static_assert(smem_bytes<3>() <= 227 * 1024, "");

__device__ __forceinline__ uint32_t idesc_bf16(uint32_t m, uint32_t n, uint32_t b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
// shared-memory descriptor, 128B swizzle, leading and stride byte offsets
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return static_cast<uint64_t>((addr & 0x3FFFFu) >> 4) | static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16 | static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32 |
         static_cast<uint64_t>(1) << 46 | static_cast<uint64_t>(2) << 61;
}
__device__ __forceinline__ bool wait_limited(uint32_t bar, uint32_t parity) { return mbar_wait_limited(bar, parity, kWaitLimit); }
// ... by a whole warp: whether all lanes saw the phase end
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, wait_limited(bar, parity)); }

// A row that came out not finite: where a key that it masks but its tiles hold ([begin, end)) has a value that is not finite, the
// row is formed again from the keys it sees and from no other (a thread; what it sees itself decides otherwise).
template <int NS, bool CAP>
__device__ __noinline__ void plain_row(const PromptAttnArgs& a, int tok0, int p, int head, int kvh, int begin, int end) {
  const long long tok = tok0 + p;
  const bf16 *q = static_cast<const bf16*>(a.q) + tok * a.ldq + head * a.q_step, *q2 = static_cast<const bf16*>(a.q2) + tok * a.heads * 64 + head * 64;
  const bf16 *kv = static_cast<const bf16*>(a.kv), *k2 = static_cast<const bf16*>(a.k2), *v2 = static_cast<const bf16*>(a.v2);
  const int lo = max(0, p - a.window + 1);
  bool beside = false;
  for (int j = begin; j < end && !beside; ++j) {
    if (j >= lo && j <= p) { j = p; continue; }
    const uint4* v = reinterpret_cast<const uint4*>(kv + static_cast<long long>(tok0 + j) * a.ldkv + a.v_off + kvh * a.v_step);
    for (int c = 0; c < kD / 8; ++c) {
      const uint4 x = v[c];
      auto odd = [](uint32_t u) { return (u & 0x7f80u) == 0x7f80u || (u & 0x7f800000u) == 0x7f800000u; };
      beside = beside || odd(x.x) || odd(x.y) || odd(x.z) || odd(x.w);
    }
  }
  if (!beside) return;
  auto score = [&](int j) {
    const bf16* k = kv + static_cast<long long>(tok0 + j) * a.ldkv + a.k_off + kvh * a.k_step;
    float s = 0.f;
    for (int d = 0; d < kD; ++d) s = fmaf(__bfloat162float(q[d]), __bfloat162float(k[d]), s);
    if (NS == 3)
      for (int d = 0; d < 64; ++d) s = fmaf(__bfloat162float(q2[d]), __bfloat162float(k2[static_cast<long long>(tok0 + j) * 64 + d]), s);
    s *= a.scale;
    return CAP ? a.softcap * tanhf(s / a.softcap) : s;
  };
  float m = a.sink ? a.sink[head] : -INFINITY;
  for (int j = lo; j <= p; ++j) m = fmaxf(m, score(j));
  float out = a.out_scale;
  if (a.gate) out *= 1.0f / (1.0f + expf(-__bfloat162float(static_cast<const bf16*>(a.gate)[tok * a.ldg + head])));
  bf16* y = static_cast<bf16*>(a.y) + tok * a.ldy + head * kD;
  for (int c0 = 0; c0 < kD; c0 += 16) {
    float acc[16] = {}, l = a.sink ? expf(a.sink[head] - m) : 0.f;
    for (int j = lo; j <= p; ++j) {
      const float w = expf(score(j) - m);
      l += w;
      const bf16 *v = kv + static_cast<long long>(tok0 + j) * a.ldkv + a.v_off + kvh * a.v_step + c0, *u = v2 + static_cast<long long>(tok0 + j) * a.heads * kD + head * kD + c0;
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        float x = __bfloat162float(v[c]);
        if (NS == 3 && isfinite(x)) x += __bfloat162float(u[c]);
        acc[c] = fmaf(w, x, acc[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < 16; ++c) y[c0 + c] = __float2bfloat16_rn(acc[c] / l * out);
  }
}

// NS: 64-column slabs of a query or key row (2, or 3 with the shared part and values in two terms)
template <int NS, bool CAP>
__global__ void __launch_bounds__(kThreads, 1)
prompt_attn_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_q2, const __grid_constant__ CUtensorMap tm_kv,
                   const __grid_constant__ CUtensorMap tm_k2, const __grid_constant__ CUtensorMap tm_v2, const __grid_constant__ PromptAttnArgs a) {
  constexpr bool LO = NS == 3;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (sbase - smem_u32(smem_raw));
  const uint32_t q_s = sbase;                               // [tile][slab]
  const uint32_t k_s = q_s + 2 * NS * kQSlab;               // [stage][slab]
  constexpr int kVStage = (LO ? 2 : 1) * kVTile;
  const uint32_t v_s = k_s + 2 * NS * kKSlab;               // [stage][term][half]
  const uint32_t bars = v_s + 2 * kVStage;
  auto k_full = [&](int s) { return bars + 8u * s; };
  auto k_empty = [&](int s) { return bars + 8u * (2 + s); };
  auto v_full = [&](int s) { return bars + 8u * (4 + s); };
  auto v_empty = [&](int s) { return bars + 8u * (6 + s); };
  auto s_full = [&](int i, int b) { return bars + 8u * (8 + 2 * i + b); };
  // Of every other tile each, as the scores': a warp is up to two tiles ahead of the slowest one of its group.
  auto p_ready = [&](int i, int b) { return bars + 8u * (12 + 2 * i + b); };     // 4 warps: S_i read, P_i in its place, O_i rescaled
  auto pv_full = [&](int i, int b) { return bars + 8u * (16 + 2 * i + b); };
  const uint32_t q_bar = bars + 8u * 20, tmem_slot = bars + 8u * 21;
  const int warp = warp_number(), lane = threadIdx.x & 31;

  if (warp == 0) {
    if (lane == 0) {
      for (int s = 0; s < 2; ++s) { mbar_init(k_full(s), 1); mbar_init(k_empty(s), 1); mbar_init(v_full(s), 1); mbar_init(v_empty(s), 1); }
      for (int i = 0; i < 2; ++i)
        for (int b = 0; b < 2; ++b) { mbar_init(s_full(i, b), 1); mbar_init(p_ready(i, b), 4); mbar_init(pv_full(i, b), 1); }
      mbar_init(q_bar, 1);
      fence_mbar_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + (tmem_slot - sbase));
  auto tm_s = [&](int i, int b) { return tmem + 64u * (2 * i + b); };
  auto tm_o = [&](int i) { return tmem + 256u + 128u * i; };

  // which sequence and which 256 of its tokens: the blocks run over all sequences' tiles in falling order of the keys they see
  int seq = -1, n = 0, q0 = 0;
  {
    auto tiles_of = [&](int s) { return s < a.nseq ? (a.seqs[s * 8 + 1] + 2 * kRows - 1) / (2 * kRows) : 0; };
    const int mine = tiles_of(lane);
    int level = mine, idx = blockIdx.y;
    for (int s = 32 + lane; s < a.nseq; s += 32) level = max(level, tiles_of(s));
    level = __reduce_max_sync(0xffffffffu, level);
    while (seq < 0 && --level >= 0)
      for (int base = 0; base < a.nseq; base += 32) {
        const unsigned have = __ballot_sync(0xffffffffu, (base ? tiles_of(base + lane) : mine) > level);
        if (idx < __popc(have)) {
          seq = base + __fns(have, 0, idx + 1);
          n = a.seqs[seq * 8 + 1];
          q0 = level * 2 * kRows;
          break;
        }
        idx -= __popc(have);
      }
  }
  if (seq >= 0) {
    const int tok0 = a.seqs[seq * 8], head = blockIdx.x, kvh = head / (a.heads / a.kv_heads);
    // first and last key tile of each row tile; none for a tile behind the sequence's end
    int first[2], last[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int p = q0 + i * kRows;
      first[i] = max(0, p - a.window + 1) / kKeys;
      last[i] = p < n ? (min(p + kRows, n) - 1) / kKeys : -1;
    }
    const int t_begin = first[0], t_end = max(last[0], last[1]) + 1;
    auto active = [&](int i, int t) { return t >= first[i] && t <= last[i]; };
    bool ok = true;

    if (warp == 0) {
      {
        const bool one = elect_one();
        const int tiles = last[1] >= 0 ? 2 : 1;
        if (one) {
          tma_prefetch_desc(&tm_q);
          tma_prefetch_desc(&tm_kv);
          mbar_arrive_expect_tx(q_bar, tiles * NS * kQSlab);
        }
        for (int i = 0; i < tiles; ++i)
          for (int s = 0; s < NS; ++s)
            if (one) tma_load_2d(q_s + (i * NS + s) * kQSlab, s < 2 ? &tm_q : &tm_q2, q_bar, s < 2 ? head * a.q_step + 64 * s : head * 64, tok0 + q0 + i * kRows, kEvictNormal);
        int nk = 0, nv = 0;      // tiles of keys and values on their way
        auto keys = [&] {
          const int st = nk & 1;
          if (!warp_wait(k_empty(st), ((nk >> 1) & 1) ^ 1u)) return false;
          if (one) mbar_arrive_expect_tx(k_full(st), NS * kKSlab);
          for (int s = 0; s < NS; ++s)
            if (one) tma_load_2d(k_s + (st * NS + s) * kKSlab, s < 2 ? &tm_kv : &tm_k2, k_full(st), s < 2 ? a.k_off + kvh * a.k_step + 64 * s : 0, tok0 + (t_begin + nk) * kKeys,
                        kEvictLast);
          ++nk;
          return true;
        };
        ok = keys();
        for (int t = t_begin; ok && t < t_end; ++t) {
          if (t + 1 < t_end && !(ok = keys())) break;      // their product goes ahead of this tile's values
          const int st = nv & 1, row = tok0 + t * kKeys;
          if (!(ok = warp_wait(v_empty(st), ((nv >> 1) & 1) ^ 1u))) break;
          if (one) mbar_arrive_expect_tx(v_full(st), kVStage);
          for (int s = 0; s < 2; ++s)
            if (one) tma_load_2d(v_s + st * kVStage + s * kKSlab, &tm_kv, v_full(st), a.v_off + kvh * a.v_step + 64 * s, row, kEvictLast);
          if constexpr (LO)
            for (int s = 0; s < 2; ++s)
              if (one) tma_load_2d(v_s + st * kVStage + kVTile + s * kKSlab, &tm_v2, v_full(st), head * kD + 64 * s, row, kEvictLast);
          ++nv;
        }
        // the copies in flight land before the CTA ends, also where it gives up
        warp_wait(q_bar, 0);
        for (int j = max(0, nk - 2); j < nk; ++j) warp_wait(k_full(j & 1), (j >> 1) & 1);
        for (int j = max(0, nv - 2); j < nv; ++j) warp_wait(v_full(j & 1), (j >> 1) & 1);
      }
    } else if (warp == 9) {
      {
        const bool one = elect_one();
        // a product takes the tensor pipe 32 to 64 cycles: they are issued four at a time, with the descriptors that the loop needs at hand
        const uint32_t id_s = idesc_bf16(kRows, kKeys, 0), id_o = idesc_bf16(kRows, kD, 1);
        const uint64_t q_d = desc_sw128(q_s, 16, 1024), k_d = desc_sw128(k_s, 16, 1024), v_d = desc_sw128(v_s, kKSlab, 1024);
        auto scores = [&](int t) {
          const int it = t - t_begin, st = it & 1;
          if (!warp_wait(k_full(st), (it >> 1) & 1)) return false;
          tc_fence_after();
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (!active(i, t)) continue;
            if (one) {
#pragma unroll
              for (int s = 0; s < NS; ++s) umma_bf16_k64(tm_s(i, t & 1), q_d + (i * NS + s) * (kQSlab >> 4), k_d + (st * NS + s) * (kKSlab >> 4), id_s, s > 0 ? 1u : 0u);
              umma_commit(s_full(i, t & 1));
            }
          }
          if (one) umma_commit(k_empty(st));
          __syncwarp();
          return true;
        };
        ok = warp_wait(q_bar, 0) && scores(t_begin);
        for (int t = t_begin; ok && t < t_end; ++t) {
          const int it = t - t_begin, st = it & 1;
          // the next scores go to the other buffers, whose readers have handed in their P of the tile before this one
          if (t + 1 < t_end && !(ok = scores(t + 1))) break;
          if (!(ok = warp_wait(v_full(st), (it >> 1) & 1))) break;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (!active(i, t)) continue;
            if (!(ok = warp_wait(p_ready(i, t & 1), ((t - first[i]) >> 1) & 1))) break;
            tc_fence_after();
            if (one) {
              umma_bf16_tmem_k64(tm_o(i), tm_s(i, t & 1), v_d + st * (kVStage >> 4), id_o, t > first[i] ? 1u : 0u);
              if (LO) umma_bf16_tmem_k64(tm_o(i), tm_s(i, t & 1), v_d + st * (kVStage >> 4) + (kVTile >> 4), id_o, 1u);
              umma_commit(pv_full(i, t & 1));
            }
          }
          if (one) umma_commit(v_empty(st));
          __syncwarp();
        }
      }
    } else {
      const int gi = (warp - 1) >> 2, q = warp & 3, row = q * 32 + lane, p = q0 + gi * kRows + row;
      const bool valid = p < n;
      const int lo = max(0, p - a.window + 1);
      const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
      float ref = -INFINITY, l = 0.f;   // what the row's weights are relative to, in units of log 2
      const float mul = CAP ? 1.0f : a.scale * 1.4426950408889634f;
      // tanh x = 1 - 2 / (e^2x + 1)
      const float pre = CAP ? 2.0f * 1.4426950408889634f * a.scale / a.softcap : 0.f, cap2 = a.softcap * 1.4426950408889634f;
      auto capped = [&](uint32_t u) { return __float_as_uint(fmaf(-2.0f * cap2, rcp_ftz(exp2_ftz(__uint_as_float(u) * pre) + 1.0f), cap2)); };
      for (int t = first[gi]; ok && t <= last[gi]; ++t) {
        const int b = t & 1, kv0 = t * kKeys;
        if (!__all_sync(0xffffffffu, wait_limited(s_full(gi, b), ((t - first[gi]) >> 1) & 1))) { ok = false; break; }
        tc_fence_after();
        uint32_t s0[32], s1[32];
        tmem_ld_32x32(tm_s(gi, b) + lane_off, s0);
        tmem_ld_32x32(tm_s(gi, b) + lane_off + 32, s1);
        tmem_ld_wait();
        // scores stay as the product left them (under a cap: capped, in units of log 2); `mul` turns them into units of log 2
        if (CAP) {
#pragma unroll
          for (int c = 0; c < 32; ++c) { s0[c] = capped(s0[c]); s1[c] = capped(s1[c]); }
        }
        if (!valid || kv0 + kKeys - 1 > p || kv0 < lo) {
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const int j0 = kv0 + c, j1 = j0 + 32;
            if (!valid || j0 > p || j0 < lo) s0[c] = 0xff800000u;
            if (!valid || j1 > p || j1 < lo) s1[c] = 0xff800000u;
          }
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 32; c += 2)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            mx[k] = fmaxf(mx[k], __uint_as_float(s0[c + k]));
            mx[2 + k] = fmaxf(mx[2 + k], __uint_as_float(s1[c + k]));
          }
        const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * mul;
        float alpha = 1.f;
        if (top > ref) {
          alpha = exp2_ftz(ref - top);
          ref = top;
        }
        const float mu = ref == -INFINITY ? 0.f : ref;
        auto weight = [&](uint32_t u) { return exp2_ftz(fmaf(__uint_as_float(u), mul, -mu)); };
        float ps = 0.f;
        uint32_t pk[32];
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          const float p0 = weight(s0[c]), p1 = weight(s0[c + 1]);
          const float p2 = weight(s1[c]), p3 = weight(s1[c + 1]);
          const uint32_t a0 = pack_bf16x2(p0, p1), a1 = pack_bf16x2(p2, p3);
          // the sum is that of the rounded weights: their roundings then cancel in the quotient where the values agree
          ps += (__uint_as_float(a0 << 16) + __uint_as_float(a0 & 0xffff0000u)) + (__uint_as_float(a1 << 16) + __uint_as_float(a1 & 0xffff0000u));
          pk[c >> 1] = a0;
          pk[16 + (c >> 1)] = a1;
        }
        l = fmaf(l, alpha, ps);
        // P in place of the scores; the products in front of it may still be under way, those of this buffer's last P are not: the scores came behind them
        tmem_st_32x32(tm_s(gi, b) + lane_off, pk);
        if (t > first[gi] && __any_sync(0xffffffffu, alpha != 1.0f)) {
          if (!__all_sync(0xffffffffu, wait_limited(pv_full(gi, b ^ 1), ((t - first[gi] - 1) >> 1) & 1))) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int c0 = 0; c0 < kD; c0 += 32) {
            uint32_t v[32];
            tmem_ld_32x32(tm_o(gi) + lane_off + c0, v);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) * alpha);
            tmem_st_32x32(tm_o(gi) + lane_off + c0, v);
          }
        }
        tmem_st_wait();
        if (kv0 + kKeys > n && (gi == 0 || !active(0, t))) {
          // values behind the sequence's end: cleared before the first product that reads the tile (that of row tile 0, where it is active)
          const int it = t - t_begin;
          if (!__all_sync(0xffffffffu, wait_limited(v_full(it & 1), (it >> 1) & 1))) { ok = false; break; }
          const int r = row & 63;
          if (kv0 + r >= n) {
            uint4* d = reinterpret_cast<uint4*>(smem + (v_s - sbase) + (it & 1) * kVStage + (row >> 6) * kKSlab + r * 128);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              d[c] = make_uint4(0, 0, 0, 0);
              if (LO) d[kVTile / 16 + c] = make_uint4(0, 0, 0, 0);
            }
          }
          fence_proxy_async();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_ready(gi, b));
      }
      if (ok && last[gi] >= 0) ok = __all_sync(0xffffffffu, wait_limited(pv_full(gi, last[gi] & 1), ((last[gi] - first[gi]) >> 1) & 1));
      if (ok && last[gi] >= 0) {
        tc_fence_after();
        bool finite = true;
        float inv = l > 0.f ? 1.f / l : 0.f;
        if (a.sink) {
          const float sk = a.sink[head] * 1.4426950408889634f, mm = fmaxf(ref, sk), back = exp2f(ref - mm);
          inv = back / fmaf(l, back, exp2f(sk - mm));
        }
        const long long tok = tok0 + p;
        if (a.gate && valid) inv *= 1.0f / (1.0f + expf(-__bfloat162float(static_cast<const bf16*>(a.gate)[tok * a.ldg + head])));
        inv *= a.out_scale;
        bf16* dst = static_cast<bf16*>(a.y) + tok * a.ldy + head * kD;
#pragma unroll
        for (int c0 = 0; c0 < kD; c0 += 32) {
          uint32_t v[32];
          tmem_ld_32x32(tm_o(gi) + lane_off + c0, v);
          tmem_ld_wait();
          if (valid) {
#pragma unroll
            for (int c = 0; c < 32; ++c) finite = finite && (v[c] & 0x7f800000u) != 0x7f800000u;
#pragma unroll
            for (int c = 0; c < 32; c += 8)
              *reinterpret_cast<uint4*>(dst + c0 + c) =
                  make_uint4(pack_bf16x2(__uint_as_float(v[c]) * inv, __uint_as_float(v[c + 1]) * inv), pack_bf16x2(__uint_as_float(v[c + 2]) * inv, __uint_as_float(v[c + 3]) * inv),
                             pack_bf16x2(__uint_as_float(v[c + 4]) * inv, __uint_as_float(v[c + 5]) * inv), pack_bf16x2(__uint_as_float(v[c + 6]) * inv, __uint_as_float(v[c + 7]) * inv));
          }
        }
        if (valid && !finite) plain_row<NS, CAP>(a, tok0, p, head, kvh, first[gi] * kKeys, min(n, (last[gi] + 1) * kKeys));
      }
    }
    if (!ok && a.error) *reinterpret_cast<volatile int*>(a.error) = 1;
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <int NS, bool CAP>
int launch(const PromptAttnArgs& a, const CUtensorMap& q, const CUtensorMap& q2, const CUtensorMap& kv, const CUtensorMap& k2, const CUtensorMap& v2, cudaStream_t st) {
  static std::atomic<unsigned long long> attr{0};
  constexpr int smem = smem_bytes<NS>();
  if (!ensure_dynamic_smem(prompt_attn_kernel<NS, CAP>, smem, &attr)) return -2;
  prompt_attn_kernel<NS, CAP><<<dim3(a.heads, a.T / (2 * kRows) + a.nseq), kThreads, smem, st>>>(q, q2, kv, k2, v2, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

__device__ __forceinline__ float rotated(const bf16* u, int i, int half, bool half_pairs, const float2* cs) {
  const float v = __bfloat162float(u[i]);
  if (i >= 2 * half) return v;
  const bool high = half_pairs ? i >= half : (i & 1);
  const float w = __bfloat162float(u[half_pairs ? (high ? i - half : i + half) : i ^ 1]);
  const float2 c = cs[half_pairs ? (high ? i - half : i) : i >> 1];
  return high ? fmaf(v, c.x, w * c.y) : fmaf(v, c.x, -w * c.y);
}

// one CTA per token: the cached latent and rotated key part, side by side with the other tokens', and the queries' rotated parts
__global__ void __launch_bounds__(128) latent_prompt_prep_kernel(LatentPromptPrepArgs a) {
  const long long t = blockIdx.x;
  const int C = a.kv_rank, R = a.rot_dim;
  const uint4* row = reinterpret_cast<const uint4*>(static_cast<const bf16*>(a.cache) + static_cast<long long>(a.slots[t]) * (C + R));
  uint4 *c = reinterpret_cast<uint4*>(static_cast<bf16*>(a.c) + t * C), *k2 = reinterpret_cast<uint4*>(static_cast<bf16*>(a.k2) + t * R);
  for (int i = threadIdx.x; i < (C + R) / 8; i += blockDim.x) {
    if (i < C / 8) c[i] = row[i];
    else k2[i - C / 8] = row[i];
  }
  const float2* cs = a.rope + static_cast<long long>(a.positions[t]) * (a.rot_dims / 2);
  const bf16* q = static_cast<const bf16*>(a.q) + t * a.ldq;
  bf16* q2 = static_cast<bf16*>(a.q2) + t * a.heads * R;
  for (int e = threadIdx.x; e < a.heads * R; e += blockDim.x) {
    const int h = e / R, i = e - h * R;
    q2[e] = __float2bfloat16_rn(rotated(q + h * (a.dim + R) + a.dim, i, a.rot_dims / 2, a.half_pairs, cs));
  }
}

// one CTA per token
__global__ void __launch_bounds__(128) window_prompt_prep_kernel(const uint4* cache, const int* slots, const float4* qn, uint4* kv, uint4* q, int kv_pieces, int q_pieces) {
  const long long t = blockIdx.x, row = slots[t];
  for (int i = threadIdx.x; i < kv_pieces; i += blockDim.x) kv[t * kv_pieces + i] = cache[row * kv_pieces + i];
  for (int i = threadIdx.x; i < q_pieces; i += blockDim.x) {
    const float4 a = qn[(t * q_pieces + i) * 2], b = qn[(t * q_pieces + i) * 2 + 1];
    q[t * q_pieces + i] = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
  }
}

// per head: rows 0 .. 127 W_uk (kept transposed), rows 128 .. 255 W_uv
__global__ void latent_stack_kernel(const bf16* uk_t, const bf16* uv, bf16* out, int C, long long total) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int c = static_cast<int>(i % C);
  const long long r = i / C, h = r / (2 * kD);
  const int d = static_cast<int>(r % (2 * kD));
  out[i] = d < kD ? uk_t[(h * C + c) * kD + d] : uv[(h * kD + d - kD) * C + c];
}

}  // namespace

bool prompt_attention_fits(const PromptAttnArgs& a) {
  auto al = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  return gemm_variant() == 2 && a.heads > 0 && a.kv_heads > 0 && a.heads % a.kv_heads == 0 && a.ldq % 8 == 0 && a.q_step % 8 == 0 && a.ldkv % 8 == 0 && a.k_off % 8 == 0 &&
         a.k_step % 8 == 0 && a.v_off % 8 == 0 && a.v_step % 8 == 0 && a.ldy % 8 == 0 && al(a.q) && al(a.q2) && al(a.kv) && al(a.k2) && al(a.v2) && al(a.y) && !a.q2 == !a.k2 && !a.q2 == !a.v2 && (!a.v2 || a.kv_heads == a.heads) &&
         a.window > 0 && a.softcap >= 0.f && a.scale > 0.f;
}

int prompt_attention(const PromptAttnArgs& a, cudaStream_t st) {
  if (a.T <= 0 || a.nseq <= 0) return 0;
  if (!prompt_attention_fits(a)) return -1;
  CUtensorMap q, q2, kv, k2, v2;
  const int kcols = a.k_off + (a.kv_heads - 1) * a.k_step + kD, vcols = a.v_off + (a.kv_heads - 1) * a.v_step + kD;
  if (tmap_encode_bf16_2d(&q, a.q, a.T, (a.heads - 1) * a.q_step + kD, a.ldq, kRows, 64, 1) ||
      tmap_encode_bf16_2d(&kv, a.kv, a.T, kcols > vcols ? kcols : vcols, a.ldkv, kKeys, 64, 1)) return -2;
  if (!a.q2) return a.softcap > 0.f ? launch<2, true>(a, q, q, kv, kv, kv, st) : launch<2, false>(a, q, q, kv, kv, kv, st);
  if (tmap_encode_bf16_2d(&q2, a.q2, a.T, a.heads * 64, a.heads * 64, kRows, 64, 1) || tmap_encode_bf16_2d(&k2, a.k2, a.T, 64, 64, kKeys, 64, 1) ||
      tmap_encode_bf16_2d(&v2, a.v2, a.T, a.heads * kD, a.heads * kD, kKeys, 64, 1)) return -2;
  return a.softcap > 0.f ? launch<3, true>(a, q, q2, kv, k2, v2, st) : launch<3, false>(a, q, q2, kv, k2, v2, st);
}

int latent_prompt_prep(const LatentPromptPrepArgs& a, cudaStream_t st) {
  if (a.T <= 0) return 0;
  if (a.kv_rank % 8 || a.rot_dim % 8 || a.rot_dims > a.rot_dim) return -1;
  latent_prompt_prep_kernel<<<a.T, 128, 0, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int window_prompt_prep(const void* cache, const int* slots, const float* qn, void* kv, void* q, int T, int heads, int kv_heads, cudaStream_t st) {
  if (T <= 0) return 0;
  window_prompt_prep_kernel<<<T, 128, 0, st>>>(static_cast<const uint4*>(cache), slots, reinterpret_cast<const float4*>(qn), static_cast<uint4*>(kv), static_cast<uint4*>(q),
                                               kv_heads * 2 * kD / 8, heads * kD / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

size_t window_prompt_ws_bytes(int rows, int heads, int kv_heads) { return static_cast<size_t>(rows) * (heads + 2 * kv_heads) * kD * 2; }

// Measured with 16 query and 4 key heads under a cap, window kernel on mma.sync -> this one with its gather, in us: one prompt of 32
// tokens 22 -> 14, of 128 26 -> 15, of 512 49 -> 31; 64 prompts of 64 95 -> 66, 16 of 128 56 -> 29, 8 of 512 127 -> 58; 4095
// tokens under a window of 1024 211 -> 95.  Many prompts of 32 fill a quarter of a CTA's 128 rows and break even (64 of them
// 63 -> 62, 32 of them 32 -> 35): below 64 tokens only while one wave of CTAs holds them all.
bool window_prompt_pays(int T, int nseq, int heads) {
  static const int least = [] { const char* e = getenv("B200_WINDOW_PROMPT"); return e ? atoi(e) : 32; }();   // A/B knob: fewest tokens a prompt, 0 = never
  const long long n = nseq;
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
  return least > 0 && T >= least * n && (T >= 2 * least * n || n * heads <= sms);
}

bool latent_prompt_fits(int dim, int vdim, int rot_dim, int kv_rank) {
  return dim == kD && vdim == kD && rot_dim == 64 && kv_rank >= kD && kv_rank % 8 == 0;
}

// Measured with 16 heads, latent-space form -> this one, in us: one prompt of 40 tokens 42 -> 25, of 128 50 -> 28, of 512
// 122 -> 47; 64 prompts of 32 223 -> 90, 128 of 16 275 -> 156, 512 of 8 1008 -> 670, 512 of 2 566 -> 619, 256 of 1 170 -> 267: a
// quarter of a CTA's 128 rows is where it wins by half, a few tokens a prompt are where it loses.  Error against 64 bits, of the
// output: 2.8e-3 -> 2.4e-3 at 64 tokens, 2.3e-3 -> 2.1e-3 at 8, 2.4e-3 -> 1.8e-3 at 2 (with values in one term 2.6e-3 at 8).
bool latent_prompt_pays(int T, int nseq) {
  static const int least = [] { const char* e = getenv("B200_LATENT_PROMPT"); return e ? atoi(e) : 32; }();   // A/B knob: fewest tokens a prompt, 0 = never
  return least > 0 && T >= static_cast<long long>(least) * nseq;
}

int latent_prompt_stack(const void* uk_t, const void* uv, void* out, int heads, int kv_rank, cudaStream_t st) {
  const long long total = static_cast<long long>(heads) * 2 * kD * kv_rank;
  latent_stack_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, st>>>(static_cast<const bf16*>(uk_t), static_cast<const bf16*>(uv), static_cast<bf16*>(out), kv_rank, total);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace b200
