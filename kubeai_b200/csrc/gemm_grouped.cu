// Grouped projection GEMM for mixtures of experts (tcgen05 cta_group::2): the rows of every expert, sorted by expert, times
// that expert's matrix, in ONE launch whose tile list is read from device memory.
//     out[r, n] = sum_k X[r, k] * W[e(r) * N + n, k]        (bf16 x bf16 -> fp32 -> bf16)
// X holds the rows of expert e at [first_e, first_e + rows_e) (the table moe_align leaves, so no count ever travels to the
// host); W is the experts' matrices stacked row-wise.  What leaves the accumulators (gemm.h GroupedOut): the bf16 rounding of
// bias and activation on the fp32 sums, the fp32 sums themselves, or a gated unit, for which the rows of W alternate in blocks
// of 64 gate rows and their 64 up rows and the output has half as many columns.
//
// A CTA pair works on a tile of 256 weight rows x up to 2 * box rows of one expert; an expert's rows are cut into equal tiles.
// box, the rows of X that a CTA stages per k-block, is 16 to 128: a step of few tokens reads the weights once and is bound by
// how fast an SM can take them in through TMA, and every byte of X that its tile does not need would come off that rate.
// (24 tokens, 16 experts of 2 x 2048 x 2048, two a token: 128-row boxes move as many bytes of X as of weights.)  The ring
// takes as many stages as fit beside the output staging.
// Work items run expert by expert, weight tile by weight tile with its row tiles side by side, so that neighbouring pairs use
// one weight slab at the same time, and are dealt to the pairs in turn.  Per CTA: one producer thread (TMA: its own 128
// weight rows and its half of the row tile), one issuing thread in the leader, four or eight epilogue warps that drain one of two
// accumulators while the other is being filled.  Every wait has an iteration limit: a pair that gives up stops its work, sets
// an error flag for the host, and still meets its peer before the tensor memory is freed.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "activations.cuh"
#include "dispatch_rules.h"
#include "gemm.h"
#include "launch.h"
#include "ptx.cuh"
#include "umma2.cuh"

namespace b200 {
namespace {

typedef __nv_bfloat16 bf16;
constexpr int kSlab = 128;      // weight rows per CTA
constexpr int kRows = 256;      // rows of X per tile, at most; TMEM columns of one accumulator
constexpr int kBlockK = 64;
// A warp that loads, one that issues the products, and one or two groups of four that drain a tile's rows in turns.  Two where
// the drain of one group outlasts the next tile's products: gated units with the accurate functions (4096 tokens, 16 experts of 4096 x
// 2048, two a token: 133 us with one group, 122 with two; one such matrix for all 70 and 58; of 500 tokens with K cut, 27 and 21) and
// the sums of two terms (34, 28).  The others keep one, whose rounds of 64 rows pass fewer barriers (Llama's gated product of 2048 tokens 310 us, 317 with two).
__host__ __device__ constexpr int groups_of(int epi) { return epi == 1 || epi == 6 ? 2 : 1; }
__host__ __device__ constexpr int threads_of(int epi) { return 64 + groups_of(epi) * 128; }
constexpr int kABytes = kSlab * kBlockK * 2;
constexpr int kRingBytes = 6 * (kABytes + kRows / 2 * kBlockK * 2), kMaxStages = 10;
constexpr int kOutRows = 64;    // rows of X in the output staging, twice: an epilogue round of one group (32 rows with fp32 output), or of two
constexpr int kOutBytes = kOutRows * kSlab * 2;
constexpr int kSmem = 1024 + kRingBytes + 256 + 2 * kOutBytes;
__host__ __device__ constexpr int stage_bytes(int box) { return kABytes + box * kBlockK * 2; }
__host__ __device__ constexpr int stages_for(int box) { return kRingBytes / stage_bytes(box) < kMaxStages ? kRingBytes / stage_bytes(box) : kMaxStages; }
static_assert(stages_for(128) == 6 && stages_for(16) == kMaxStages, "ring depths");
static_assert(8 * (2 * kMaxStages + 4) + 4 <= 256, "the barriers fit in front of the output staging");
constexpr int kWaitLimit = 1 << 22;

struct Tile {
  int wrow;      // first row of the stacked weight matrix
  int n0;        // the same within the expert's matrix
  int row0;      // first row of X
  int rows;      // rows of X (at most kRows)
  int id;        // number of the tile (one matrix)
  int part;      // which part of K
  int kb0, kb1;  // its 64-wide steps
};

// Walks this pair's items: `next` advances by one item of the pair, expert by expert.
struct Walk {
  const int* expert_rows;
  int experts, mt, N, rows, tile;   // without a table: one matrix, `rows` rows from 0; tile: rows of a tile at most
  int parts, KB;                    // K in parts (one matrix only), in 64-wide steps
  int e = 0;
  long long base = 0;    // items of the experts before e
  __device__ bool at(long long item, Tile* t) {
    while (e < experts) {
      const int cnt = expert_rows ? expert_rows[2 * e + 1] : rows;
      const int ntt = (cnt + tile - 1) / tile;
      const long long n = static_cast<long long>(ntt) * mt * parts;
      if (item < base + n) {
        int r = static_cast<int>(item - base);
        t->part = 0; t->kb0 = 0; t->kb1 = KB;
        if (parts > 1) {
          t->id = r / parts;
          t->part = r - t->id * parts;
          t->kb0 = KB * t->part / parts;
          t->kb1 = KB * (t->part + 1) / parts;
          r = t->id;
        }
        const int m = r / ntt, tt = r - m * ntt;
        const int per = ((cnt + ntt - 1) / ntt + 15) & ~15;     // equal tiles, whole 16-row steps (at most `tile`)
        t->n0 = m * 2 * kSlab;
        t->wrow = e * N + t->n0;
        t->row0 = (expert_rows ? expert_rows[2 * e] : 0) + tt * per;
        t->rows = min(per, cnt - tt * per);
        if (t->rows > 0) return true;
        t->rows = 0;       // rounding up to 16 may leave the last tile of an expert empty
        return true;
      }
      base += n;
      ++e;
    }
    return false;
  }
};

__device__ __forceinline__ bool wait_limited(uint32_t bar, uint32_t parity) { return mbar_wait_limited(bar, parity, kWaitLimit); }
// ... by a whole warp: whether all lanes saw the phase end
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, wait_limited(bar, parity)); }
template <int EPI>
__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, %0;" ::"n"(groups_of(EPI) * 128) : "memory"); }
// whether all epilogue threads say yes (they also meet here)
template <int EPI>
__device__ __forceinline__ bool all_epilogue(bool v) {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 p, %1, 0;\n"
      "barrier.cta.red.and.pred q, 2, %2, p;\n"
      "selp.u32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(r)
      : "r"(v ? 1u : 0u), "n"(groups_of(EPI) * 128)
      : "memory");
  return r != 0;
}

// Split K (one matrix, and fewer tiles than pairs): a tile's K is cut into parts, an item each, side by side on neighbouring
// pairs.  Every part leaves its fp32 sums in the workspace and counts itself in; the part that comes last adds all of them
// in their order and goes on to the epilogue, so nobody waits for anybody and the sum does not depend on who came last.
struct SplitK {
  float* ws;       // [tile][part][rank][rows of the tile][128]
  int* counters;   // [tile][rank], zero between launches
  int parts;
  int tile;        // rows of a tile
};
template <int EPI>
constexpr bool gates = EPI == 1 || EPI == 5 || EPI == 7;
// EPI 5: SiLU rounded to bf16 before the product, the rounding points of the Llama path's own kernel (elementwise.cu silu_mul)
template <int EPI>
__device__ __forceinline__ float gated(float g, float u, bool clamp, const GroupedOut& o) {
  return EPI == 5 ? __bfloat162float(silu_bf16(g)) * u : gated_unit<EPI == 7>(g, u, clamp, o.p0, o.p1, o.p2);
}
__device__ __forceinline__ float left_over(float s) { return s - __bfloat162float(__float2bfloat16_rn(s)); }
// Eight neighbouring columns of one row: the parts' sums added in their order.
__device__ __forceinline__ void add_parts(float* v, const float* p, int step, int parts) {
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = 0.f;
  for (int k = 0; k < parts; ++k) {
    const float4 a = *reinterpret_cast<const float4*>(p + k * step), b = *(reinterpret_cast<const float4*>(p + k * step) + 1);
    v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
    v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
  }
}
__device__ __forceinline__ void store8(bf16* p, const float* v) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}
// n rows of a split tile, their parts in shared memory, to the rows from row0 of the output: a thread takes eight columns of a row
template <int EPI>
__device__ __forceinline__ void finish_rows(const float* sums, int step, int parts, int n, int row0, int n0, int N, const GroupedOut& o, int et) {
  constexpr int kPieces = gates<EPI> ? 8 : 16;
  for (int it = et; it < n * kPieces; it += groups_of(EPI) * 128) {
    const int j = it / kPieces, c = (it % kPieces) * 8;
    const float* p = sums + j * kSlab + c;
    const size_t r = row0 + j;
    float v[8];
    if constexpr (gates<EPI>) {
      if (n0 + kSlab > N) continue;
      float u[8];
      add_parts(v, p, step, parts);
      add_parts(u, p + 64, step, parts);
      const bool clamp = o.p0 < INFINITY;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        v[i] = gated<EPI>(__bfloat162float(__float2bfloat16_rn(v[i])), __bfloat162float(__float2bfloat16_rn(u[i])), clamp, o);
      store8(static_cast<bf16*>(o.y) + r * o.ldy + n0 / 2 + c, v);
    } else {
      if (n0 + c >= N) continue;
      add_parts(v, p, step, parts);
      if ((EPI == 3 || EPI == 4) && o.bias) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (n0 + c + i < N) v[i] += __ldg(o.bias + n0 + c + i);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (EPI == 3 && o.epi == GROUPED_RELU2) v[i] = fmaxf(v[i], 0.f) * fmaxf(v[i], 0.f);
        if (EPI == 4) v[i] = xielu_fast(v[i], o.p0, o.p1);
      }
      store8(static_cast<bf16*>(o.y) + r * o.ldy + n0 + c, v);
      if (EPI == 6 && (n0 & kSlab)) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = left_over(v[i]);
        store8(static_cast<bf16*>(o.y2) + r * (N / 2) + (n0 - kSlab) / 2 + c, v);
      }
    }
  }
}
// The epilogue of a split tile, from the workspace (`first`: the tile's first part, `step` floats to the next).  The parts come
// through the operand ring, which is free (a split launch gives a pair one item), by cp.async: with plain loads the registers
// bound what is in flight, and 256 rows in two parts took 25 us where this takes 13.
template <int EPI>
__device__ __forceinline__ void finish_parts(float* ring, const float* first, size_t step, int parts, const Tile& t, int n0, int N, const GroupedOut& o, int et) {
  const int chunk = min(t.rows, kRingBytes / (kSlab * 4) / parts), sstep = chunk * kSlab;      // rows a round brings in
  const uint32_t sring = smem_u32(ring);
  for (int r0 = 0; r0 < t.rows; r0 += chunk) {
    const int n = min(chunk, t.rows - r0);
    for (int k = 0; k < parts; ++k)
      for (int it = et; it < n * (kSlab / 4); it += groups_of(EPI) * 128)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sring + (k * sstep + it * 4) * 4), "l"(first + k * step + r0 * kSlab + it * 4) : "memory");
    asm volatile("cp.async.wait_all;" ::: "memory");
    epilogue_sync<EPI>();
    finish_rows<EPI>(ring, sstep, parts, n, t.row0 + r0, n0, N, o, et);
    epilogue_sync<EPI>();
  }
}

// EPI 0: bf16(sum); 1: the gated unit; 2: fp32 sum + bias; 3: bf16(relu2(sum + bias)), or without an activation; 4: bf16(xielu(sum + bias));
// 5: the SiLU-gated unit with its inner rounding; 6: bf16(sum), and of the pair's second slab what that rounding left;
// 7: the gated unit with fast functions, for the design whose units are formed so in every kernel with an epilogue (Dabodra; 4095 tokens 1577 us,
// 1659 with the accurate ones: a tile's drain then outlasts the next tile's products).
// A form of its own for the plain product: looking the activation up per element made its drain a sixth of the launch longer.
// FULL: 128-row boxes, their sizes known to the compiler.
template <int EPI, bool FULL>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(threads_of(EPI), 1)
gemm_grouped_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const int* expert_rows, int experts, int rows,
                    const __grid_constant__ GroupedOut o, int N, int K, int box_rows, const __grid_constant__ SplitK split, int* error) {
  constexpr int G = groups_of(EPI), kTurn = EPI == 2 ? 32 : kOutRows / G;      // groups, rows of a round
  const int box = FULL ? 128 : box_rows, stages = stages_for(box);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar_base = smem_base + kRingBytes, stage_step = stage_bytes(box);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };                     // the leader's copy is the live one
  auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };        // both CTAs
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * kMaxStages + a); };    // both CTAs
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * kMaxStages + 2 + a); };   // the leader's copy
  const uint32_t tmem_slot = bar_base + 8u * (2 * kMaxStages + 4);
  uint8_t* stage_out = smem_raw + (bar_base + 256 - smem_u32(smem_raw));
  const int warp = warp_number(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int units = gridDim.x >> 1, unit = blockIdx.x >> 1, KB = (K + kBlockK - 1) / kBlockK;
  Walk walk;
  walk.expert_rows = expert_rows; walk.experts = experts; walk.mt = (N + 2 * kSlab - 1) / (2 * kSlab); walk.N = N; walk.rows = rows;
  walk.tile = split.tile; walk.parts = split.parts; walk.KB = KB;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
  }
  if (warp == 1) {
    if (lane == 0) {
      for (int s = 0; s < stages; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
      for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar(a), 1); mbar_init(tempty_bar(a), 8 * G); }   // the epilogue warps of both CTAs
      fence_mbar_init();
    }
    __syncwarp();
    tmem_alloc2(tmem_slot, 512);
    tmem_relinquish2();
  }
  tc_fence_before();
  cluster_sync_all();   // barrier inits and the TMEM allocation are visible to the peer
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  bool ok = true;
  griddep_launch();
  // Every role walks the table.  Without one only the loading thread has something to do before the kernel in front has ended; the
  // others wait for that here, so that no limited wait below runs out over the length of another kernel.
  if (expert_rows || warp != 0) griddep_wait();

  if (warp == 0) {
    const bool one = elect_one();
    int stage = 0, ahead = 0, filled = 0;
    uint32_t phase = 0;
    Tile t;
    auto load_w = [&](int st, int kb) {
      if (!one) return;
      if (leader) mbar_arrive_expect_tx(full_bar(st), 2u * stage_step);
      tma_load_2d_pair(smem_base + st * stage_step, &tm_w, full_bar(st), kb * kBlockK, t.wrow + static_cast<int>(rank) * kSlab, kEvictNormal);
    };
    if (!expert_rows) {
      // the weights do not wait for the kernel in front: the ring's first stages of them are on their way before it ends
      if (walk.at(unit, &t) && t.rows)
        for (; ahead < min(stages, t.kb1 - t.kb0); ++ahead) load_w(ahead, t.kb0 + ahead);
      griddep_wait();
    }
    for (long long item = unit; ok && walk.at(item, &t); item += units) {
      if (!t.rows) continue;
      const int nc = (t.rows + 15) & ~15;
      for (int kb = t.kb0; kb < t.kb1; ++kb) {
        const uint32_t sa = smem_base + stage * stage_step;
        if (ahead > 0) {
          --ahead;
        } else {
          if (!warp_wait(empty_bar(stage), phase ^ 1u)) { ok = false; break; }
          load_w(stage, kb);
        }
        filled = min(filled + 1, stages);
        // this CTA stages the rank-th half of the row tile (rows of the box past nc / 2 are not used)
        if (one) tma_load_2d_pair(sa + kABytes, &tm_x, full_bar(stage), kb * kBlockK, t.row0 + static_cast<int>(rank) * (nc >> 1), kEvictLast);
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
    }
    // The copies started last have landed before the CTA ends, also where a role gave up: the leader's barriers count both CTAs'
    // bytes.  (Where none did, they were waited for long ago.)
    if (leader)
      for (int i = 0; i < filled; ++i) {
        if (--stage < 0) { stage = stages - 1; phase ^= 1u; }
        wait_limited(full_bar(stage), phase);
      }
    __syncwarp();
  } else if (warp == 1) {
    if (leader) {
      const bool one = elect_one();
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      Tile t;
      for (long long item = unit; ok && walk.at(item, &t); item += units) {
        if (!t.rows) continue;
        const uint32_t idesc = umma_idesc_bf16(2 * kSlab, (t.rows + 15) & ~15);
        if (!warp_wait(tempty_bar(acc), acc_phase ^ 1u)) { ok = false; break; }
        tc_fence_after();
        for (int kb = t.kb0; kb < t.kb1; ++kb) {
          if (!warp_wait(full_bar(stage), phase)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_base + stage * stage_step;
          const uint64_t a_desc = umma_desc_kmajor_sw128(sa), b_desc = umma_desc_kmajor_sw128(sa + kABytes);
          if (one) {
            umma2_bf16_k64(tmem_base + acc * kRows, a_desc, b_desc, idesc, kb > t.kb0 ? 1u : 0u);
            umma2_commit_pair(empty_bar(stage), 3);
            if (kb == t.kb1 - 1) umma2_commit_pair(tfull_bar(acc), 3);
          }
          __syncwarp();
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else {
    const int q = warp & 3, row = q * 32 + lane, ea = threadIdx.x - 64, grp = ea >> 7, et = ea & 127;
    auto group_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(3 + grp) : "memory"); };
    int acc = 0, sbuf = 0;
    uint32_t acc_phase = 0;
    Tile t;
    for (long long item = unit; ok && walk.at(item, &t); item += units) {
      if (!t.rows) continue;
      ok = all_epilogue<EPI>(wait_limited(tfull_bar(acc), acc_phase));
      if (!ok) break;
      tc_fence_after();
      const int n0 = t.n0 + static_cast<int>(rank) * kSlab;    // first column of this CTA's slab in the expert's output
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * kRows;
      const float bias = EPI >= 2 && EPI <= 4 && o.bias && n0 + row < N ? __ldg(o.bias + n0 + row) : 0.f;   // a thread's accumulator row is one output column
      const bool relu2 = EPI == 3 && o.epi == GROUPED_RELU2;
      bool whole = true;
      if (EPI != 2 && split.parts > 1) {
        whole = false;
        const size_t slab = static_cast<size_t>(split.tile) * kSlab;
        float* first = split.ws + (static_cast<size_t>(t.id) * split.parts * 2 + rank) * slab;
        float* mine = first + 2 * t.part * slab + row;
        for (int c0 = 32 * grp; c0 < t.rows; c0 += 32 * G) {
          uint32_t v[32];
          tmem_ld_32x32(taddr + c0, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c0 + j < t.rows) __stcg(mine + static_cast<size_t>(c0 + j) * kSlab, __uint_as_float(v[j]));
        }
        __threadfence();
        epilogue_sync<EPI>();
        bool last = false;
        if (ea == 0) {
          last = atomicAdd(split.counters + 2 * t.id + rank, 1) == split.parts - 1;
          if (last) split.counters[2 * t.id + rank] = 0;
          __threadfence();
        }
        last = !all_epilogue<EPI>(!last);       // thread 0's answer reaches all
        if constexpr (EPI != 2)
          if (last) finish_parts<EPI>(reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw))), first, 2 * slab, split.parts, t, n0, N, o, ea);
      }
      for (int c0 = grp * kTurn; whole && c0 < t.rows; c0 += G * kTurn) {
        const bool two = kTurn == 64 && c0 + 32 < t.rows;
        uint32_t v0[32], v1[kTurn == 64 ? 32 : 1];
        tmem_ld_32x32(taddr + c0, v0);
        if constexpr (kTurn == 64) {
          if (two) tmem_ld_32x32(taddr + c0 + 32, v1);
        }
        tmem_ld_wait();
        uint8_t* stage = stage_out + (2 * grp + sbuf) * (kOutBytes / G);
        const int left = t.rows - c0;
        if constexpr (EPI == 2) {
          float* sf = reinterpret_cast<float*>(stage);
#pragma unroll
          for (int j = 0; j < 32; ++j) sf[j * kSlab + row] = __uint_as_float(v0[j]) + bias;
        } else {
          bf16* sb = reinterpret_cast<bf16*>(stage);
          auto put = [&](int j, uint32_t u) {
            float v = __uint_as_float(u);
            if (EPI == 3 || EPI == 4) v += bias;
            if (EPI == 3) v = relu2 ? fmaxf(v, 0.f) * fmaxf(v, 0.f) : v;
            if (EPI == 4) v = xielu_fast(v, o.p0, o.p1);
            sb[j * kSlab + row] = __float2bfloat16_rn(v);
          };
#pragma unroll
          for (int j = 0; j < 32; ++j) put(j, v0[j]);
          if constexpr (kTurn == 64) {
            if (two) {
#pragma unroll
              for (int j = 0; j < 32; ++j) put(32 + j, v1[j]);
            }
          }
        }
        // one barrier per round: a thread past it has finished its pass over the buffer staged two rounds ago
        group_sync();
        if constexpr (EPI == 2) {
          float* dst = static_cast<float*>(o.y) + static_cast<size_t>(t.row0 + c0) * o.ldy;
          const float* sf = reinterpret_cast<const float*>(stage);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int it = et + i * 128, j = it >> 5, c = (it & 31) * 4;
            if (j < left && n0 + c < N)
              *reinterpret_cast<float4*>(dst + static_cast<size_t>(j) * o.ldy + n0 + c) = *reinterpret_cast<const float4*>(sf + j * kSlab + c);
          }
        } else if constexpr (gates<EPI>) {
          // rows 0..63 of the slab are gate rows, 64..127 the matching up rows: output columns n0 / 2 ..
          bf16* dst = static_cast<bf16*>(o.y) + static_cast<size_t>(t.row0 + c0) * o.ldy;
          const bf16* sb = reinterpret_cast<const bf16*>(stage);
          const bool clamp = o.p0 < INFINITY;
#pragma unroll
          for (int i = 0; i < kTurn / 16; ++i) {
            const int it = et + i * 128, j = it >> 3, c = (it & 7) * 8;
            if (j < left && n0 + kSlab <= N) {
              const uint4 g = *reinterpret_cast<const uint4*>(sb + j * kSlab + c), u = *reinterpret_cast<const uint4*>(sb + j * kSlab + 64 + c);
              const uint32_t gu[4] = {g.x, g.y, g.z, g.w}, uu[4] = {u.x, u.y, u.z, u.w};
              uint32_t r[4];
#pragma unroll
              for (int k = 0; k < 4; ++k)
                r[k] = pack_bf16x2(gated<EPI>(__uint_as_float(gu[k] << 16), __uint_as_float(uu[k] << 16), clamp, o),
                                   gated<EPI>(__uint_as_float(gu[k] & 0xffff0000u), __uint_as_float(uu[k] & 0xffff0000u), clamp, o));
              *reinterpret_cast<uint4*>(dst + static_cast<size_t>(j) * o.ldy + n0 / 2 + c) = make_uint4(r[0], r[1], r[2], r[3]);
            }
          }
        } else {
          bf16* dst = static_cast<bf16*>(o.y) + static_cast<size_t>(t.row0 + c0) * o.ldy;
          const bf16* sb = reinterpret_cast<const bf16*>(stage);
#pragma unroll
          for (int i = 0; i < kTurn / 8; ++i) {
            const int it = et + i * 128, j = it >> 4, c = (it & 15) * 8;
            if (j < left && n0 + c < N)
              *reinterpret_cast<uint4*>(dst + static_cast<size_t>(j) * o.ldy + n0 + c) = *reinterpret_cast<const uint4*>(sb + j * kSlab + c);
          }
          if (EPI == 6 && rank == 1) {      // one more round for the second terms
            sbuf ^= 1;
            bf16* s2 = reinterpret_cast<bf16*>(stage_out + (2 * grp + sbuf) * (kOutBytes / G));
#pragma unroll
            for (int j = 0; j < 32; ++j) s2[j * kSlab + row] = __float2bfloat16_rn(left_over(__uint_as_float(v0[j])));
            group_sync();
            bf16* d2 = static_cast<bf16*>(o.y2) + static_cast<size_t>(t.row0 + c0) * (N / 2) + t.n0 / 2;
#pragma unroll
            for (int i = 0; i < kTurn / 8; ++i) {
              const int it = et + i * 128, j = it >> 4, c = (it & 15) * 8;
              if (j < left) *reinterpret_cast<uint4*>(d2 + static_cast<size_t>(j) * (N / 2) + c) = *reinterpret_cast<const uint4*>(s2 + j * kSlab + c);
            }
          }
        }
        sbuf ^= 1;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (leader) mbar_arrive(tempty_bar(acc));
        else mbar_arrive_cluster_relaxed(tempty_bar(acc), 0);
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  }
  if (!ok && error) *reinterpret_cast<volatile int*>(error) = 1;
  tc_fence_before();
  __syncwarp();
  cluster_sync_all();   // nobody of the pair works any more
  tc_fence_after();
  if (warp == 1) tmem_dealloc2(tmem_base, 512);
}

}  // namespace

int gemm_grouped_plan(GroupedPlan* p, const void* W, int experts, int N, int K) {
  if (experts < 1 || N < 8 || K < 8 || N % 8 || K % 8 || reinterpret_cast<uintptr_t>(W) % 16) return -1;
  p->experts = experts; p->N = N; p->K = K;
  return tmap_encode_bf16_2d(&p->tm_w, W, static_cast<uint64_t>(experts) * N, K, K, kSlab, kBlockK, 1);
}

constexpr int kBoxes[kGroupedBoxes] = {16, 32, 64, 128};

int gemm_grouped_x_maps(GroupedX* x, const void* X, int rows, int K) {
  for (int i = 0; i < kGroupedBoxes; ++i)
    if (const int rc = tmap_encode_bf16_2d(&x->box[i], X, rows, K, K, kBoxes[i], kBlockK, 1)) return rc;
  return 0;
}

namespace {
int launch(const CUtensorMap& tm_w, int experts, int N, int K, const CUtensorMap& tm_x, int box, const int* expert_rows, int rows, const GroupedOut& o,
           const SplitK& split, int units, int* error, cudaStream_t st) {
  const bool f32 = o.epi == GROUPED_F32, gated = o.epi == GROUPED_GATED || o.epi == GROUPED_GATED_FAST || o.epi == GROUPED_SILU;
  if ((!expert_rows && (experts != 1 || rows < 1)) || !o.y || o.ldy % (f32 ? 4 : 8) || N % (f32 ? 4 : 8) || reinterpret_cast<uintptr_t>(o.y) % 16 || units < 1 ||
      (gated && (N % kSlab || o.bias)) || (o.epi == GROUPED_TWO_TERMS && (N % (2 * kSlab) || o.bias || !o.y2 || reinterpret_cast<uintptr_t>(o.y2) % 16)) || (o.bias && experts != 1) || (f32 && split.parts > 1) || split.tile < 16 || split.tile % 16 || split.tile > 2 * box) return -1;
  static std::atomic<unsigned long long> attr[16];
  auto start = [&](auto kernel, int i) {
    if (!ensure_dynamic_smem(kernel, kSmem, &attr[i])) return -2;
    return launch_pdl(kernel, dim3(2 * units), dim3(threads_of(i / 2)), kSmem, st, tm_w, tm_x, expert_rows, experts, rows, o, N, K, box, split, error) == cudaSuccess ? 0 : -2;
  };
#define RUN(E) return box == 128 ? start(gemm_grouped_kernel<E, true>, 2 * E) : start(gemm_grouped_kernel<E, false>, 2 * E + 1)
  if (o.epi == GROUPED_SILU) RUN(5);
  if (o.epi == GROUPED_TWO_TERMS) RUN(6);
  if (o.epi == GROUPED_GATED_FAST) RUN(7);
  if (gated) RUN(1);
  if (f32) RUN(2);
  if (o.epi == GROUPED_XIELU) RUN(4);
  if (o.epi == GROUPED_RELU2 || o.bias) RUN(3);
  RUN(0);
#undef RUN
}
}  // namespace

int gemm_grouped_run(const GroupedPlan& p, const GroupedX& x, int most_rows, const int* expert_rows, const GroupedOut& o, int sms, int* error, cudaStream_t st) {
  if (!expert_rows) return -1;
  int i = 0;
  while (i + 1 < kGroupedBoxes && 2 * kBoxes[i] < most_rows) ++i;      // (smaller tiles for experts of many rows: 107 -> 114 us at up to 128 of 512 rows)
  return launch(p.tm_w, p.experts, p.N, p.K, x.box[i], kBoxes[i], expert_rows, 0, o, {nullptr, nullptr, 1, 2 * kBoxes[i]}, sms / 2, error, st);
}

namespace {
int whole_units(const GemmPlan& p, int tile, int parts, int rows) {
  return static_cast<int>(std::min<long long>(p.max_ctas / 2, static_cast<long long>((p.N + 2 * kSlab - 1) / (2 * kSlab)) * ((rows + tile - 1) / tile) * parts));
}
}  // namespace

int gemm_whole_run_as(const GemmPlan& p, const CUtensorMap& tm_x, int box, int tile, int parts, int rows, const GroupedOut& o, int* error, cudaStream_t st) {
  if (rows < 1 || tile < 1 || parts < 1 || parts > (p.K + kBlockK - 1) / kBlockK) return -1;
  const long long tiles = static_cast<long long>((p.N + 2 * kSlab - 1) / (2 * kSlab)) * ((rows + tile - 1) / tile);
  if (parts > 1 && (tiles * parts > p.max_ctas / 2 || tiles * parts * 2 * tile * kSlab * static_cast<long long>(sizeof(float)) > static_cast<long long>(p.ws_bytes) ||
                    !p.ws || !p.counters)) return -1;
  return launch(p.tm_w, 1, p.N, p.K, tm_x, box, nullptr, rows, o, {p.ws, p.counters, parts, tile}, whole_units(p, tile, parts, rows), error, st);
}

WholeTiles gemm_whole_tiles(const GemmPlan& p, int rows, bool cut) {
  WholeTiles w = {16, 1, 0};
  rules::whole_tiles(rows, p.N, p.K, p.max_ctas / 2, cut, &w.tile, &w.parts);
  while (w.box + 1 < kGroupedBoxes && 2 * kBoxes[w.box] < w.tile) ++w.box;
  return w;
}

int gemm_whole_ctas(const GemmPlan& p, const WholeTiles& w, int rows) { return 2 * whole_units(p, w.tile, w.parts, rows); }

int gemm_whole_run(const GemmPlan& p, const CUtensorMap* x_maps, int rows, const GroupedOut& o, cudaStream_t st) {
  if (rows < 1) return 0;
  const WholeTiles w = gemm_whole_tiles(p, rows, o.epi != GROUPED_F32);      // (fp32 outputs have no split form)
  return gemm_whole_run_as(p, x_maps[w.box], kBoxes[w.box], w.tile, w.parts, rows, o, p.error, st);      // the maps of the four smallest token-tile sizes have these boxes
}

int gemm_whole_run(const GemmPlan& p, const void* X, int x_rows, int ldx, const WholeTiles& w, int rows, const GroupedOut& o, cudaStream_t st) {
  CUtensorMap tm_x;
  if (ldx % 8) return -5;
  if (const int rc = tmap_encode_bf16_2d(&tm_x, X, x_rows, p.K, ldx, kBoxes[w.box], kBlockK, 1)) return rc;
  return gemm_whole_run_as(p, tm_x, kBoxes[w.box], w.tile, w.parts, rows, o, p.error, st);
}

int gemm_whole_direct(const void* W, int ldw, const void* X, int ldx, int N, int K, int rows, const GroupedOut& o, int* error, cudaStream_t st) {
  CUtensorMap tm_w, tm_x;
  int dev = 0, sms = 0, i = 0, tile, parts;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -2;
  rules::whole_tiles(rows, N, K, sms / 2, false, &tile, &parts);
  while (i + 1 < kGroupedBoxes && 2 * kBoxes[i] < tile) ++i;
  const int box = kBoxes[i];
  if (tmap_encode_bf16_2d(&tm_w, W, N, K, ldw, kSlab, kBlockK, 1) || tmap_encode_bf16_2d(&tm_x, X, rows, K, ldx, box, kBlockK, 1)) return -2;
  const long long tiles = static_cast<long long>((N + 2 * kSlab - 1) / (2 * kSlab)) * ((rows + tile - 1) / tile);
  return launch(tm_w, 1, N, K, tm_x, box, nullptr, rows, o, {nullptr, nullptr, 1, tile}, static_cast<int>(std::min<long long>(sms / 2, tiles)), error, st);
}

bool gemm_whole_fits(const GemmPlan& p, const void* out, int ldo) {
  return gemm_variant() == 2 && p.N % 8 == 0 && ldo % 8 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
}

}  // namespace b200
