// A few rows of X against a wide bf16 matrix, the projections of a decode step: one pass over the weights on every SM.
//
// What bounds it: the weights' bytes, and for the sizes of a decode step (4 to 40 MB a launch) just as much the chain wait ->
// load -> sum -> store.  So
//   * the rows of W are dealt out evenly, ceil(N / SMs) neighbouring rows a CTA (no tile size to round up to, no sum between
//     CTAs); the warps of a CTA take the 64-wide pieces of K in turn and their sums meet once in shared memory, in a fixed order;
//   * every warp runs a ring of its own in shared memory, filled by 16-byte asynchronous copies (whole 128-byte lines of W), so
//     loads never wait for products and no barrier stands in the loop;
//   * the ring is filled with weights before the wait for the kernel in front: W is nobody's output.  A CTA takes 163 to 210 KB, so
//     this overlaps kernels that use little shared memory (a norm, an activation, attention of single tokens), and between two such products
//     in a row nothing does: a smaller ring lost more than that would give (Layout).
// Products are mma.sync m16n8k16 with 16 rows of W as the first operand and 8 tokens as the second: at up to 16 tokens the
// kernel needs a twentieth of the tensor cores' rate, and rows that a tile has too many cost nothing.
// The order of one output element's sums depends on N and K alone, not on what else is in the batch.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdlib.h>

#include <algorithm>

#include "griddep.cuh"
#include "launch.h"
#include "linear_finish.cuh"
#include "mixers.h"

namespace b200 {
namespace {

using namespace linfin;
constexpr int kPiece = 64;     // values of K in one stage: a 128-byte line of a row

__device__ __forceinline__ void copy16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void ldm4(uint32_t* r, uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void mma16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int kWarps = 8;
// The shape of a launch: tokens in blocks of 8 (NB), 16-row blocks of W in a stage (MT).  A warp's ring has as many stages as
// fit 200 KB a CTA, which the loads in flight need more than a second CTA on the SM: 8192 x 2048, 8 tokens, with 64 KB 8.5 us,
// with 144 KB 7.0, with 200 KB 6.6; 2048 x 8192 13.0, 7.1 and 7.0.
template <int NB, int MT> struct Layout {
  static constexpr int kW = MT * 16 * 128, kStage = kW + NB * 8 * 128;
  static constexpr int kLd = MT * 16 + 4;     // a token's row of partial sums: the pad keeps the fragments' stores apart
  static constexpr int kPart = kWarps / 2 * NB * 8 * kLd * 4;
  static constexpr int kRoom = 226 * 1024 - kPart < 200 * 1024 ? 226 * 1024 - kPart : 200 * 1024;
  static constexpr int kFit = kRoom / (kWarps * kStage), kStages = kFit > 8 ? 8 : kFit;
  static_assert(kStages >= 2, "a ring of at least two stages");
  static constexpr int kRing = kWarps * kStages * kStage, kBytes = kRing + kPart;
};
// CTA b: rows [b * per_cta, + per_cta) of W in `blocks` blocks of at most `rows` <= 16 MT rows.
template <typename TY, int NB, int MT, bool PAIRS>
__global__ void __launch_bounds__(kWarps * 32) linear_stream_kernel(LinearArgs a, LinearPairs q, int per_cta, int rows) {
  typedef Layout<NB, MT> L;
  constexpr int D = L::kStages;
  extern __shared__ __align__(128) uint8_t sm[];
  const int lane = threadIdx.x & 31, wrp = threadIdx.x >> 5;
  float* part = reinterpret_cast<float*>(sm + L::kRing);                  // [pair of warps][token][row]
  const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(sm)) + wrp * D * L::kStage;
  const int n0 = blockIdx.x * per_cta, n1 = min(a.N, n0 + per_cta);
  const int pieces = (a.K + kPiece - 1) / kPiece, mine = wrp < pieces ? (pieces - wrp + kWarps - 1) / kWarps : 0;
  const bf16* W = static_cast<const bf16*>(a.W);
  const bf16* X = static_cast<const bf16*>(a.X);
  // a lane copies 16 bytes of rows lane / 8, lane / 8 + 4, ...; 16-byte pieces of a row are stored exchanged by the row's low bits
  const int lr = lane >> 3, lp = lane & 7;
  auto load_w = [&](int first, int piece, int slot) {
    const int live = min(rows, n1 - first), k = piece * kPiece + lp * 8;
    const bf16* src = W + static_cast<long long>(PAIRS ? row_of_pair(first + lr) : first + lr) * a.ldw + (k < a.K ? k : 0);
    const uint32_t dst = ring + slot * L::kStage;
    // paired rows step by two of W, and by 64 more past the end of their 64 (a block is shorter than that)
    const int end = PAIRS ? 63 - (((first + lr) >> 1) & 63) : 0;
#pragma unroll
    for (int i = 0; i < 4 * MT; ++i) {
      const int r = lr + 4 * i, step = PAIRS ? 2 * i + (2 * i > end ? 64 : 0) : 4 * i;
      if (r < live) copy16(dst + r * 128 + ((lp ^ (r & 7)) << 4), src + static_cast<long long>(step) * a.ldw, k < a.K ? 16 : 0);
    }
  };
  auto load_x = [&](int piece, int slot) {
    const int k = piece * kPiece + lp * 8;
    const bf16* src = X + static_cast<long long>(lr) * a.ldx + (k < a.K ? k : 0);
    const uint32_t dst = ring + slot * L::kStage + L::kW;
#pragma unroll
    for (int i = 0; i < 2 * NB; ++i) {
      const int t = lr + 4 * i;
      if (t < a.T) copy16(dst + t * 128 + ((lp ^ (t & 7)) << 4), src + static_cast<long long>(4 * i) * a.ldx, k < a.K ? 16 : 0);
    }
  };
  // the cursor of the loads runs D pieces ahead of the products', through the CTA's row blocks
  int lfirst = n0, li = 0;
  auto step = [&] { if (++li >= mine) { li = 0; lfirst += rows; } };
  griddep_launch();
  if (mine) {
#pragma unroll
    for (int s = 0; s < D; ++s) {
      if (lfirst < n1) { load_w(lfirst, wrp + li * kWarps, s); step(); }
      copy_commit();
    }
  }
  griddep_wait();
  if (mine) {
    int f = n0, i = 0;
#pragma unroll
    for (int s = 0; s < D; ++s) {
      if (f < n1) { load_x(wrp + i * kWarps, s); if (++i >= mine) { i = 0; f += rows; } }
      copy_commit();
    }
  }
  int slot = 0;
  for (int first = n0; first < n1; first += rows) {
    float acc[MT][NB][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][j][e] = 0.f;
    for (int p = 0; p < mine; ++p) {
      copy_wait<D - 1>();
      __syncwarp();
      const uint32_t at = ring + slot * L::kStage;
      const int r8 = lane & 7, mi = lane >> 3;
      uint32_t b[NB][8];
#pragma unroll
      for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) ldm4(&b[j][4 * h], at + L::kW + (8 * j + r8) * 128 + (((4 * h + mi) ^ r8) << 4));
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          uint32_t w[4];
          ldm4(w, at + (16 * m + r8 + 8 * (mi & 1)) * 128 + (((2 * kk + (mi >> 1)) ^ r8) << 4));
#pragma unroll
          for (int j = 0; j < NB; ++j) mma16816(acc[m][j], w, b[j][2 * kk], b[j][2 * kk + 1]);
        }
      __syncwarp();
      if (lfirst < n1) { load_w(lfirst, wrp + li * kWarps, slot); load_x(wrp + li * kWarps, slot); step(); }
      copy_commit();
      slot = slot + 1 == D ? 0 : slot + 1;
    }
    // the upper half of the warps leaves its sums, the lower half adds its own: half the room, and a fixed order
    const int g = lane >> 2, t4 = lane & 3;
    float* own = part + (wrp % (kWarps / 2)) * NB * 8 * L::kLd;
#pragma unroll
    for (int half = 1; half >= 0; --half) {
      if (wrp / (kWarps / 2) == half) {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int j = 0; j < NB; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float* q = own + (8 * j + 2 * t4 + (e & 1)) * L::kLd + 16 * m + g + 8 * (e >> 1);
              *q = half ? acc[m][j][e] : acc[m][j][e] + *q;
            }
      }
      __syncthreads();
    }
    const int live = min(rows, n1 - first);
    auto sum = [&](int t, int r) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps / 2; ++w) v += part[(w * NB * 8 + t) * L::kLd + r];
      return v;
    };
    if (PAIRS) {
      const int pairs = live >> 1;
      for (int e = threadIdx.x; e < pairs * a.T; e += kWarps * 32) {
        const int t = e / pairs, r = 2 * (e - t * pairs);
        finish_pair(a, q, t, (first + r) >> 1, bf16r(sum(t, r)), bf16r(sum(t, r + 1)));
      }
    } else {
      for (int e = threadIdx.x; e < live * a.T; e += kWarps * 32) {
        const int t = e / live, r = e - t * live, n = first + r;
        put(static_cast<TY*>(a.Y) + static_cast<long long>(t) * a.ldy + n, finish_one<TY>(a, sum(t, r), t, n));
      }
    }
    if (first + rows < n1) __syncthreads();
  }
}

template <typename TY, int NB, int MT, bool PAIRS>
int launch(const LinearArgs& a, const LinearPairs& q, int per_cta, int rows, cudaStream_t st) {
  static std::atomic<unsigned long long> set{0};
  if (!ensure_dynamic_smem(linear_stream_kernel<TY, NB, MT, PAIRS>, Layout<NB, MT>::kBytes, &set)) return -2;
  const int ctas = (a.N + per_cta - 1) / per_cta;
  launch_pdl(linear_stream_kernel<TY, NB, MT, PAIRS>, ctas, kWarps * 32, Layout<NB, MT>::kBytes, st, a, q, per_cta, rows);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
// n rows in `parts` shares, whole pairs each
int share(int n, int parts, bool pairs) { return pairs ? (n / 2 + parts - 1) / parts * 2 : (n + parts - 1) / parts; }
template <typename TY, int NB, bool PAIRS>
int pick_rows(const LinearArgs& a, const LinearPairs& q, int sms, cudaStream_t st) {
  // rows of W at a time: more of them use a token's row more often, fewer leave room for more stages.  28672 x 4096, 8 tokens:
  // 64 at a time 38.7 us, 48 35.8, 32 35.8, 16 37.5 (all rows of a CTA side by side, so that a piece of X is read once: 38.5,
  // and 36 -> 38 with one token: neighbouring pieces of a row are better read together); 6144 x 2048, 41 rows a CTA: 5.5 at once, 6.1 as twice 21.
  constexpr int kMost = NB <= 4 ? 48 : 32;
  const int per_cta = share(a.N, sms, PAIRS), rows = share(per_cta, (per_cta + kMost - 1) / kMost, PAIRS);
  switch ((rows + 15) / 16) {
    case 1: return launch<TY, NB, 1, PAIRS>(a, q, per_cta, rows, st);
    case 2: return launch<TY, NB, 2, PAIRS>(a, q, per_cta, rows, st);
    default: return launch<TY, NB, kMost / 16, PAIRS>(a, q, per_cta, rows, st);
  }
}
template <typename TY, bool PAIRS>
int pick_tokens(const LinearArgs& a, const LinearPairs& q, cudaStream_t st) {
  const int sms = sm_count();
  if (a.T <= 8) return pick_rows<TY, 1, PAIRS>(a, q, sms, st);
  if (a.T <= 16) return pick_rows<TY, 2, PAIRS>(a, q, sms, st);
  if (a.T <= 24) return pick_rows<TY, 3, PAIRS>(a, q, sms, st);
  if (a.T <= 32) return pick_rows<TY, 4, PAIRS>(a, q, sms, st);
  return pick_rows<TY, 6, PAIRS>(a, q, sms, st);
}

}  // namespace

// The lines were drawn where the whole-tile product (gemm_grouped.cu) and the pair kernel (gemm2_tcgen05.cu) cross, weights from
// HBM, us a launch here / there:
//   2048 x 8192:   8 tokens 7.0 / 13.0   32 tokens 10.5 / 14.4   48 tokens 14.5 / 15.3
//   1792 x 2048:   8 tokens 3.0 /  8.3   32 tokens  4.1 /  9.5   48 tokens  5.5 / 10.4
//   8192 x 2048:   8 tokens 6.6 / 11.7   32 tokens  9.4 / 12.4   48 tokens 13.2 / 13.4
//   28672 x 4096:  8 tokens 36.1 / 42.5  16 tokens 39.0 / 43.0, in a second of nothing else 38.5 / 43.5 and 43.7 / 44.0
// More tokens cost their rows once a CTA and block of its rows, which is what narrow matrices can afford longest.  With a long K the
// whole tiles win earlier (rules::stream_pays, rules::tiles_ahead); a product without a plan for them still comes here.
bool linear_streams(const LinearArgs& a, const LinearPairs* q) {
  static const int most = [] { const char* e = getenv("B200_LIN_STREAM"); return e ? atoi(e) : 48; }();     // A/B knob: the most rows, 0: none
  const int sms = sm_count();
  if (a.T > most || a.T > (a.N <= 32 * sms ? 48 : a.N <= 80 * sms ? 32 : 8)) return false;
  if (q && (a.N % 128 || a.ty != DT_BF16 || a.bias || a.row_scale || a.act != LIN_NONE)) return false;
  return a.T > 0 && a.N > 0 && a.K > 0 && a.tx == DT_BF16 && a.tw == DT_BF16 && a.batch == 1 && !a.x_rows && !a.tile_group && a.K % 8 == 0 && a.ldx % 8 == 0 &&
         a.ldw % 8 == 0 && (reinterpret_cast<uintptr_t>(a.X) | reinterpret_cast<uintptr_t>(a.W)) % 16 == 0;
}

int linear_stream(const LinearArgs& a, const LinearPairs* q, cudaStream_t st) {
  if (!linear_streams(a, q)) return -1;
  if (q) return pick_tokens<bf16, true>(a, *q, st);
  return a.ty == DT_BF16 ? pick_tokens<bf16, false>(a, LinearPairs(), st) : pick_tokens<float, false>(a, LinearPairs(), st);
}

int linear_stream_ctas(const LinearArgs& a, const LinearPairs* q) {
  const int per_cta = share(a.N, sm_count(), q != nullptr);
  return (a.N + per_cta - 1) / per_cta;
}

}  // namespace b200
