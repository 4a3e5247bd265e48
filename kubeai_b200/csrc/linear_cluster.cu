// Steps of some tens to a few hundred tokens against a matrix: the product cut over every SM, K over the CTAs of a cluster.
//
// Such a step is too large for linear_stream.cu, where every CTA reads all of X, and too small for whole 256 x 256 tiles
// (gemm_grouped.cu): 2048 x 2048 has eight of them, so K is cut over the pairs, and the part that comes last reads all the
// others' sums through one pair's share of L2 bandwidth.  Here a cluster of C CTAs owns R rows of W and all tokens; each CTA
// multiplies its share of K (tcgen05, tokens as the 128 rows of D, the R rows of W as its columns, fp32 in TMEM), and the sums meet by
// reduce-scatter through distributed shared memory: CTA c gets columns [c R / C, + R / C) of every CTA, adds them in the CTAs'
// order and finishes them.  No sum goes through global memory and nobody waits outside its cluster.
// What bounds it: (T + R) K / C values through each SM's port and about 6 us of fixed steps.  Operands come by 16-byte asynchronous copies into the layout of the 128-byte swizzle, W ahead of the wait for the kernel in
// front.  The order of one output's sums depends on the shape that T, N and K give.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdlib.h>

#include <algorithm>

#include "griddep.cuh"
#include "launch.h"
#include "linear_finish.cuh"
#include "mixers.h"
#include "umma2.cuh"

namespace b200 {
namespace {

using namespace linfin;
constexpr int kLoaders = 8, kThreads = (kLoaders + 1) * 32;     // loading warps, which also finish; one issues the products
constexpr int kMaxStages = 8;
constexpr int KS = 2;     // 64-wide pieces of K in a stage: fewer barriers to pass.  2048 x 2048, 100 tokens: one piece 9.0 us, two 8.0
constexpr int kWaitLimit = 1 << 22;
constexpr int kRing = 160 * 1024, kSums = 64 * 1024;

__device__ __forceinline__ void copy16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}
// this thread's copies so far, once they are through, count as its arrival
__device__ __forceinline__ void copies_arrive(uint32_t bar) { asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool wait_limited(uint32_t bar, uint32_t parity) { return mbar_wait_limited(bar, parity, kWaitLimit); }
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void store_cluster(uint32_t at, const uint32_t* v) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}

struct Shape {
  int C, R, D, cols;     // CTAs of a cluster, rows of W, stages, TMEM columns
};

// MT: blocks of 128 tokens.  Cluster i: rows [i R, + R) of W.
template <typename TY, int MT>
__global__ void __launch_bounds__(kThreads, 1) linear_cluster_kernel(LinearArgs a, Shape s) {
  extern __shared__ uint8_t raw[];
  const uint32_t base = (smem_u32(raw) + 1023u) & ~1023u;
  const int C = s.C, R = s.R, D = s.D, block = MT * 16384 + R * 128, stage = KS * block;
  uint8_t* ring = raw + (base - smem_u32(raw));
  const uint32_t sums_at = base + kRing, bars = sums_at + kSums;
  auto full = [&](int i) { return bars + 8u * i; };
  auto empty = [&](int i) { return bars + 8u * (kMaxStages + i); };
  const uint32_t done = bars + 8u * 2 * kMaxStages, slot = done + 8;
  const int tid = threadIdx.x, lane = tid & 31, warp = warp_number();
  const int rank = static_cast<int>(cluster_ctarank()), n0 = blockIdx.x / C * R;
  const int KB = (a.K + 64 * KS - 1) / (64 * KS), kb0 = rank * KB / C, kbn = (rank + 1) * KB / C - kb0;
  if (warp == kLoaders) {
    if (lane == 0) {
      for (int i = 0; i < D; ++i) { mbar_init(full(i), kLoaders * 32); mbar_init(empty(i), 1); }
      mbar_init(done, 1);
      fence_mbar_init();
    }
    __syncwarp();
    tmem_alloc(slot, s.cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(ring + (slot - base));
  if (C > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");     // this CTA runs: its shared memory can be written
  griddep_launch();     // behind the allocation: a kernel that starts early allocates after this one
  bool ok = true;
  if (warp < kLoaders) {
    const bf16 *W = static_cast<const bf16*>(a.W), *X = static_cast<const bf16*>(a.X);
    const int lr = warp * 4 + (lane >> 3), lp = lane & 7;     // a lane copies 16 bytes of rows lr, lr + 32, ...
    // every cluster starts elsewhere in K: all of them asking L2 for the same rows of X at once is slower than X is large
    const int turn = (blockIdx.x / C) % kbn;
    auto piece = [&](int i) { const int p = i + turn; return kb0 + (p < kbn ? p : p - kbn); };
    auto load_w = [&](int kb, int i) {
#pragma unroll
      for (int h = 0; h < KS; ++h) {
        const int k = (piece(kb) * KS + h) * 64 + lp * 8;
        const uint32_t dst = base + i * stage + h * block + MT * 16384;
        for (int r = lr; r < R; r += 32)
          if (n0 + r < a.N)
            copy16(dst + r * 128 + ((lp ^ (r & 7)) << 4), W + static_cast<long long>(n0 + r) * a.ldw + (k < a.K ? k : 0), k < a.K ? 16 : 0);
      }
    };
    auto load_x = [&](int kb, int i) {
#pragma unroll
      for (int h = 0; h < KS; ++h) {
        const int k = (piece(kb) * KS + h) * 64 + lp * 8;
        const uint32_t dst = base + i * stage + h * block;
        for (int t = lr; t < a.T; t += 32)
          copy16(dst + t * 128 + ((lp ^ (t & 7)) << 4), X + static_cast<long long>(t) * a.ldx + (k < a.K ? k : 0), k < a.K ? 16 : 0);
      }
    };
    const int ahead = min(D, kbn);
    for (int i = 0; i < ahead; ++i) load_w(i, i);
    griddep_wait();
    for (int i = 0; i < ahead; ++i) { load_x(i, i); copies_arrive(full(i)); }
    for (int i = D; i < kbn; ++i) {
      if (!wait_limited(empty(i % D), (i / D - 1) & 1)) { ok = false; break; }
      load_w(i, i % D);
      load_x(i, i % D);
      copies_arrive(full(i % D));
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    const bool one = elect_one();
    const uint32_t idesc = umma_idesc_bf16(128, R);
    for (int i = 0; i < kbn && ok; ++i) {
      ok = __all_sync(0xffffffffu, wait_limited(full(i % D), (i / D) & 1));
      if (!ok) break;
      fence_proxy_async();      // the copies wrote through the generic proxy, the tensor cores read through the other
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < KS; ++h) {
        const uint32_t at = base + (i % D) * stage + h * block;
        const uint64_t bd = umma_desc_kmajor_sw128(at + MT * 16384);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const uint64_t ad = umma_desc_kmajor_sw128(at + m * 16384);
          if (one) umma_bf16_k64(tmem + m * R, ad, bd, idesc, (i > 0 || h > 0) ? 1u : 0u);
        }
      }
      if (one) umma_commit(empty(i % D));
      __syncwarp();
    }
    if (one) umma_commit(done);
  }
  __syncwarp();
  ok = wait_limited(done, 0) && ok;
  if (!ok && a.error) *reinterpret_cast<volatile int*>(a.error) = 1;
  __syncwarp();
  tc_fence_after();
  // the sums, [source][four columns][token], to their owners (who are known to run)
  if (C > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  const int S = R / C, S4 = S / 4, Tp = (a.T + 31) & ~31;
  if (warp < kLoaders) {
    const int quarter = warp & 3, m = MT == 1 ? 0 : warp >> 2, t = 128 * m + 32 * quarter + lane;
    if (128 * m + 32 * quarter < a.T) {
      for (int c = MT == 1 ? warp >> 2 : 0; c < R / 16; c += MT == 1 ? 2 : 1) {
        uint32_t v[16];
        tmem_ld_32x16(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + m * R + 16 * c, v);
        tmem_ld_wait();
        if (t < a.T) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const int col = 16 * c + 4 * g, owner = col / S, c4 = (col - owner * S) >> 2;
            const uint32_t at = sums_at + ((rank * S4 + c4) * Tp + t) * 16;
            store_cluster(C > 1 ? mapa_u32(at, owner) : at, v + 4 * g);
          }
        }
        __syncwarp();
      }
    }
  }
  tc_fence_before();
  if (C > 1) cluster_sync_all();
  else __syncthreads();
  if (warp == kLoaders) {
    tc_fence_after();
    tmem_dealloc(tmem, s.cols);
    return;
  }
  const float4* sums = reinterpret_cast<const float4*>(ring + kRing);
  const bool wide = a.ldy % 4 == 0 && reinterpret_cast<uintptr_t>(a.Y) % (4 * sizeof(TY)) == 0;
  for (int e = tid; e < S4 * a.T; e += kLoaders * 32) {
    const int t = e / S4, c4 = e - t * S4, n = n0 + rank * S + 4 * c4;
    if (n >= a.N) continue;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = 0; c < C; ++c) {
      const float4 x = sums[(c * S4 + c4) * Tp + t];
      v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
    }
    TY* y = static_cast<TY*>(a.Y) + static_cast<long long>(t) * a.ldy + n;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (n + i < a.N) v[i] = finish_one<TY>(a, v[i], t, n + i);
    if (wide && n + 3 < a.N) {
      if constexpr (sizeof(TY) == 2) *reinterpret_cast<uint2*>(y) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
      else *reinterpret_cast<float4*>(y) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (n + i < a.N) put(y + i, v[i]);
    }
  }
}

template <typename TY, int MT>
int launch(const LinearArgs& a, const Shape& s, cudaStream_t st) {
  static std::atomic<unsigned long long> set{0};
  constexpr int smem = kRing + kSums + 1024 + 8 * (2 * kMaxStages + 2);
  if (!ensure_dynamic_smem(linear_cluster_kernel<TY, MT>, smem, &set)) return -2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.N + s.R - 1) / s.R * s.C);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = s.C; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, linear_cluster_kernel<TY, MT>, a, s) == cudaSuccess ? 0 : -2;
}

// Four CTAs a cluster and 64 rows of W put 2048 rows on 128 SMs; a long K with up to 128 tokens has less of X to read with six and
// 96 rows (at most 22 such clusters run at once, and 33 of four).  us a launch, weights from HBM, whole tiles of 256 rows / here:
//   2048 x 2048   64 tokens 11.1 / 7.2   100 tokens 13.6 / 8.0    256 tokens 14.9 / 11.6
//   2048 x 4096   64 tokens 13.0 / 10.3  128 tokens 18.0 / 11.8   256 tokens 24.4 / 16.1
//   2048 x 8192   64 tokens 16.3 / 15.2  128 tokens 21.4 / 17.2   256 tokens 32.1 / 25.3
//   3072 x 1024   64 tokens  8.4 / 6.6   128 tokens  9.1 / 8.0    256 tokens 10.5 / 12.4
// From 4096 rows on those are as fast or faster: they read X once for 256 rows.  So they are with a long K (rules::cluster_pays), and tiles whose
// rows are chosen for the call are from 129 tokens on (rules::tiles_ahead); a product without a plan for them still comes here.
bool pick_shape(int T, int N, int K, Shape* s) {
  s->C = 4;
  if (N <= 2112) {
    const bool six = K >= 4096 && T <= 128;
    if (six) s->C = 6;
    s->R = six ? 96 : 64;
  } else if (N <= 33 * 96 && T <= 128) {
    s->R = 96;
  } else {
    return false;
  }
  const int mt = (T + 127) / 128;
  s->D = std::min(kMaxStages, kRing / (KS * (mt * 16384 + s->R * 128)));
  s->cols = 32;
  while (s->cols < mt * s->R) s->cols *= 2;
  return s->D >= 2 && (K + 64 * KS - 1) / (64 * KS) >= s->C && s->R * ((T + 31) & ~31) * 4 <= kSums;
}

}  // namespace

bool linear_clusters(const LinearArgs& a) {
  static const bool on = [] { const char* e = getenv("B200_LIN_CLUSTER"); return !e || atoi(e) != 0; }();     // A/B knob
  Shape s;
  // its waits have a limit, so it runs only where a wait that ran out can be reported
  return on && a.error && a.T > 32 && a.T <= 256 && a.N >= 1024 && a.tx == DT_BF16 && a.tw == DT_BF16 && a.batch == 1 && !a.x_rows && !a.tile_group && a.K % 8 == 0 &&
         a.ldx % 8 == 0 && a.ldw % 8 == 0 && (reinterpret_cast<uintptr_t>(a.X) | reinterpret_cast<uintptr_t>(a.W)) % 16 == 0 && pick_shape(a.T, a.N, a.K, &s);
}

int linear_cluster(const LinearArgs& a, cudaStream_t st) {
  Shape s;
  if (!linear_clusters(a) || !pick_shape(a.T, a.N, a.K, &s)) return -1;
  if (a.T <= 128) return a.ty == DT_BF16 ? launch<bf16, 1>(a, s, st) : launch<float, 1>(a, s, st);
  return a.ty == DT_BF16 ? launch<bf16, 2>(a, s, st) : launch<float, 2>(a, s, st);
}

}  // namespace b200
