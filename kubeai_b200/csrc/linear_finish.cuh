// What linear_stream.cu and linear_cluster.cu do with a finished sum: scale, bias and activation of one output, or the two sums of a
// pair of rows (LinearPairs, mixers.h).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "activations.cuh"
#include "mixers.h"
#include "ptx.cuh"

namespace b200 {
namespace linfin {

typedef __nv_bfloat16 bf16;
__device__ __forceinline__ void put(float* p, float v) { *p = v; }
__device__ __forceinline__ void put(bf16* p, float v) { *p = __float2bfloat16_rn(v); }
// scale, bias and activation of output n of token t (TY: the type it is rounded to)
template <typename TY>
__device__ __forceinline__ float finish_one(const LinearArgs& a, float v, int t, int n) {
  if (a.row_scale) v *= a.row_scale[t];
  if (a.bias) v += a.bias[n];
  if (a.act == LIN_RELU2) { v = fmaxf(v, 0.f); v = v * v; }
  else if (a.act == LIN_XIELU) v = sizeof(TY) == 2 ? xielu_fast(v, a.a_pos, a.a_neg) : xielu(v, a.a_pos, a.a_neg);
  return v;
}

// In the paired form rows i and i + 64 of every 128 of W belong together (gate and up rows of the same outputs, the two halves
// of a head): a CTA takes them as neighbours, row n of this order being row_of_pair(n) of W.
__device__ __forceinline__ int row_of_pair(int n) { const int p = n >> 1; return p + (p & ~63) + ((n & 1) << 6); }

__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
// Both rows of pair p of token t, rounded to bf16, to their output; the arithmetic is that of gemm_grouped.cu's gated epilogues
// and of elementwise.cu's rope_kv_kernel.
__device__ __forceinline__ void finish_pair(const LinearArgs& a, const LinearPairs& q, int t, int p, float x, float y) {
  bf16* Y = static_cast<bf16*>(a.Y) + static_cast<long long>(t) * a.ldy;
  if (q.kind == PAIRS_GATED) Y[p] = __float2bfloat16_rn(gated_unit<false>(x, y, q.limit < INFINITY, q.limit, q.slope, q.up_offset));
  else if (q.kind == PAIRS_SILU) Y[p] = __float2bfloat16_rn(__bfloat162float(silu_bf16(x)) * y);
  else {
    const int head = p >> 6, i = p & 63, slot = q.slots[t];
    bf16* dst = Y + head * 128 + i;
    if (head >= q.heads) {     // a key or value head: its row of the page, and nothing for a token without one
      if (slot < 0) return;
      const long long page = static_cast<long long>(q.kv_heads) * 16 * 128;
      const int kv_head = head - q.heads, value = kv_head >= q.kv_heads;
      dst = static_cast<bf16*>(q.kv_layer) + (2 * static_cast<long long>(slot >> 4) + value) * page + ((kv_head - (value ? q.kv_heads : 0)) * 16 + (slot & 15)) * 128 + i;
    }
    if (head < q.heads + q.kv_heads) {
      const int pos = min(max(q.positions[t], 0), q.max_pos - 1);
      const bf16* cs = static_cast<const bf16*>(q.cos_sin) + static_cast<long long>(pos) * 128;
      const float c = __bfloat162float(cs[i]), s = __bfloat162float(cs[64 + i]);
      const float xc = bf16r(__fmul_rn(x, c)), ys = bf16r(__fmul_rn(y, s)), yc = bf16r(__fmul_rn(y, c)), xs = bf16r(__fmul_rn(x, s));
      x = xc - ys;
      y = yc + xs;
    }
    dst[0] = __float2bfloat16_rn(x);
    dst[64] = __float2bfloat16_rn(y);
  }
}

}  // namespace linfin
}  // namespace b200
