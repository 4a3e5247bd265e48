// The gated delta rule (mixers.h DeltaArgs): a recurrent mixer whose per-head state S [dim, vdim] is a memory from unit keys
// to values.  Every token decays it by one scalar, reads what it holds under the token's key, and writes only beta times
// the difference to the token's value:  S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q.
//
// The sequential scan: the columns of S are independent.  A column's key rows are shared by P neighbouring lanes of one warp
// (P a power of two, at most 32 rows each, in registers for the whole step), so the two sums a token needs over the rows,
// S^T k and S^T q, are P-lane shuffle reductions and the token loop has no barrier.  Both sums are taken over the state in
// front of the write, in one pass: with s = g S^T k and u = beta (v - s), the read-out after the write is
// o = g S^T q + (k . q) u, and k . q is formed once per token while it is staged.  A round stages G tokens in shared
// memory: a warp per token normalises its query and key (sums of squares in fp32), forms k . q, the step size beta and
// the decay g with the accurate library functions.  Everything is fp32, and the same operations run in the same order
// however a sequence was cut into steps.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdlib.h>

#include <algorithm>

#include "dispatch_rules.h"
#include "griddep.cuh"
#include "launch.h"
#include "mixers.h"

namespace b200 {
namespace {

typedef __nv_bfloat16 bf16;
__device__ __forceinline__ float ldf(const float* p) { return __ldg(p); }
__device__ __forceinline__ float ldf(const bf16* p) { return __bfloat162float(__ldg(p)); }
__device__ __forceinline__ float softplusf_(float x) { return x > 20.0f ? x : log1pf(expf(x)); }

constexpr int kPieces = 8;      // float4 pieces of a state column held by one thread (32 rows)
constexpr int kGroup = 16;      // tokens staged per round (fewer when dim is large)
constexpr int kThreads = 128;

// grid: (ceil(vdim / cols), heads, nseq), cols = kThreads / P.  A column's rows come in float4 pieces dealt to its P lanes in
// turn: lane p's m-th piece holds rows 4 (m P + p) .. + 3, m < M; Dp = 4 P M >= dim is the padded row length.
template <typename T>
__global__ void __launch_bounds__(kThreads) delta_scan_kernel(DeltaArgs a, int P, int M, int G) {
  extern __shared__ __align__(16) float sm[];
  const int seq = blockIdx.z, head = blockIdx.y;
  const int tok0 = a.seqs[seq * 8 + 0], n = a.seqs[seq * 8 + 1], pos0 = a.seqs[seq * 8 + 2], slot = a.seqs[seq * 8 + 3];
  const int D = a.dim, Dv = a.vdim, Dp = 4 * P * M, cols = kThreads / P;
  const int tid = threadIdx.x, lane = tid & 31, wrp = tid >> 5;
  const int p = lane & (P - 1), c = tid / P, j = blockIdx.x * cols + c;
  float* qs = sm;                     // [G][Dp] unit queries times q_scale
  float* ks = qs + G * Dp;            // [G][Dp] unit keys
  float* vs = ks + G * Dp;            // [G][cols]
  float* os = vs + G * cols;          // [G][cols]
  float* sc = os + G * cols;          // [3][G] decay, step size, k . q
  const T* base = static_cast<const T*>(a.qkv);
  const int g = head / (a.heads / a.kv_heads);
  float* Sg = a.states + (static_cast<long long>(slot) * a.heads + head) * D * Dv + j;
  const bool live = j < Dv;
  float S[kPieces][4];
  {
    const float* r = Sg + static_cast<long long>(4 * p) * Dv;      // one pointer walks the lane's rows
    const long long skip = static_cast<long long>(4 * P - 4) * Dv;
    const bool held = live && pos0 > 0;
#pragma unroll
    for (int m = 0; m < kPieces; ++m, r += skip)
#pragma unroll
      for (int e = 0; e < 4; ++e, r += Dv) S[m][e] = (held && m < M && 4 * (m * P + p) + e < D) ? *r : 0.f;
  }
  const float rate = a.rate[head], dt_bias = a.dt_bias[head];
  for (int g0 = 0; g0 < n; g0 += G) {
    const int gn = min(G, n - g0);
    __syncthreads();
    for (int tt = wrp; tt < gn; tt += kThreads / 32) {
      const long long row = static_cast<long long>(tok0) + g0 + tt;
      const T* q = base + row * a.ld + a.q_off + static_cast<long long>(g) * D;
      const T* k = base + row * a.ld + a.k_off + static_cast<long long>(g) * D;
      float qq = 0.f, kk = 0.f, qk = 0.f;
      for (int i = lane; i < D; i += 32) {
        const float x = ldf(q + i), y = ldf(k + i);
        qq = fmaf(x, x, qq); kk = fmaf(y, y, kk); qk = fmaf(x, y, qk);
      }
      for (int o = 16; o > 0; o >>= 1) {
        qq += __shfl_xor_sync(0xffffffffu, qq, o);
        kk += __shfl_xor_sync(0xffffffffu, kk, o);
        qk += __shfl_xor_sync(0xffffffffu, qk, o);
      }
      const float iq = a.q_scale / sqrtf(qq + a.unit_eps), ik = 1.0f / sqrtf(kk + a.unit_eps);
      for (int i = lane; i < Dp; i += 32) {
        qs[tt * Dp + i] = i < D ? ldf(q + i) * iq : 0.f;
        ks[tt * Dp + i] = i < D ? ldf(k + i) * ik : 0.f;
      }
      if (lane == 0) {
        const float b = ldf(static_cast<const T*>(a.beta_pre) + row * a.ld_gate + head);
        const float d = softplusf_(ldf(static_cast<const T*>(a.dt_pre) + row * a.ld_gate + head) + dt_bias);
        sc[tt] = expf(rate * d);
        sc[G + tt] = 1.0f / (1.0f + expf(-b));
        sc[2 * G + tt] = qk * iq * ik;
      }
    }
    for (int e = tid; e < gn * cols; e += kThreads) {
      const int tt = e / cols, cc = e - tt * cols, jc = blockIdx.x * cols + cc;
      vs[e] = jc < Dv ? ldf(base + (static_cast<long long>(tok0) + g0 + tt) * a.ld + a.v_off + static_cast<long long>(head) * Dv + jc) : 0.f;
    }
    __syncthreads();
    for (int tt = 0; tt < gn; ++tt) {
      const float4* q4 = reinterpret_cast<const float4*>(qs + tt * Dp);
      const float4* k4 = reinterpret_cast<const float4*>(ks + tt * Dp);
      const float decay = sc[tt];
      float rk[4] = {0.f, 0.f, 0.f, 0.f}, rq[4] = {0.f, 0.f, 0.f, 0.f};
      float4 kv[kPieces];
#pragma unroll
      for (int m = 0; m < kPieces; ++m) {
        if (m < M) {
          const float4 qa = q4[m * P + p];
          kv[m] = k4[m * P + p];
          rk[0] = fmaf(S[m][0], kv[m].x, rk[0]); rq[0] = fmaf(S[m][0], qa.x, rq[0]);
          rk[1] = fmaf(S[m][1], kv[m].y, rk[1]); rq[1] = fmaf(S[m][1], qa.y, rq[1]);
          rk[2] = fmaf(S[m][2], kv[m].z, rk[2]); rq[2] = fmaf(S[m][2], qa.z, rq[2]);
          rk[3] = fmaf(S[m][3], kv[m].w, rk[3]); rq[3] = fmaf(S[m][3], qa.w, rq[3]);
        }
      }
      float sk = (rk[0] + rk[1]) + (rk[2] + rk[3]), sq = (rq[0] + rq[1]) + (rq[2] + rq[3]);
      for (int o = P >> 1; o > 0; o >>= 1) {
        sk += __shfl_xor_sync(0xffffffffu, sk, o);
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
      }
      const float u = sc[G + tt] * fmaf(-decay, sk, vs[tt * cols + c]);
      if (p == 0) os[tt * cols + c] = fmaf(sc[2 * G + tt], u, decay * sq);
#pragma unroll
      for (int m = 0; m < kPieces; ++m) {
        if (m < M) {
          S[m][0] = fmaf(kv[m].x, u, decay * S[m][0]);
          S[m][1] = fmaf(kv[m].y, u, decay * S[m][1]);
          S[m][2] = fmaf(kv[m].z, u, decay * S[m][2]);
          S[m][3] = fmaf(kv[m].w, u, decay * S[m][3]);
        }
      }
    }
    __syncthreads();
    for (int e = tid; e < gn * cols; e += kThreads) {
      const int tt = e / cols, cc = e - tt * cols, jc = blockIdx.x * cols + cc;
      if (jc < Dv) a.o[(static_cast<long long>(tok0) + g0 + tt) * (static_cast<long long>(a.heads) * Dv) + static_cast<long long>(head) * Dv + jc] = os[e];
    }
  }
  if (live) {
    float* r = Sg + static_cast<long long>(4 * p) * Dv;
    const long long skip = static_cast<long long>(4 * P - 4) * Dv;
#pragma unroll
    for (int m = 0; m < kPieces; ++m, r += skip)
#pragma unroll
      for (int e = 0; e < 4; ++e, r += Dv)
        if (m < M && 4 * (m * P + p) + e < D) *r = S[m][e];
  }
}

// Steps in which every sequence brings one token: a pass over the states as in gla.cu's gla_step_kernel, with the sums S^T k and
// S^T q taken before the write.  A CTA takes 64 value columns of a (head, sequence): sixteen lanes a row in 16-byte pieces, RPT
// rows a thread, every load in flight at once.  100 sequences of 16 heads of 128 x 128: 74 us in the scan, 37 here.
constexpr int kStepCols = 64, kStepWarps = 8;
template <typename T, int RPT>
__global__ void __launch_bounds__(kStepWarps * 32) delta_step_kernel(DeltaArgs a) {
  griddep_launch();
  __shared__ __align__(16) float qs[16 * RPT], ks[16 * RPT];
  __shared__ __align__(16) float part[2][kStepWarps][kStepCols];
  __shared__ float sc[3];
  const int seq = blockIdx.z, head = blockIdx.y, tid = threadIdx.x, lane = tid & 31, wrp = tid >> 5, D = a.dim, Dv = a.vdim;
  const int tok = a.seqs[seq * 8 + 0], pos = a.seqs[seq * 8 + 2], slot = a.seqs[seq * 8 + 3];     // the step's inputs, uploaded before its first kernel
  const int jc = (tid & 15) * 4, j0 = blockIdx.x * kStepCols + jc, r0 = tid >> 4;
  const bool live = j0 < Dv, held = pos > 0;
  float* Sg = a.states + (static_cast<long long>(slot) * a.heads + head) * D * Dv + j0;
  if (held && live && (tid & 7) == 0)
    for (int m = 0; m < RPT; ++m)
      if (r0 + 16 * m < D) asm volatile("prefetch.global.L2 [%0];" ::"l"(Sg + static_cast<long long>(r0 + 16 * m) * Dv));
  griddep_wait();
  float4 S[RPT];
#pragma unroll
  for (int m = 0; m < RPT; ++m) {
    const int i = r0 + 16 * m;
    S[m] = held && live && i < D ? *reinterpret_cast<const float4*>(Sg + static_cast<long long>(i) * Dv) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  auto ld = [](const T* p) { return static_cast<float>(*p); };      // rows that an earlier kernel of the step wrote
  const T* row = static_cast<const T*>(a.qkv) + static_cast<long long>(tok) * a.ld;
  if (wrp == 0) {
    const int g = head / (a.heads / a.kv_heads);
    const T *q = row + a.q_off + static_cast<long long>(g) * D, *k = row + a.k_off + static_cast<long long>(g) * D;
    float qq = 0.f, kk = 0.f, qk = 0.f;
    for (int i = lane; i < D; i += 32) {
      const float x = ld(q + i), y = ld(k + i);
      qs[i] = x; ks[i] = y;
      qq = fmaf(x, x, qq); kk = fmaf(y, y, kk); qk = fmaf(x, y, qk);
    }
    for (int o = 16; o > 0; o >>= 1) {
      qq += __shfl_xor_sync(0xffffffffu, qq, o);
      kk += __shfl_xor_sync(0xffffffffu, kk, o);
      qk += __shfl_xor_sync(0xffffffffu, qk, o);
    }
    const float iq = a.q_scale / sqrtf(qq + a.unit_eps), ik = 1.0f / sqrtf(kk + a.unit_eps);
    for (int i = lane; i < 16 * RPT; i += 32) {
      qs[i] = i < D ? qs[i] * iq : 0.f;
      ks[i] = i < D ? ks[i] * ik : 0.f;
    }
    if (lane == 0) sc[2] = qk * iq * ik;
  } else if (tid == 32) {
    const float b = ld(static_cast<const T*>(a.beta_pre) + static_cast<long long>(tok) * a.ld_gate + head);
    const float d = softplusf_(ld(static_cast<const T*>(a.dt_pre) + static_cast<long long>(tok) * a.ld_gate + head) + a.dt_bias[head]);
    sc[0] = expf(a.rate[head] * d);
    sc[1] = 1.0f / (1.0f + expf(-b));
  }
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (live) {
    const T* vp = row + a.v_off + static_cast<long long>(head) * Dv + j0;
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = ld(vp + e);
  }
  __syncthreads();
  const float decay = sc[0];
  float sk[4] = {0.f, 0.f, 0.f, 0.f}, sq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int m = 0; m < RPT; ++m) {
    const float k = ks[r0 + 16 * m], q = qs[r0 + 16 * m], s4[4] = {S[m].x, S[m].y, S[m].z, S[m].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) { sk[e] = fmaf(s4[e], k, sk[e]); sq[e] = fmaf(s4[e], q, sq[e]); }
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    sk[e] += __shfl_xor_sync(0xffffffffu, sk[e], 16);
    sq[e] += __shfl_xor_sync(0xffffffffu, sq[e], 16);
  }
  if (lane < 16) {
    *reinterpret_cast<float4*>(&part[0][wrp][jc]) = make_float4(sk[0], sk[1], sk[2], sk[3]);
    *reinterpret_cast<float4*>(&part[1][wrp][jc]) = make_float4(sq[0], sq[1], sq[2], sq[3]);
  }
  __syncthreads();
  float u[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float tk = 0.f;
#pragma unroll
    for (int w = 0; w < kStepWarps; ++w) tk += part[0][w][jc + e];
    u[e] = sc[1] * fmaf(-decay, tk, v[e]);
  }
  if (r0 == 0 && live) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float tq = 0.f;
#pragma unroll
      for (int w = 0; w < kStepWarps; ++w) tq += part[1][w][jc + e];
      a.o[static_cast<long long>(tok) * (static_cast<long long>(a.heads) * Dv) + static_cast<long long>(head) * Dv + j0 + e] = fmaf(sc[2], u[e], decay * tq);
    }
  }
  if (live) {
#pragma unroll
    for (int m = 0; m < RPT; ++m) {
      const int i = r0 + 16 * m;
      const float k = ks[i];
      if (i < D)
        *reinterpret_cast<float4*>(Sg + static_cast<long long>(i) * Dv) =
            make_float4(fmaf(k, u[0], decay * S[m].x), fmaf(k, u[1], decay * S[m].y), fmaf(k, u[2], decay * S[m].z), fmaf(k, u[3], decay * S[m].w));
    }
  }
}

}  // namespace

int delta_scan(const DeltaArgs& a, cudaStream_t st, int max_rows) {
  if (a.nseq <= 0 || a.T <= 0) return 0;
  if (!a.qkv || !a.beta_pre || !a.dt_pre || !a.dt_bias || !a.rate || !a.states || !a.seqs || !a.o || a.heads < 1 || a.kv_heads < 1 ||
      a.heads % a.kv_heads || a.dim < 1 || a.vdim < 1) return -1;
  if (delta_chunk_fits(a)) {
    // steps that bring portions (B200_DELTA_CHUNK: A/B knob, the mean portion from which the chunked form runs; 0 = never)
    const char* e = getenv("B200_DELTA_CHUNK");
    const int from = e ? atoi(e) : 8;
    if (from > 0 && a.T >= static_cast<long long>(from) * a.nseq) return delta_chunk(a, st, max_rows);
  }
  // B200_SCAN_STEP: A/B knob, 0 = single tokens stay in the scan, 1 = never there where the pass takes their sizes.  fp32 models stay there,
  // whose outputs are promised to be the same bits however a sequence was cut into steps
  const char* se = getenv("B200_SCAN_STEP");
  if (a.t == DT_BF16 && a.T == a.nseq && a.dim <= 256 && a.vdim % 4 == 0 && reinterpret_cast<uintptr_t>(a.states) % 16 == 0 &&
      (se ? atoi(se) != 0 : rules::single_step_pays(static_cast<long long>(a.heads) * a.nseq, a.dim, a.vdim, true, sm_count()))) {
    dim3 grid((a.vdim + kStepCols - 1) / kStepCols, a.heads, a.nseq);
    if (a.dim <= 64) launch_pdl(delta_step_kernel<bf16, 4>, grid, kStepWarps * 32, 0, st, a);
    else if (a.dim <= 128) launch_pdl(delta_step_kernel<bf16, 8>, grid, kStepWarps * 32, 0, st, a);
    else launch_pdl(delta_step_kernel<bf16, 16>, grid, kStepWarps * 32, 0, st, a);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
  }
  int P = 1;
  while (P * 4 * kPieces < a.dim) P <<= 1;
  if (P > 32) return -1;   // dim <= 1024
  const int M = (a.dim + 4 * P - 1) / (4 * P), cols = kThreads / P;
  auto smem_for = [&](int G) { return static_cast<size_t>(G) * (2 * 4 * P * M + 2 * cols + 3) * sizeof(float); };
  int G = kGroup;
  while (G > 1 && smem_for(G) > 44 * 1024) G >>= 1;
  dim3 grid((a.vdim + cols - 1) / cols, a.heads, a.nseq);
  if (a.t == DT_BF16) delta_scan_kernel<bf16><<<grid, kThreads, smem_for(G), st>>>(a, P, M, G);
  else delta_scan_kernel<float><<<grid, kThreads, smem_for(G), st>>>(a, P, M, G);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace b200
