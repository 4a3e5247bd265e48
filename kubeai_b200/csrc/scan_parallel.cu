// The recurrent scan (mixers.h GlaArgs) for steps of prompt portions, every chunk of 64 tokens by itself: learned decays per
// key channel (gated linear attention, HGRN2) and scalar gates per token (mLSTM with its normaliser).
//
// With l_t the log decay of token t (a vector over the key channels), S <- diag(e^l_t) S + k_t v_t^T and o_t = S^T q_t unroll
// inside a chunk, whose incoming state is S_0 and c_t = l_1 + ... + l_t, to
//
//   o_t  = S_0^T (q_t e^c_t) + sum_{j <= t} (sum_i q_ti k_ji e^(c_ti - c_ji)) v_j,
//   S'   = diag(e^c_last) S_0 + sum_j (k_j e^(c_last - c_j)) v_j^T.
//
// Three launches: the sums over a chunk's own tokens for all (chunk, head) at once, a pass over them that turns each into the
// chunk's incoming state (elementwise, in place, and the slot's new state), the outputs for all (chunk, head) at once.  The
// token-by-token form (gla.cu) is a chain as long as the longest sequence on as many CTAs as there are heads and sequences:
// HGRN2, 16 heads of 128 x 128, 3 sequences of 455 to 2275 tokens took 3255 us there.
//
// Precision is that of fp32.  No factor is the inverse of a decay: a chunk's four blocks of 16 tokens carry their queries from
// the block's start and their keys to its end, both with exponents of at most 0, and what lies between two blocks is a third
// such factor; the blocks on the diagonal are scanned token by token in fp32 as the plain form does.  Every fp32 operand of a
// tensor-core product is split into three bf16 terms: all three against values, which are bf16 as the projection left them,
// the six term pairs down to 2^-24 against another fp32 operand.  Log decays are sums of at most 64 terms of one sign.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "launch.h"
#include "mixers.h"
#include "seq_tiles.cuh"
#include "mma_frag.cuh"

namespace b200 {
namespace {

using namespace frag;
typedef __nv_bfloat16 bf16;
constexpr int kQ = 64, kB = 16;             // tokens per chunk, per block
constexpr int kMaxD = 128, kCols = 128;     // key channels at most, value columns per CTA
constexpr int kThreads = 256;
constexpr int kLd = 136;                    // leading dimension of every shared tile: fragment rows fall into distinct banks
constexpr float kLowest = -87.f;            // log decays below it are as good as zero in fp32

enum Mode { VEC_Z = 0, VEC_FGATE = 1, SCALAR = 2 };

struct Work {
  float *s, *d, *n, *la;   // [chunk][head][dim][vdim] sums, then incoming states; [chunk][head][dim] decays, normaliser; [T][heads * dim]
};

__device__ __forceinline__ float floor_log(float x) { return x < kLowest ? kLowest : x; }   // keeps NaN
__device__ __forceinline__ float bf(const bf16* p) { return __bfloat162float(__ldg(p)); }

// forget gate pre-activation -> (log decay, key); 1 - f keeps its low bits where f is near 1, and f where it is near 0
__device__ __forceinline__ void forget_gate(float g, float lower, float* la, float* key) {
  const float e = expf(-fabsf(g)), r = 1.0f / (1.0f + e), er = e * r;
  const float hi = g >= 0.f ? r : er, lo = g >= 0.f ? er : r;
  const float f = fmaf(1.0f - lower, hi, lower), w = (1.0f - lower) * lo;
  *key = w;
  *la = floor_log(f > 0.5f ? log1pf(-w) : logf(f));
}
// log decay and key scale of a token's scalar gates
__device__ __forceinline__ void scalar_gate(const GlaArgs& a, long long row, int head, float* la, float* ks) {
  *la = floor_log(logf(__ldg(a.tok_decay + row * a.heads + head)));
  *ks = __ldg(a.tok_kscale + row * a.heads + head);
}

// z -> log decay in place: inv_tau * logsigmoid(z + bias)
__global__ void log_decay_kernel(float* z, const float* bias, int HD, float inv_tau, long long total) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const float v = z[i] + bias[i % HD];
  z[i] = floor_log((fminf(v, 0.f) - log1pf(expf(-fabsf(v)))) * inv_tau);
}

// 64 tokens x 128 columns of values into shared memory; zeros past the portion and past the last column
__device__ __forceinline__ void fetch_values(const GlaArgs& a, bf16* Vs, int tok0, int q, int head, int p0) {
  const bf16* base = static_cast<const bf16*>(a.qkv) + a.v_off + head * a.vdim + p0;
  for (int e = threadIdx.x; e < kQ * (kCols / 8); e += kThreads) {
    const int t = e / (kCols / 8), c = (e % (kCols / 8)) * 8;
    bf16* d = Vs + t * kLd + c;
    if (t < q && p0 + c < a.vdim) cp_async16(smem_addr(d), base + static_cast<long long>(tok0 + t) * a.ld + c);
    else *reinterpret_cast<uint4*>(d) = make_uint4(0, 0, 0, 0);
  }
}

// a chunk's scalar gates into shared memory (log decays, key scales; 0 past the portion); ends with a barrier
__device__ __forceinline__ void fetch_gates(const GlaArgs& a, float* gates, int tok0, int q, int head) {
  if (threadIdx.x < kQ) {
    float la = 0.f, ks = 0.f;
    if (threadIdx.x < q) scalar_gate(a, tok0 + threadIdx.x, head, &la, &ks);
    gates[threadIdx.x] = la;
    gates[kQ + threadIdx.x] = ks;
  }
  __syncthreads();
}

// ---------------------------------------------------------------- a chunk's own sums
// grid (chunks, heads, column blocks).  A thread owns a key channel and half of the chunk's tokens; its keys, carried to the
// chunk's end, go to shared memory in three terms and are the transposed left operand of keys^T values.
constexpr int kSumSmem = 3 * kQ * kLd * 2 + kQ * kLd * 2 + 2 * kMaxD * 8 + 2 * kMaxD * 4 + 2 * kQ * 4;
template <int MODE, bool NRM>
__global__ void __launch_bounds__(kThreads, 2) chunk_sums_kernel(GlaArgs a, Work w) {
  extern __shared__ __align__(16) unsigned char smraw[];
  bf16* Ks = reinterpret_cast<bf16*>(smraw);     // [3][kQ][kLd]
  bf16* Vs = Ks + 3 * kQ * kLd;                  // [kQ][kLd]
  double* half = reinterpret_cast<double*>(Vs + kQ * kLd);   // [2][kMaxD] log decay over half of the tokens
  float* nsum = reinterpret_cast<float*>(half + 2 * kMaxD);  // [2][kMaxD]
  float* gates = nsum + 2 * kMaxD;               // [2][kQ] a scalar gate's log decays and key scales
  int seq, chunk;
  if (!find_tile(a.seqs, a.nseq, kQ, blockIdx.x, &seq, &chunk)) return;
  const int head = blockIdx.y, p0 = blockIdx.z * kCols, D = a.dim, P = a.vdim, HD = a.heads * D;
  const int tok0 = a.seqs[seq * 8] + chunk * kQ, q = min(kQ, a.seqs[seq * 8 + 1] - chunk * kQ);
  const int tid = threadIdx.x, lane = tid & 31, wrp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  fetch_values(a, Vs, tok0, q, head, p0);
  if (MODE == SCALAR) fetch_gates(a, gates, tok0, q, head);
  const int i = tid & (kMaxD - 1), hf = tid / kMaxD;
  const bool ch = i < D;
  float la[kQ / 2], kv[kQ / 2];
  {
    const bf16* kp = static_cast<const bf16*>(a.qkv) + a.k_off + (head / a.group) * D + i;
    const float fb = MODE == VEC_FGATE && ch ? __ldg(a.z_bias + head * D + i) : 0.f, fl = MODE == VEC_FGATE && ch ? __ldg(a.fgate_lower + head * D + i) : 0.f;
    double sum = 0.0;
#pragma unroll
    for (int jj = 0; jj < kQ / 2; ++jj) {
      const int j = hf * (kQ / 2) + jj;
      la[jj] = 0.f; kv[jj] = 0.f;
      if (ch && j < q) {
        const long long row = tok0 + j;
        float k = bf(kp + row * a.ld);
        if (MODE == VEC_Z) la[jj] = __ldg(a.z + row * HD + head * D + i);
        if (MODE == VEC_FGATE) {
          forget_gate(k + fb, fl, &la[jj], &k);
          if (blockIdx.z == 0) w.la[row * HD + head * D + i] = la[jj];
        }
        if (MODE == SCALAR) { la[jj] = gates[j]; k *= gates[kQ + j]; }
        kv[jj] = k * a.k_scale;
      }
      sum += la[jj];
    }
    half[hf * kMaxD + i] = sum;
  }
  __syncthreads();
  {
    double rest = hf == 0 ? half[kMaxD + i] : 0.0;    // log decay from behind the token to the chunk's end
    float ns = 0.f;
#pragma unroll
    for (int jj = kQ / 2 - 1; jj >= 0; --jj) {
      float k = kv[jj] * expf(static_cast<float>(rest));
      rest += la[jj];
      if (NRM) ns += k;
      bf16* d = Ks + (hf * (kQ / 2) + jj) * kLd + i;
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        const bf16 b = __float2bfloat16_rn(k);
        d[s * kQ * kLd] = b;
        k -= __bfloat162float(b);
      }
    }
    const long long r = (static_cast<long long>(blockIdx.x) * a.heads + head) * D + i;
    if (hf == 0 && ch && blockIdx.z == 0) w.d[r] = expf(static_cast<float>(rest));
    if (NRM) nsum[hf * kMaxD + i] = ns;
  }
  cp_async_wait_all();
  __syncthreads();
  if (NRM && tid < D && blockIdx.z == 0) w.n[(static_cast<long long>(blockIdx.x) * a.heads + head) * D + tid] = nsum[tid] + nsum[kMaxD + tid];
  if (16 * wrp >= D) return;
  float acc[kCols / 8][4];
#pragma unroll
  for (int nt = 0; nt < kCols / 8; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
  const int ncol = min(kCols, P - p0);
#pragma unroll
  for (int jb = 0; jb < kQ / kB; ++jb) {
    if (jb * kB >= q) break;
    uint32_t af[3][4];
#pragma unroll
    for (int s = 0; s < 3; ++s) ldsm_x4_trans(af[s], at_addr(Ks + s * kQ * kLd, kLd, jb * kB, 16 * wrp, lane));
#pragma unroll
    for (int np = 0; np < kCols / 16; ++np) {
      if (np * 16 < ncol) {
        uint32_t b[4];
        ldsm_x4_trans(b, bt_addr(Vs, kLd, jb * kB, np * 16, lane));
#pragma unroll
        for (int s = 2; s >= 0; --s) {
          mma(acc[2 * np], af[s], b[0], b[1]);
          mma(acc[2 * np + 1], af[s], b[2], b[3]);
        }
      }
    }
  }
  float* out = w.s + ((static_cast<long long>(blockIdx.x) * a.heads + head) * D + 16 * wrp + g) * P + p0 + 2 * t4;
#pragma unroll
  for (int nt = 0; nt < kCols / 8; ++nt)
    if (nt * 8 < ncol) {
      *reinterpret_cast<float2*>(out + nt * 8) = make_float2(acc[nt][0], acc[nt][1]);
      *reinterpret_cast<float2*>(out + 8ll * P + nt * 8) = make_float2(acc[nt][2], acc[nt][3]);
    }
}

// ---------------------------------------------------------------- sums -> incoming states
// grid (four state entries per thread, heads, sequences): S <- d S + sum chunk by chunk, each sum replaced by the state in
// front of it; the loads of several chunks are in flight at once.
template <bool NRM>
__global__ void __launch_bounds__(kThreads) chunk_states_kernel(GlaArgs a, Work w) {
  const int seq = blockIdx.z, head = blockIdx.y, D = a.dim, P = a.vdim, lane = threadIdx.x & 31;
  int first = 0;
  for (int s0 = 0; s0 < seq; s0 += 32) {
    int c = s0 + lane < seq ? (a.seqs[(s0 + lane) * 8 + 1] + kQ - 1) / kQ : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    first += c;
  }
  const int nc = (a.seqs[seq * 8 + 1] + kQ - 1) / kQ, slot = a.seqs[seq * 8 + 3];
  const bool old = a.seqs[seq * 8 + 2] > 0;
  const long long cstep = static_cast<long long>(a.heads) * D, hrow = static_cast<long long>(first) * cstep + head * D;
  const int e = (blockIdx.x * kThreads + threadIdx.x) * 4;
  constexpr int U = 4;
  if (e < D * P) {
    const int i = e / P;
    float* sp = w.s + hrow * P + e;
    const float* dp = w.d + hrow + i;
    float4* state = reinterpret_cast<float4*>(a.states + (static_cast<long long>(slot) * a.heads + head) * D * P + e);
    float4 s = old ? *state : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c = 0; c < nc; c += U) {
      float4 t[U];
      float d[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (c + u < nc) { t[u] = *reinterpret_cast<const float4*>(sp + (c + u) * cstep * P); d[u] = dp[(c + u) * cstep]; }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (c + u < nc) {
          if (old || c + u > 0) *reinterpret_cast<float4*>(sp + (c + u) * cstep * P) = s;
          s = make_float4(fmaf(d[u], s.x, t[u].x), fmaf(d[u], s.y, t[u].y), fmaf(d[u], s.z, t[u].z), fmaf(d[u], s.w, t[u].w));
        }
    }
    if (nc > 0) *state = s;
  }
  if (NRM && blockIdx.x == 0 && threadIdx.x < D) {
    const int i = threadIdx.x;
    float* st = a.nstate + (static_cast<long long>(slot) * a.heads + head) * D + i;
    float s = old ? *st : 0.f;
    for (int c = 0; c < nc; ++c) {
      float* p = w.n + hrow + c * cstep + i;
      const float t = *p;
      *p = s;
      s = fmaf(w.d[hrow + c * cstep + i], s, t);
    }
    if (nc > 0) *st = s;
  }
}

// ---------------------------------------------------------------- a chunk's outputs
__device__ __forceinline__ void mma6(float* c, const uint32_t (*A)[4], const uint32_t (*B)[2]) {
  mma(c, A[2], B[0][0], B[0][1]);
  mma(c, A[0], B[2][0], B[2][1]);
  mma(c, A[1], B[1][0], B[1][1]);
  mma(c, A[1], B[0][0], B[0][1]);
  mma(c, A[0], B[1][0], B[1][1]);
  mma(c, A[0], B[0][0], B[0][1]);
}
__device__ __forceinline__ bool finite2(uint32_t x) { return (x & 0x7f80u) != 0x7f80u && (x & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ float2 mul2(float2 x, float2 y) { return make_float2(x.x * y.x, x.y * y.y); }

// grid (chunks, heads, column blocks).  Warp w: tokens of block w / 2, value columns of half w % 2.
constexpr int kRows = 32;     // state rows staged per round, in three terms, where the keys were
struct OutSmem {
  float Q[kQ * kLd];          // queries, then carried from their block's start
  float K[kQ * kLd];          // keys, then carried to their block's end; then [3][kRows][kLd] bf16 terms of the state
  bf16 V[kQ * kLd];
  float diag[8][kB][kB + 1];  // scores inside a block, one half of the key channels each
  float tot[4][kMaxD];        // log decay over a block
  float from0[4][kMaxD];      // decay from the chunk's start to a block's start
  float mid[3][kMaxD];        // decay over block 1, block 2, both
  float n0[kMaxD];            // incoming normaliser
  float gates[2 * kQ];        // scalar gates
};
static_assert(3 * kRows * kLd * 2 <= kQ * kLd * 4, "the state's terms fit where the keys were");
template <int MODE, bool NRM>
__global__ void __launch_bounds__(kThreads, 2) chunk_out_kernel(GlaArgs a, Work w) {
  extern __shared__ __align__(16) unsigned char smraw[];
  OutSmem& sm = *reinterpret_cast<OutSmem*>(smraw);
  int seq, chunk;
  if (!find_tile(a.seqs, a.nseq, kQ, blockIdx.x, &seq, &chunk)) return;
  const int head = blockIdx.y, p0 = blockIdx.z * kCols, D = a.dim, P = a.vdim, HD = a.heads * D, nk = D / 16;
  const int tok0 = a.seqs[seq * 8] + chunk * kQ, q = min(kQ, a.seqs[seq * 8 + 1] - chunk * kQ);
  const bool has_state = chunk > 0 || a.seqs[seq * 8 + 2] > 0;
  const int tid = threadIdx.x, lane = tid & 31, wrp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const float* lap = MODE == VEC_Z ? a.z : w.la;
  fetch_values(a, sm.V, tok0, q, head, p0);
  if (MODE == SCALAR) fetch_gates(a, sm.gates, tok0, q, head);
  {
    const int i = tid & (kMaxD - 1), hf = tid / kMaxD;
    const bool ch = i < D;
    const bf16* base = static_cast<const bf16*>(a.qkv) + (head / a.group) * D + i;
    const float fb = MODE == VEC_FGATE && ch ? __ldg(a.z_bias + head * D + i) : 0.f, fl = MODE == VEC_FGATE && ch ? __ldg(a.fgate_lower + head * D + i) : 0.f;
#pragma unroll 8
    for (int jj = 0; jj < kQ / 2; ++jj) {
      const int j = hf * (kQ / 2) + jj;
      float qv = 0.f, kv = 0.f;
      if (ch && j < q) {
        const long long row = tok0 + j;
        qv = bf(base + row * a.ld + a.q_off);
        kv = bf(base + row * a.ld + a.k_off);
        if (a.act == GLA_ACT_SILU_Q) qv = qv / (1.0f + expf(-qv));
        if (MODE == VEC_FGATE) { float l; forget_gate(kv + fb, fl, &l, &kv); }
        if (MODE == SCALAR) kv *= sm.gates[kQ + j];
      }
      sm.Q[j * kLd + i] = qv * a.q_scale;
      sm.K[j * kLd + i] = kv * a.k_scale;
    }
    if (NRM && tid < kMaxD) sm.n0[tid] = has_state && tid < D ? w.n[(static_cast<long long>(blockIdx.x) * a.heads + head) * D + tid] : 0.f;
  }
  __syncthreads();
  // ---- blocks on the diagonal, token by token: a lane holds the decayed keys of its two channels
  {
    const int b = wrp >> 1, c = (wrp & 1) * 64 + 2 * lane;
    float2 W[kB];
#pragma unroll
    for (int t = 0; t < kB; ++t) {
      const int tt = b * kB + t;
      float2 al = make_float2(1.f, 1.f);
      if (tt < q && t > 0) {
        if (MODE == SCALAR) al.x = al.y = expf(sm.gates[tt]);
        else if (c < D) {
          const float2 l = *reinterpret_cast<const float2*>(lap + static_cast<long long>(tok0 + tt) * HD + head * D + c);
          al = make_float2(expf(l.x), expf(l.y));
        }
      }
      const float2 qt = *reinterpret_cast<const float2*>(sm.Q + tt * kLd + c), kt = *reinterpret_cast<const float2*>(sm.K + tt * kLd + c);
      float p[kB];
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        if (j < t) W[j] = mul2(W[j], al);
        if (j == t) W[j] = kt;
        p[j] = j <= t ? fmaf(qt.x, W[j].x, qt.y * W[j].y) : 0.f;
      }
      // sixteen sums over the warp: each step halves the number a lane holds
#pragma unroll
      for (int o = 16, n = 8; n >= 1; o >>= 1, n >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < n) {
            const float keep = up ? p[j + n] : p[j], send = up ? p[j] : p[j + n];
            p[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
      }
      p[0] += __shfl_xor_sync(0xffffffffu, p[0], 1);
      if (!(lane & 1)) sm.diag[wrp][t][lane >> 1] = p[0];
    }
  }
  __syncthreads();
  // ---- queries from their block's start, keys to their block's end
  {
    const int i = tid & (kMaxD - 1), hf = tid / kMaxD;
    if (i < D) {
#pragma unroll
      for (int bb = 0; bb < 2; ++bb) {
        const int b = 2 * hf + bb;
        float la[kB];
#pragma unroll
        for (int t = 0; t < kB; ++t) {
          const int tt = b * kB + t;
          la[t] = 0.f;
          if (tt < q) {
            if (MODE == SCALAR) la[t] = sm.gates[tt];
            else la[t] = lap[static_cast<long long>(tok0 + tt) * HD + head * D + i];
          }
        }
        float run = 0.f;
#pragma unroll
        for (int t = 0; t < kB; ++t) { run += la[t]; sm.Q[(b * kB + t) * kLd + i] *= expf(run); }
        sm.tot[b][i] = run;
        run = 0.f;
#pragma unroll
        for (int t = kB - 1; t >= 0; --t) { sm.K[(b * kB + t) * kLd + i] *= expf(run); run += la[t]; }
      }
    }
  }
  __syncthreads();
  if (tid < D) {
    const float l0 = sm.tot[0][tid], l1 = sm.tot[1][tid], l2 = sm.tot[2][tid];
    sm.from0[0][tid] = 1.f; sm.from0[1][tid] = expf(l0); sm.from0[2][tid] = expf(l0 + l1); sm.from0[3][tid] = expf(l0 + l1 + l2);
    sm.mid[0][tid] = expf(l1); sm.mid[1][tid] = expf(l2); sm.mid[2][tid] = expf(l1 + l2);
  }
  cp_async_wait_all();
  __syncthreads();
  // ---- scores of the warp's 16 tokens against the blocks in front
  const int b = wrp >> 1, half = wrp & 1, ncol = min(64, P - p0 - 64 * half);
  const float* Qr = sm.Q + (b * kB + g) * kLd + 2 * t4;
  float sc[3][2][4];
#pragma unroll
  for (int x = 0; x < 3; ++x)
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) sc[x][nt][0] = sc[x][nt][1] = sc[x][nt][2] = sc[x][nt][3] = 0.f;
  const bool live = b * kB < q;
  if (live && b > 0) {
    for (int ks = 0; ks < nk; ++ks) {
      uint32_t A[3][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float2 v = *reinterpret_cast<const float2*>(Qr + (r & 1) * 8 * kLd + ks * 16 + (r >> 1) * 8);
        split3(v.x, v.y, &A[0][r], &A[1][r], &A[2][r]);
      }
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        if (x < b) {
          // from block x's end to block b's start: nothing, block 1, block 2 or both
          const float* m = b - x == 1 ? nullptr : (b - x == 3 ? sm.mid[2] : sm.mid[x]);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            uint32_t B[3][2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const int col = ks * 16 + r * 8 + 2 * t4;
              float2 v = *reinterpret_cast<const float2*>(sm.K + (x * kB + nt * 8 + g) * kLd + col);
              if (m) v = mul2(v, *reinterpret_cast<const float2*>(m + col));
              split3(v.x, v.y, &B[0][r], &B[1][r], &B[2][r]);
            }
            mma6(sc[x][nt], A, B);
          }
        }
      }
    }
  }
  float o[8][4];
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) o[nt][0] = o[nt][1] = o[nt][2] = o[nt][3] = 0.f;
  float nq[2] = {0.f, 0.f};      // n . q of tokens g and g + 8, this lane's part
  auto values = [&](const float (*s)[4], int blk) {     // o += scores (16 tokens x 16 keys) * values of block blk
    uint32_t A[3][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) split3(s[r >> 1][2 * (r & 1)], s[r >> 1][2 * (r & 1) + 1], &A[0][r], &A[1][r], &A[2][r]);
    if (NRM) {
      nq[0] += (s[0][0] + s[0][1]) + (s[1][0] + s[1][1]);
      nq[1] += (s[0][2] + s[0][3]) + (s[1][2] + s[1][3]);
    }
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      if (np * 16 < ncol) {
        uint32_t v[4];
        ldsm_x4_trans(v, bt_addr(sm.V, kLd, blk * kB, half * 64 + np * 16, lane));
#pragma unroll
        for (int k = 2; k >= 0; --k) {
          mma(o[2 * np], A[k], v[0], v[1]);
          mma(o[2 * np + 1], A[k], v[2], v[3]);
        }
      }
    }
  };
  if (live) {
#pragma unroll
    for (int x = 0; x < 3; ++x)
      if (x < b) values(sc[x], x);
    float d[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = g + 8 * (e >> 1), j = nt * 8 + 2 * t4 + (e & 1);
        d[nt][e] = sm.diag[2 * b][t][j] + sm.diag[2 * b + 1][t][j];
      }
    // A token's weight for the block's later keys is 0, which a product would turn into NaN where their value is infinite or NaN:
    // such a block is summed key by key, up to the token.
    bool finite = true;
#pragma unroll
    for (int e = 0; e < kB * 8; e += 32) {
      const uint4 v = *reinterpret_cast<const uint4*>(sm.V + (b * kB + (e + lane) / 8) * kLd + half * 64 + (e + lane) % 8 * 8);
      finite = finite && finite2(v.x) && finite2(v.y) && finite2(v.z) && finite2(v.w);
    }
    if (__all_sync(0xffffffffu, finite)) {
      values(d, b);
    } else {
      if (NRM) {
        nq[0] += (d[0][0] + d[0][1]) + (d[1][0] + d[1][1]);
        nq[1] += (d[0][2] + d[0][3]) + (d[1][2] + d[1][3]);
      }
      for (int r = 0; r < 2; ++r)
        for (int j = 0; j <= g + 8 * r; ++j) {
          const float w = sm.diag[2 * b][g + 8 * r][j] + sm.diag[2 * b + 1][g + 8 * r][j];
          const bf16* v = sm.V + (b * kB + j) * kLd + half * 64 + 2 * t4;
#pragma unroll
          for (int nt = 0; nt < 8; ++nt) {
            if (r == 0) { o[nt][0] = fmaf(w, __bfloat162float(v[nt * 8]), o[nt][0]); o[nt][1] = fmaf(w, __bfloat162float(v[nt * 8 + 1]), o[nt][1]); }
            else { o[nt][2] = fmaf(w, __bfloat162float(v[nt * 8]), o[nt][2]); o[nt][3] = fmaf(w, __bfloat162float(v[nt * 8 + 1]), o[nt][3]); }
          }
        }
    }
  }
  // ---- the incoming state's part
  if (has_state) {
    bf16* Ss = reinterpret_cast<bf16*>(sm.K);
    const float* S = w.s + ((static_cast<long long>(blockIdx.x) * a.heads + head) * D) * P + p0;
    const int r0 = tid >> 5, c0 = (tid & 31) * 4;      // rows r0, r0 + 8, ... of a round
    float4 nx[kRows / 8];
    auto fetch = [&](int i0) {
#pragma unroll
      for (int u = 0; u < kRows / 8; ++u) {
        const int i = i0 + r0 + 8 * u;
        nx[u] = i < D && p0 + c0 < P ? *reinterpret_cast<const float4*>(S + static_cast<long long>(i) * P + c0) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    fetch(0);
    for (int i0 = 0; i0 < D; i0 += kRows) {
      __syncthreads();       // the keys, or the last rows, are no longer read
#pragma unroll
      for (int u = 0; u < kRows / 8; ++u) {
        uint32_t x[3], y[3];
        split3(nx[u].x, nx[u].y, &x[0], &x[1], &x[2]);
        split3(nx[u].z, nx[u].w, &y[0], &y[1], &y[2]);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint2*>(Ss + (k * kRows + r0 + 8 * u) * kLd + c0) = make_uint2(x[k], y[k]);
      }
      __syncthreads();
      if (i0 + kRows < D) fetch(i0 + kRows);
      if (!live) continue;
#pragma unroll
      for (int kk = 0; kk < kRows / 16; ++kk) {
        if (i0 + kk * 16 < D) {
          uint32_t A[3][4];
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int col = i0 + kk * 16 + (r >> 1) * 8;
            float2 v = *reinterpret_cast<const float2*>(Qr + (r & 1) * 8 * kLd + col);
            v = mul2(v, *reinterpret_cast<const float2*>(sm.from0[b] + col + 2 * t4));
            if (NRM) {
              const float2 n = *reinterpret_cast<const float2*>(sm.n0 + col + 2 * t4);
              nq[r & 1] = fmaf(v.x, n.x, fmaf(v.y, n.y, nq[r & 1]));
            }
            split3(v.x, v.y, &A[0][r], &A[1][r], &A[2][r]);
          }
#pragma unroll
          for (int np = 0; np < 4; ++np) {
            if (np * 16 < ncol) {
              uint32_t t[3][4];
#pragma unroll
              for (int k = 0; k < 3; ++k) ldsm_x4_trans(t[k], bt_addr(Ss + k * kRows * kLd, kLd, kk * 16, half * 64 + np * 16, lane));
              const uint32_t B0[3][2] = {{t[0][0], t[0][1]}, {t[1][0], t[1][1]}, {t[2][0], t[2][1]}};
              const uint32_t B1[3][2] = {{t[0][2], t[0][3]}, {t[1][2], t[1][3]}, {t[2][2], t[2][3]}};
              mma6(o[2 * np], A, B0);
              mma6(o[2 * np + 1], A, B1);
            }
          }
        }
      }
    }
  }
  if (!live) return;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int t = b * kB + g + 8 * r;
    float n = nq[r];
    if (NRM) {
      n += __shfl_xor_sync(0xffffffffu, n, 1);
      n += __shfl_xor_sync(0xffffffffu, n, 2);
      if (t < q && half == 0 && t4 == 0 && blockIdx.z == 0) a.nq[static_cast<long long>(tok0 + t) * a.heads + head] = n;
    }
    if (t >= q) continue;
    float* out = a.o + static_cast<long long>(tok0 + t) * (a.heads * P) + head * P + p0 + 64 * half + 2 * t4;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
      if (nt * 8 < ncol) *reinterpret_cast<float2*>(out + nt * 8) = make_float2(o[nt][2 * r], o[nt][2 * r + 1]);
  }
}

template <int MODE, bool NRM>
int run(const GlaArgs& a, const Work& w, int chunks, cudaStream_t st) {
  static std::atomic<unsigned long long> attr[2];
  if (!ensure_dynamic_smem(chunk_sums_kernel<MODE, NRM>, kSumSmem, &attr[0]) || !ensure_dynamic_smem(chunk_out_kernel<MODE, NRM>, static_cast<int>(sizeof(OutSmem)), &attr[1])) return -2;
  const dim3 grid(chunks, a.heads, (a.vdim + kCols - 1) / kCols);
  chunk_sums_kernel<MODE, NRM><<<grid, kThreads, kSumSmem, st>>>(a, w);
  chunk_states_kernel<NRM><<<dim3((a.dim * a.vdim / 4 + kThreads - 1) / kThreads, a.heads, a.nseq), kThreads, 0, st>>>(a, w);
  chunk_out_kernel<MODE, NRM><<<grid, kThreads, sizeof(OutSmem), st>>>(a, w);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace

size_t scan_parallel_ws_floats(int tokens, int seqs, int heads, int dim, int vdim, bool fgate) {
  const size_t chunks = static_cast<size_t>(tokens) / kQ + seqs;
  return chunks * heads * dim * (static_cast<size_t>(vdim) + 2) + (fgate ? static_cast<size_t>(tokens) * heads * dim : 0);
}

bool scan_parallel_fits(const GlaArgs& a) {
  auto al = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  return a.par_ws && a.t == DT_BF16 && (a.act == GLA_ACT_NONE || a.act == GLA_ACT_SILU_Q) && !a.rope && !a.head_decay && !a.dt_pre && !a.tok_decay == !a.nstate && a.dim % 16 == 0 && a.dim <= kMaxD &&
         a.vdim % 8 == 0 && a.ld % 8 == 0 && a.v_off % 8 == 0 && al(a.qkv) && al(a.states) && al(a.o) && al(a.par_ws) && (a.tok_decay || a.fgate_lower || al(a.z)) &&
         scan_parallel_ws_floats(a.T, a.nseq, a.heads, a.dim, a.vdim, a.fgate_lower != nullptr) <= a.par_ws_floats;
}

int scan_parallel(const GlaArgs& a, cudaStream_t st) {
  if (!scan_parallel_fits(a)) return -1;
  const int chunks = a.T / kQ + a.nseq;
  const size_t rows = static_cast<size_t>(chunks) * a.heads * a.dim;
  Work w;
  w.s = a.par_ws;
  w.d = w.s + rows * a.vdim;
  w.n = w.d + rows;
  w.la = w.n + rows;
  if (a.tok_decay) return run<SCALAR, true>(a, w, chunks, st);
  if (a.fgate_lower) return run<VEC_FGATE, false>(a, w, chunks, st);
  const long long total = static_cast<long long>(a.T) * a.heads * a.dim;
  if (total > 0) log_decay_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, st>>>(a.z, a.z_bias, a.heads * a.dim, a.inv_tau, total);
  return run<VEC_Z, false>(a, w, chunks, st);
}

}  // namespace b200
