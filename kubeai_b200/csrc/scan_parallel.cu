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
// HGRN2, 16 heads of 128 x 128, 3 sequences of 455 to 2275 tokens took 3255 us there, 226 here (GLA 200, mLSTM 193; 380, 365 and
// 296 while a thread waited for each token's load before it issued the next one's: two thirds of both kernels' cycles).
//
// What bounds it: two CTAs of eight warps an SM (shared memory and registers allow no more) go through phases that each lean on
// something else: loads, the blocks on the diagonal (issue slots), scores and state (tensor cores, mma.sync: a third of the time
// at its peak rate).  Cycles of a CTA with a second one beside it, GLA: sums 7.8k loads, 3.4k terms, 7k products and stores; outputs
// 9.6k loads, 8.2k diagonal, 3.6k carrying, 6.5k scores, 5.3k values, 13k state.  Three CTAs of the first kernel an SM spill: slower.
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
#include <type_traits>

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
  float *s, *d, *n;   // [chunk][head][dim][vdim] sums, then incoming states; [chunk][head][dim] decays, normaliser
};

__device__ __forceinline__ float floor_log(float x) { return x < kLowest ? kLowest : x; }   // keeps NaN

// sigmoid(x) and sigmoid(-x) without a branch, so that the gates of several tokens are under way at once: quotients over
// d = 1 + e^-|x| from an approximate reciprocal with a Newton step each, whose residuals count what the rounding of d left out
__device__ __forceinline__ void sigmoids(float x, float* pos, float* neg) {
  const float e = expf(-fabsf(x)), d = 1.0f + e, dd = e - (d - 1.0f);
  float r = __fdividef(1.0f, d);
  r = fmaf(r, fmaf(-dd, r, fmaf(-d, r, 1.0f)), r);
  float er = e * r;
  er = fmaf(r, fmaf(-dd, er, fmaf(-d, er, e)), er);
  *pos = x >= 0.f ? r : er;
  *neg = x >= 0.f ? er : r;
}
// forget gate pre-activation -> (log decay, key); 1 - f keeps its low bits where f is near 1, and f where it is near 0.  There
// log f is that of the rounded f plus what the rounding left out, (1 - w) - f, over f (Kahan's way to log(1 + x); 1 - f is exact
// above a half): one logarithm, where two on either side of a branch had every warp take both, one token after the other (a
// gate 150 cycles of a warp's share of an SM, now 75; against 64 bits both the largest and the mean error are smaller).
__device__ __forceinline__ void forget_gate(float g, float lower, float* la, float* key) {
  float hi, lo;
  sigmoids(g, &hi, &lo);
  const float f = fmaf(1.0f - lower, hi, lower), w = (1.0f - lower) * lo;
  *key = w;
  const float left = f > 0.5f ? (1.0f - f) - w : 0.0f;    // over f = 1 - w: times 1 + w + w^2 + w^3
  *la = floor_log(logf(f) + fmaf(left * w, fmaf(w, 1.0f + w, 1.0f), left));
}
// log decay and key scale of a token's scalar gates
__device__ __forceinline__ void scalar_gate(const GlaArgs& a, long long row, int head, float* la, float* ks) {
  *la = floor_log(logf(__ldg(a.tok_decay + row * a.heads + head)));
  *ks = __ldg(a.tok_kscale + row * a.heads + head);
}

// z -> log decay in place: inv_tau * logsigmoid(z + bias); grid (tokens, blocks of 1024 channels)
__global__ void __launch_bounds__(256) log_decay_kernel(float* z, const float* bias, int HD, float inv_tau) {
  const int i = (blockIdx.y * 256 + threadIdx.x) * 4;
  if (i >= HD) return;
  float4* p = reinterpret_cast<float4*>(z + static_cast<long long>(blockIdx.x) * HD + i);
  const float4 x = *p;
  auto decay = [&](float a, int n) {
    const float v = a + __ldg(bias + i + n);
    return floor_log((fminf(v, 0.f) - log1pf(expf(-fabsf(v)))) * inv_tau);
  };
  *p = make_float4(decay(x.x, 0), decay(x.y, 1), decay(x.z, 2), decay(x.w, 3));
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

// 64 tokens x dim of keys into the first bf16 tile; what is past the portion or the last channel stays unwritten
__device__ __forceinline__ void fetch_keys(const GlaArgs& a, bf16* Ks, int tok0, int q, int head) {
  const bf16* base = static_cast<const bf16*>(a.qkv) + a.k_off + (head / a.group) * a.dim;
  for (int e = threadIdx.x; e < kQ * (kMaxD / 8); e += kThreads) {
    const int t = e / (kMaxD / 8), c = (e % (kMaxD / 8)) * 8;
    if (t >= q || c >= a.dim) continue;
    cp_async16(smem_addr(Ks + t * kLd + c), base + static_cast<long long>(tok0 + t) * a.ld + c);
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
  const int i = tid & (kMaxD - 1), hf = tid / kMaxD;
  const bool ch = i < D;
  float la[kQ / 2], kv[kQ / 2];
  // every load of the chunk is in flight before the first is waited for: the keys on their way to shared memory, where their
  // terms go afterwards, the decays to registers
  fetch_keys(a, Ks, tok0, q, head);
  if (MODE == VEC_Z) {
    const float* zp = a.z + static_cast<long long>(tok0) * HD + head * D + (ch ? i : 0);
#pragma unroll
    for (int jj = 0; jj < kQ / 2; ++jj) la[jj] = __ldg(zp + static_cast<long long>(min(hf * (kQ / 2) + jj, q - 1)) * HD);
  }
  if (MODE == SCALAR) fetch_gates(a, gates, tok0, q, head);
  cp_async_wait_all();
  __syncthreads();
  {
    const bf16* kp = Ks + i;
    const float fb = MODE == VEC_FGATE && ch ? __ldg(a.z_bias + head * D + i) : 0.f, fl = MODE == VEC_FGATE && ch ? __ldg(a.fgate_lower + head * D + i) : 0.f;
    double sum = 0.0;
#pragma unroll
    for (int jj = 0; jj < kQ / 2; ++jj) {
      const int j = hf * (kQ / 2) + jj;
      const bool in = ch && j < q;
      float k = __bfloat162float(kp[j * kLd]);
      if (MODE == VEC_FGATE) forget_gate(k + fb, fl, &la[jj], &k);
      if (MODE == SCALAR) { la[jj] = gates[j]; k *= gates[kQ + j]; }
      if (!in) la[jj] = 0.f;
      kv[jj] = in ? k * a.k_scale : 0.f;
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
  constexpr int U = 8;
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
// N tiles of one left operand, term pairs outside: neighbouring products go to different sums, so none waits for the one in front
template <int N>
__device__ __forceinline__ void mma6(float* const* c, const uint32_t (*A)[4], const uint32_t (*B)[3][2]) {
  constexpr int ta[6] = {2, 0, 1, 1, 0, 0}, tb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
  for (int p = 0; p < 6; ++p)
#pragma unroll
    for (int n = 0; n < N; ++n) mma(c[n], A[ta[p]], B[n][tb[p]][0], B[n][tb[p]][1]);
}
__device__ __forceinline__ bool finite2(uint32_t x) { return (x & 0x7f80u) != 0x7f80u && (x & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ float2 mul2(float2 x, float2 y) { return make_float2(x.x * y.x, x.y * y.y); }

// grid (chunks, heads, column blocks).  Warp w: tokens of block w / 2, key channels and then value columns of half w % 2.  All
// loads of a phase are issued before the first is waited for; a lane's queries, keys and decays are its own until the scores.
constexpr int kRows = 32;     // state rows staged per round, in three terms, where the keys were
struct OutSmem {
  float Q[kQ * kLd];          // queries, then carried from their block's start
  float K[kQ * kLd];          // keys, then carried to their block's end; then [3][kRows][kLd] bf16 terms of the state
  bf16 V[kQ * kLd];
  float diag[8][kB][kB + 1];  // scores inside a block, one half of the key channels each
  float cross[6][kB][24];     // scores between two blocks: of block b against x in b (b - 1) / 2 + x
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
  const int b = wrp >> 1, half = wrp & 1;
  const long long hrow = (static_cast<long long>(blockIdx.x) * a.heads + head) * D;
  fetch_values(a, sm.V, tok0, q, head, p0);
  // A lane's own part: the 16 tokens of its warp's block, two channels.  All of its loads are in flight before the first is waited
  // for (addresses of tokens and channels that are not there are those of ones that are).
  const int c = half * 64 + 2 * lane;
  const bool ch = c < D;
  float2 la[kB];               // log decays; scalar gates: in shared memory
  {
    uint32_t qr[kB], kr[kB];
    const int c1 = ch ? c : 0;
    const bf16* base = static_cast<const bf16*>(a.qkv) + (head / a.group) * D + c1;
#pragma unroll
    for (int t = 0; t < kB; ++t) {
      const long long row = tok0 + min(b * kB + t, q - 1);
      qr[t] = __ldg(reinterpret_cast<const unsigned int*>(base + row * a.ld + a.q_off));
      kr[t] = __ldg(reinterpret_cast<const unsigned int*>(base + row * a.ld + a.k_off));
      if (MODE == VEC_Z) la[t] = *reinterpret_cast<const float2*>(a.z + row * HD + head * D + c1);
    }
    float2 fb = make_float2(0.f, 0.f), fl = fb;
    if (MODE == VEC_FGATE) {
      fb = make_float2(__ldg(a.z_bias + head * D + c1), __ldg(a.z_bias + head * D + c1 + 1));
      fl = make_float2(__ldg(a.fgate_lower + head * D + c1), __ldg(a.fgate_lower + head * D + c1 + 1));
    }
    if (MODE == SCALAR) fetch_gates(a, sm.gates, tok0, q, head);
    const bool silu = a.act == GLA_ACT_SILU_Q;
#pragma unroll
    for (int t = 0; t < kB; ++t) {
      const int tt = b * kB + t;
      const bool in = ch && tt < q;
      float2 qv = make_float2(low(qr[t]), high(qr[t])), kv = make_float2(low(kr[t]), high(kr[t]));
      if (silu) {
        float2 s, rest;
        sigmoids(qv.x, &s.x, &rest.x);
        sigmoids(qv.y, &s.y, &rest.y);
        qv = mul2(qv, s);
      }
      if (MODE == VEC_FGATE) { forget_gate(kv.x + fb.x, fl.x, &la[t].x, &kv.x); forget_gate(kv.y + fb.y, fl.y, &la[t].y, &kv.y); }
      if (MODE == SCALAR) { kv.x *= sm.gates[kQ + tt]; kv.y *= sm.gates[kQ + tt]; }
      else if (!in) la[t] = make_float2(0.f, 0.f);
      *reinterpret_cast<float2*>(sm.Q + tt * kLd + c) = in ? make_float2(qv.x * a.q_scale, qv.y * a.q_scale) : make_float2(0.f, 0.f);
      *reinterpret_cast<float2*>(sm.K + tt * kLd + c) = in ? make_float2(kv.x * a.k_scale, kv.y * a.k_scale) : make_float2(0.f, 0.f);
    }
    if (NRM && tid < kMaxD) sm.n0[tid] = has_state && tid < D ? w.n[hrow + tid] : 0.f;
  }
  // ---- blocks on the diagonal, token by token: a lane holds the decayed keys of its two channels
  {
    float2 W[kB];
#pragma unroll
    for (int t = 0; t < kB; ++t) {
      const int tt = b * kB + t;
      float2 al = make_float2(1.f, 1.f);
      if (t > 0) {
        if (MODE == SCALAR) al.x = al.y = expf(sm.gates[tt]);
        else al = make_float2(expf(la[t].x), expf(la[t].y));
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
  // ---- the lane's queries from the block's start, its keys to the block's end
  if (ch) {
    float2 run = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = 0; t < kB; ++t) {
      if (MODE == SCALAR) la[t].x = la[t].y = sm.gates[b * kB + t];
      run.x += la[t].x; run.y += la[t].y;
      float2* p = reinterpret_cast<float2*>(sm.Q + (b * kB + t) * kLd + c);
      *p = mul2(*p, make_float2(expf(run.x), expf(run.y)));
    }
    *reinterpret_cast<float2*>(sm.tot[b] + c) = run;
    run = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = kB - 1; t >= 0; --t) {
      float2* p = reinterpret_cast<float2*>(sm.K + (b * kB + t) * kLd + c);
      *p = mul2(*p, make_float2(expf(run.x), expf(run.y)));
      run.x += la[t].x; run.y += la[t].y;
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
  // the state's first rows, on their way during the scores
  const float* S = w.s + hrow * P + p0;
  const int r0 = tid >> 5, c0 = (tid & 31) * 4;      // rows r0, r0 + 8, ... of a round
  float4 nx[kRows / 8];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int u = 0; u < kRows / 8; ++u) {
      const int i = i0 + r0 + 8 * u;
      nx[u] = i < D && p0 + c0 < P ? *reinterpret_cast<const float4*>(S + static_cast<long long>(i) * P + c0) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  if (has_state) fetch(0);
  // ---- scores against the blocks in front: six pairs of blocks, at most two for the two warps of a block, which take eight keys
  // each; block 0's warps have block 3's first pair
  const bool live = b * kB < q;
  const int ncol = min(64, P - p0 - 64 * half);
  const float* Qr = sm.Q + (b * kB + g) * kLd + 2 * t4;
  {
    const int qb = b == 0 ? 3 : b, x0 = b == 3 ? 1 : 0;
    const float* Qs = sm.Q + (qb * kB + g) * kLd + 2 * t4;
    auto scores = [&](auto pairs) {
      constexpr int N = decltype(pairs)::value;
      float sc[N][4];
      float* at[N];
      const float* m[N];       // from block x's end to block qb's start: nothing, block 1, block 2 or both
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const int x = x0 + n;
        at[n] = sc[n];
        sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.f;
        m[n] = qb - x == 1 ? nullptr : (qb - x == 3 ? sm.mid[2] : sm.mid[x]);
      }
      for (int ks = 0; ks < nk; ++ks) {
        uint32_t A[3][4], B[N][3][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float2 v = *reinterpret_cast<const float2*>(Qs + (r & 1) * 8 * kLd + ks * 16 + (r >> 1) * 8);
          split3(v.x, v.y, &A[0][r], &A[1][r], &A[2][r]);
        }
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int col = ks * 16 + r * 8 + 2 * t4;
            float2 v = *reinterpret_cast<const float2*>(sm.K + ((x0 + n) * kB + half * 8 + g) * kLd + col);
            if (m[n]) v = mul2(v, *reinterpret_cast<const float2*>(m[n] + col));
            split3(v.x, v.y, &B[n][0][r], &B[n][1][r], &B[n][2][r]);
          }
        mma6<N>(at, A, B);
      }
#pragma unroll
      for (int n = 0; n < N; ++n) {
        float (*d)[24] = sm.cross[qb * (qb - 1) / 2 + x0 + n];
        *reinterpret_cast<float2*>(&d[g][half * 8 + 2 * t4]) = make_float2(sc[n][0], sc[n][1]);
        *reinterpret_cast<float2*>(&d[g + 8][half * 8 + 2 * t4]) = make_float2(sc[n][2], sc[n][3]);
      }
    };
    if (qb * kB < q) {
      if (b < 2) scores(std::integral_constant<int, 1>());
      else scores(std::integral_constant<int, 2>());
    }
  }
  __syncthreads();
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
    for (int np = 0; np < 4; np += 2) {
      if (np * 16 < ncol) {      // two 16-column tiles at a time; what is past the last column is zero
        uint32_t v[2][4];
        ldsm_x4_trans(v[0], bt_addr(sm.V, kLd, blk * kB, half * 64 + np * 16, lane));
        ldsm_x4_trans(v[1], bt_addr(sm.V, kLd, blk * kB, half * 64 + np * 16 + 16, lane));
#pragma unroll
        for (int k = 2; k >= 0; --k)
#pragma unroll
          for (int n = 0; n < 4; ++n) mma(o[2 * np + n], A[k], v[n >> 1][2 * (n & 1)], v[n >> 1][2 * (n & 1) + 1]);
      }
    }
  };
  if (live) {
#pragma unroll
    for (int x = 0; x < 3; ++x)
      if (x < b) {
        float s[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const float2 v = *reinterpret_cast<const float2*>(&sm.cross[b * (b - 1) / 2 + x][g + 8 * r][nt * 8 + 2 * t4]);
            s[nt][2 * r] = v.x; s[nt][2 * r + 1] = v.y;
          }
        values(s, x);
      }
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
    for (int i0 = 0; i0 < D; i0 += kRows) {
      if (i0 > 0) __syncthreads();       // the last rows are no longer read (nor the keys, since the barrier behind the scores)
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
          for (int np = 0; np < 4; np += 2) {
            if (np * 16 < ncol) {
              uint32_t B[4][3][2];
              float* at[4];
#pragma unroll
              for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                  uint32_t t[4];
                  ldsm_x4_trans(t, bt_addr(Ss + k * kRows * kLd, kLd, kk * 16, half * 64 + (np + n) * 16, lane));
                  B[2 * n][k][0] = t[0]; B[2 * n][k][1] = t[1];
                  B[2 * n + 1][k][0] = t[2]; B[2 * n + 1][k][1] = t[3];
                }
#pragma unroll
              for (int n = 0; n < 4; ++n) at[n] = o[2 * np + n];
              mma6<4>(at, A, B);
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

size_t scan_parallel_ws_floats(int tokens, int seqs, int heads, int dim, int vdim) {
  const size_t chunks = static_cast<size_t>(tokens) / kQ + seqs;
  return chunks * heads * dim * (static_cast<size_t>(vdim) + 2);
}

bool scan_parallel_fits(const GlaArgs& a) {
  auto al = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  return a.par_ws && a.t == DT_BF16 && (a.act == GLA_ACT_NONE || a.act == GLA_ACT_SILU_Q) && !a.rope && !a.head_decay && !a.dt_pre && !a.tok_decay == !a.nstate && a.dim % 16 == 0 && a.dim <= kMaxD &&
         a.vdim % 8 == 0 && a.ld % 8 == 0 && a.q_off % 8 == 0 && a.k_off % 8 == 0 && a.v_off % 8 == 0 && al(a.qkv) && al(a.states) && al(a.o) && al(a.par_ws) && (a.tok_decay || a.fgate_lower || al(a.z)) &&
         scan_parallel_ws_floats(a.T, a.nseq, a.heads, a.dim, a.vdim) <= a.par_ws_floats;
}

int scan_parallel(const GlaArgs& a, cudaStream_t st) {
  if (!scan_parallel_fits(a)) return -1;
  const int chunks = a.T / kQ + a.nseq;
  const size_t rows = static_cast<size_t>(chunks) * a.heads * a.dim;
  Work w;
  w.s = a.par_ws;
  w.d = w.s + rows * a.vdim;
  w.n = w.d + rows;
  if (a.tok_decay) return run<SCALAR, true>(a, w, chunks, st);
  if (a.fgate_lower) return run<VEC_FGATE, false>(a, w, chunks, st);
  if (a.T > 0) log_decay_kernel<<<dim3(a.T, (a.heads * a.dim / 4 + 255) / 256), 256, 0, st>>>(a.z, a.z_bias, a.heads * a.dim, a.inv_tau);
  return run<VEC_Z, false>(a, w, chunks, st);
}

}  // namespace b200
