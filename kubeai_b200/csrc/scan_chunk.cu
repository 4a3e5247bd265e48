// The chunked form of the scalar-decay scan (mixers.h GlaArgs, dt_pre) for steps of prompt portions, on the tensor cores.
//
// With a_t = dt_rate d_t (the log decay of token t), c_t = a_1 + ... + a_t inside a chunk of 64 tokens and S the state in
// front of it, the recurrence S <- exp(a_t) S + d_t B_t x_t^T, y_t = S^T C_t unrolls to
//
//   y_t = exp(c_t) S^T C_t + sum_{j <= t} (B_j . C_t) exp(c_t - c_j) d_j x_j,
//   S'  = exp(c_last) S + sum_j exp(c_last - c_j) d_j B_j x_j^T,
//
// four matrix products per chunk.  Every exponent is at most 0 (no factor is ever the inverse of a decay), all sums and the
// state are fp32, and the products keep fp32 precision: B, C and x are bf16 as the convolution left them, so only the other
// operand (state, weighted scores, weighted x) needs more than one bf16 term, and it is split into three, 24 bits
// (mma_frag.cuh).  The result differs from the token-by-token scan by fp32 rounding alone.
//
// Few long sequences leave most of the device to a chain of chunks on few CTAs.  They are cut into segments of kSegment
// tokens: the sums of all segments at once (PART_SUMS), a pass that turns them into incoming states, the outputs of all segments at
// once (PART_OUT).  64 heads of 128 x 64, 3 sequences of 455, 1365 and 2275 tokens: one chain each (PART_ALL) 330 us, segments 214.
// The sums cost a third of the products again, so sequences whose chains fill the device stay whole (rules::segments_pay).
//
// One CTA owns 64 value columns of a (head, sequence or segment) and walks its chunks: 4 warps, each with 16 value columns.  The state
// lives transposed (value columns x state rows) in the warps' accumulators, which are the left operand of the next chunk's
// y without leaving the registers; the scores C B^T are computed 16 tokens per warp and shared through shared memory.
//
// What bounds it: two to four warps a scheduler (registers, shared memory), which stand behind fixed latencies for half of their time; tensor cores
// (mma.sync) 40 % of the time, issue slots 31 %.  So the terms of a split operand go round over several sums (three products in a row on one sum wait
// for each other), a thread's copies step along one column, and in chains and sums the next chunk's keys, values and gates (a chain's queries, once
// they are read) come in while this one is worked on.  The outputs of a segment, four chunks at most, have three CTAs an SM and one set
// of tiles instead: 145 us against 174 with two and two (the shape above).  Without all that: a chain 455 us, sums 77, outputs 172; now 330, 57, 145.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdlib.h>

#include <algorithm>
#include <atomic>

#include "dispatch_rules.h"
#include "launch.h"
#include "mixers.h"
#include "mma_frag.cuh"
#include "seq_tiles.cuh"

namespace b200 {
namespace {

typedef __nv_bfloat16 bf16;
constexpr int kQ = 64;          // tokens per chunk
constexpr int kCols = 64;       // value columns per CTA
constexpr int kThreads = 128;
constexpr int kLdX = kCols + 8, kLdM = kQ + 8;

__device__ __forceinline__ float softplusf_(float x) { return x > 20.0f ? x : log1pf(expf(x)); }

// per token: c_t, exp(c_t), d_t (0 past the portion), exp(c_last - c_t) d_t
struct Gates {
  float cum[kQ], ecum[kQ], dts[kQ], wts[kQ];
};
enum Part { PART_ALL = 0, PART_SUMS, PART_OUT };
__host__ __device__ constexpr int buffers_for(int part) { return part == PART_OUT ? 1 : 2; }       // of keys, values and gates
size_t chunk_smem(int N, int part) {
  const size_t nb = buffers_for(part), qk = part == PART_SUMS ? nb : nb + 1, scores = part == PART_SUMS ? 0 : 3ull * kQ * kLdM * 2;
  return qk * kQ * (N + 8) * 2 + nb * kQ * kLdX * 2 + scores + nb * sizeof(Gates);
}

constexpr int kSegment = 256;
// of every segment and head: its sums [dim][vdim], then the state in front of it; the decay over it
struct Segments {
  float *s, *d;
};

// CTAs an SM is to hold: what shared memory allows with the registers that leaves.  Up to 32 state rows segments live on them: 64 heads of 64 x 16, one sequence of 2000
// tokens, 71 us with four and three of them, 56 so; 64 x 32 76 and 60.
__host__ __device__ constexpr int ctas_per_sm(int nk, int part) {
  return part == PART_SUMS ? (nk == 2 ? 6 : 4) : part == PART_OUT ? (nk == 2 ? 4 : 3) : nk == 2 ? 3 : 2;
}

// NK: state rows in units of 16, at most (N = a.dim is any multiple of 16 up to 16 NK)
template <int NK, int PART>
__global__ void __launch_bounds__(kThreads, ctas_per_sm(NK, PART)) scalar_decay_chunk_kernel(GlaArgs a, Segments sg) {
  using namespace frag;
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int NB = buffers_for(PART);
  const int N = a.dim, P = a.vdim, nk = N / 16, LDN = N + 8;
  bf16* Bbuf = reinterpret_cast<bf16*>(smraw);   // [NB][kQ][LDN] keys
  bf16* Xbuf = Bbuf + NB * kQ * LDN;             // [NB][kQ][kLdX] values of the CTA's columns
  Gates* gates = reinterpret_cast<Gates*>(Xbuf + NB * kQ * kLdX);   // [NB]
  bf16* Cs = reinterpret_cast<bf16*>(gates + NB);   // [kQ][LDN] queries
  bf16* Ms = Cs + kQ * LDN;                      // [3][kQ (t)][kLdM (j)] weighted scores, three bf16 terms
  const int head = blockIdx.y, p0 = (PART == PART_ALL ? blockIdx.x : blockIdx.z) * kCols;
  int seq = blockIdx.z, segment = 0;
  if (PART != PART_ALL && !find_tile(a.seqs, a.nseq, kSegment, blockIdx.x, &seq, &segment)) return;
  const int tok0 = a.seqs[seq * 8 + 0] + segment * kSegment, pos0 = a.seqs[seq * 8 + 2] + segment * kSegment, slot = a.seqs[seq * 8 + 3];
  const int n = PART == PART_ALL ? a.seqs[seq * 8 + 1] : min(kSegment, a.seqs[seq * 8 + 1] - segment * kSegment);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const bf16* base = static_cast<const bf16*>(a.qkv);
  const int qk0 = (head / a.group) * N;
  const bool live = p0 + 16 * w < P;             // warps past the last value column only help with the scores
  float* Sg = PART == PART_ALL ? a.states + (static_cast<long long>(slot) * a.heads + head) * N * P
                               : sg.s + (static_cast<long long>(blockIdx.x) * a.heads + head) * N * P;
  float total = 0.f;                             // log decay over the segment
  const int pr[2] = {p0 + 16 * w + g, p0 + 16 * w + g + 8};
  float S[NK][2][4];                             // [16 state rows][half][c]: value column pr[c / 2], state row 16 k + 8 half + 2 t4 + c % 2
#pragma unroll
  for (int k = 0; k < NK; ++k)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int nn = 16 * k + 8 * h + 2 * t4 + (c & 1), p = pr[c >> 1];
        S[k][h][c] = (PART != PART_SUMS && k < nk && p < P && pos0 > 0) ? Sg[static_cast<long long>(nn) * P + p] : 0.f;
      }
  const float rate = a.dt_rate[head], dbias = a.dt_bias[head];

  // a chunk's rows of one column block (keys or queries), 16 bytes a thread and step; rows past the portion become zeros
  auto fetch_rows = [&](bf16* dst, int off, int c0) {
    constexpr int kPieces = 2 * NK, kRows = kThreads / kPieces;    // of a row (those past N idle); rows at a time
    const int t0 = tid / kPieces, c = (tid % kPieces) * 8;
    if (c >= N) return;
    const bf16* src = base + static_cast<long long>(tok0 + c0 + t0) * a.ld + off + qk0 + c;
    bf16* d = dst + t0 * LDN + c;
#pragma unroll
    for (int t = 0; t < kQ; t += kRows, src += static_cast<long long>(kRows) * a.ld, d += kRows * LDN) {
      if (c0 + t0 + t < n) cp_async16(smem_addr(d), src);
      else *reinterpret_cast<uint4*>(d) = make_uint4(0, 0, 0, 0);
    }
  };
  auto fetch_values = [&](bf16* dst, int c0) {
    constexpr int kPieces = kCols / 8, kRows = kThreads / kPieces;
    const int t0 = tid / kPieces, c = (tid % kPieces) * 8;
    const bf16* src = base + static_cast<long long>(tok0 + c0 + t0) * a.ld + a.v_off + head * P + p0 + c;
    bf16* d = dst + t0 * kLdX + c;
#pragma unroll
    for (int t = 0; t < kQ; t += kRows, src += static_cast<long long>(kRows) * a.ld, d += kRows * kLdX) {
      if (c0 + t0 + t < n && p0 + c < P) cp_async16(smem_addr(d), src);
      else *reinterpret_cast<uint4*>(d) = make_uint4(0, 0, 0, 0);
    }
  };
  // step sizes and running log decays of a chunk, by one warp: lane l owns tokens 2l and 2l + 1
  auto make_gates = [&](Gates& G, int c0) {
    float d[2], s[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = 2 * lane + i;
      d[i] = c0 + t < n ? softplusf_(__bfloat162float(static_cast<const bf16*>(a.dt_pre)[static_cast<long long>(tok0 + c0 + t) * a.ld_dt + head]) + dbias) : 0.f;
      s[i] = rate * d[i];
    }
    float run = s[0] + s[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float v = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += v;
    }
    const float last = __shfl_sync(0xffffffffu, run, 31);
    total += last;
    const float before = __shfl_up_sync(0xffffffffu, run, 1);
    const float cc[2] = {(lane ? before : 0.f) + s[0], run};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = 2 * lane + i;
      G.cum[t] = cc[i];
      G.ecum[t] = expf(cc[i]);
      G.dts[t] = d[i];
      G.wts[t] = expf(last - cc[i]) * d[i];
    }
  };
  auto fetch_all = [&](int c0) {
    fetch_rows(Bbuf, a.k_off, c0);
    if (PART != PART_SUMS) fetch_rows(Cs, a.q_off, c0);
    fetch_values(Xbuf, c0);
    if (w == 0) make_gates(gates[0], c0);
  };
  if (NB == 2) fetch_all(0);

  for (int c0 = 0, buf = 0; c0 < n; c0 += kQ, buf ^= NB - 1) {
    const int q = min(kQ, n - c0);
    const bool more = NB == 2 && c0 + kQ < n;
    if (NB == 1) {
      __syncthreads();   // the last chunk's tiles are no longer read
      fetch_all(c0);
    }
    const bf16 *Bs = Bbuf + buf * kQ * LDN, *Xs = Xbuf + buf * kQ * kLdX;
    const Gates& G = gates[buf];
    cp_async_wait_all();
    __syncthreads();     // this chunk's tiles and gates are in place; nobody works on the last chunk any more
    if (more) {
      fetch_rows(Bbuf + (buf ^ 1) * kQ * LDN, a.k_off, c0 + kQ);
      fetch_values(Xbuf + (buf ^ 1) * kQ * kLdX, c0 + kQ);
    }

    // ---- weighted scores: this warp's 16 tokens t against the keys of its own and earlier blocks
    if (PART != PART_SUMS) {
      float D[4][2][4];
#pragma unroll
      for (int jb = 0; jb < 4; ++jb)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int c = 0; c < 4; ++c) D[jb][h][c] = 0.f;
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        if (k < nk) {
          uint32_t af[4];
          ldsm_x4(af, a_addr(Cs, LDN, 16 * w, 16 * k, lane));
#pragma unroll
          for (int jb = 0; jb < 4; ++jb) {
            if (jb <= w) {
              uint32_t bf_[4];
              ldsm_x4(bf_, b_addr(Bs, LDN, 16 * jb, 16 * k, lane));
              mma(D[jb][0], af, bf_[0], bf_[1]);
              mma(D[jb][1], af, bf_[2], bf_[3]);
            }
          }
        }
      }
      const float ct[2] = {G.cum[16 * w + g], G.cum[16 * w + g + 8]};
#pragma unroll
      for (int jb = 0; jb < 4; ++jb) {
        if (jb <= w) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int j = 16 * jb + 8 * h + 2 * t4;
            const float2 cj = *reinterpret_cast<const float2*>(G.cum + j), dj = *reinterpret_cast<const float2*>(G.dts + j);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              const int t = 16 * w + g + 8 * hf;
              uint32_t x[3];
              split3(j <= t ? D[jb][h][2 * hf] * (expf(ct[hf] - cj.x) * dj.x) : 0.f, j + 1 <= t ? D[jb][h][2 * hf + 1] * (expf(ct[hf] - cj.y) * dj.y) : 0.f,
                     &x[0], &x[1], &x[2]);
#pragma unroll
              for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(Ms + (s * kQ + t) * kLdM + j) = x[s];
            }
          }
        }
      }
      if (w == 0 && more) make_gates(gates[buf ^ 1], c0 + kQ);
      __syncthreads();
    } else if (w == 0 && more) {
      make_gates(gates[buf ^ 1], c0 + kQ);
    }

    float Y[4][2][4];
    if (live) {
      // ---- y^T [16 value columns x 64 tokens]: the state's part, scaled per token, then the chunk's own
#pragma unroll
      for (int tb = 0; tb < 4; ++tb)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int c = 0; c < 4; ++c) Y[tb][h][c] = 0.f;
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        if (PART != PART_SUMS && k < nk) {
          uint32_t st[3][4];
#pragma unroll
          for (int r = 0; r < 4; ++r) split3(S[k][r >> 1][2 * (r & 1)], S[k][r >> 1][2 * (r & 1) + 1], &st[0][r], &st[1][r], &st[2][r]);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t b[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i) ldsm_x4(b[i], b_addr(Cs, LDN, 32 * half + 16 * i, 16 * k, lane));
#pragma unroll
            for (int term = 2; term >= 0; --term)
#pragma unroll
              for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) mma(Y[2 * half + i][h], st[term], b[i][2 * h], b[i][2 * h + 1]);
          }
        }
      }
#pragma unroll
      for (int tb = 0; tb < 4; ++tb)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 e = *reinterpret_cast<const float2*>(G.ecum + 16 * tb + 8 * h + 2 * t4);
          Y[tb][h][0] *= e.x; Y[tb][h][1] *= e.y; Y[tb][h][2] *= e.x; Y[tb][h][3] *= e.y;
        }
      const float decay = G.ecum[kQ - 1];
#pragma unroll
      for (int k = 0; k < NK; ++k)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int c = 0; c < 4; ++c) S[k][h][c] *= decay;
    }
    if (PART != PART_SUMS && more) {
      __syncthreads();   // the queries are no longer read
      fetch_rows(Cs, a.q_off, c0 + kQ);
    }
    if (live) {
#pragma unroll
      for (int jb = 0; jb < 4; ++jb) {
        if (16 * jb >= q) break;       // no tokens there
        uint32_t xf[4];
        ldsm_x4_trans(xf, at_addr(Xs, kLdX, 16 * jb, 16 * w, lane));
        if (PART != PART_SUMS) {
#pragma unroll
          for (int s = 2; s >= 0; --s) {
#pragma unroll
            for (int tb = jb; tb < 4; ++tb) {
              uint32_t b[4];
              ldsm_x4(b, b_addr(Ms + s * kQ * kLdM, kLdM, 16 * tb, 16 * jb, lane));
              mma(Y[tb][0], xf, b[0], b[1]);
              mma(Y[tb][1], xf, b[2], b[3]);
            }
          }
        }
        if (PART == PART_OUT && c0 + kQ >= n) continue;   // nobody asks for the state behind the last chunk
        // the state takes exp(c_last - c_j) d_j x_j B_j^T
        const float2 wl = *reinterpret_cast<const float2*>(G.wts + 16 * jb + 2 * t4), wh = *reinterpret_cast<const float2*>(G.wts + 16 * jb + 8 + 2 * t4);
        uint32_t x[3][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) split3(low(xf[r]) * (r < 2 ? wl.x : wh.x), high(xf[r]) * (r < 2 ? wl.y : wh.y), &x[0][r], &x[1][r], &x[2][r]);
#pragma unroll
        for (int k = 0; k < NK; k += 2) {
          if (k < nk) {
            uint32_t b[2][4];
            ldsm_x4_trans(b[0], bt_addr(Bs, LDN, 16 * jb, 16 * k, lane));
            if (k + 1 < nk) ldsm_x4_trans(b[1], bt_addr(Bs, LDN, 16 * jb, 16 * (k + 1), lane));
#pragma unroll
            for (int term = 2; term >= 0; --term)
#pragma unroll
              for (int i = 0; i < 2; ++i)
                if (k + i < nk) {
                  mma(S[k + i][0], x[term], b[i][0], b[i][1]);
                  mma(S[k + i][1], x[term], b[i][2], b[i][3]);
                }
          }
        }
      }
      if (PART == PART_SUMS) continue;
      const int HP = a.heads * P;
      float* out = a.o + static_cast<long long>(tok0 + c0 + 2 * t4) * HP + head * P + pr[0];
#pragma unroll
      for (int tb = 0; tb < 4; ++tb)
#pragma unroll
        for (int h = 0; h < 2; ++h, out += 8ll * HP)
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (16 * tb + 8 * h + 2 * t4 + (c & 1) < q && pr[c >> 1] < P) out[(c & 1 ? HP : 0) + 8 * (c >> 1)] = Y[tb][h][c];
    }
  }
  if (PART == PART_SUMS && p0 == 0 && tid == 0) sg.d[static_cast<long long>(blockIdx.x) * a.heads + head] = expf(total);
  if (PART == PART_OUT) return;
#pragma unroll
  for (int k = 0; k < NK; ++k)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int nn = 16 * k + 8 * h + 2 * t4 + (c & 1), p = pr[c >> 1];
        if (k < nk && p < P) Sg[static_cast<long long>(nn) * P + p] = S[k][h][c];
      }
}

// grid (four state entries a thread, heads, sequences): each segment's sums replaced by the state in front of it, S <- d S + sums
__global__ void __launch_bounds__(256) segment_states_kernel(GlaArgs a, Segments sg) {
  const int seq = blockIdx.z, head = blockIdx.y, NP = a.dim * a.vdim, lane = threadIdx.x & 31;
  int first = 0;
  for (int s0 = 0; s0 < seq; s0 += 32) {
    int c = s0 + lane < seq ? (a.seqs[(s0 + lane) * 8 + 1] + kSegment - 1) / kSegment : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    first += c;
  }
  const int e = (blockIdx.x * 256 + threadIdx.x) * 4, segs = (a.seqs[seq * 8 + 1] + kSegment - 1) / kSegment, slot = a.seqs[seq * 8 + 3];
  if (e >= NP || segs <= 0) return;
  const bool old = a.seqs[seq * 8 + 2] > 0;
  float4* state = reinterpret_cast<float4*>(a.states + (static_cast<long long>(slot) * a.heads + head) * NP + e);
  float4 s = old ? *state : make_float4(0.f, 0.f, 0.f, 0.f);
  constexpr int U = 4;      // segments in flight
  for (int i = 0; i < segs; i += U) {
    float4 t[U];
    float d[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u < segs) {
        const long long r = static_cast<long long>(first + i + u) * a.heads + head;
        t[u] = *reinterpret_cast<const float4*>(sg.s + r * NP + e);
        d[u] = sg.d[r];
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u < segs) {
        *reinterpret_cast<float4*>(sg.s + (static_cast<long long>(first + i + u) * a.heads + head) * NP + e) = s;
        s = make_float4(fmaf(d[u], s.x, t[u].x), fmaf(d[u], s.y, t[u].y), fmaf(d[u], s.z, t[u].z), fmaf(d[u], s.w, t[u].w));
      }
  }
  *state = s;
}

template <int NK, int PART>
int launch_part(const GlaArgs& a, const Segments& sg, dim3 grid, cudaStream_t st) {
  static std::atomic<unsigned long long> attr{0};
  if (!ensure_dynamic_smem(scalar_decay_chunk_kernel<NK, PART>, static_cast<int>(chunk_smem(16 * NK, PART)), &attr)) return -2;
  scalar_decay_chunk_kernel<NK, PART><<<grid, kThreads, chunk_smem(a.dim, PART), st>>>(a, sg);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
// Segments where they are the shorter way (slots: CTAs of the chain that run at once), and their workspace is there.
bool cut_into_segments(const GlaArgs& a, int slots) {
  const char* e = getenv("B200_SCAN_SEGMENTS");      // A/B knob: 0 = never, 1 = wherever they fit
  const int force = e ? atoi(e) : -1;
  if (force == 0 || !a.par_ws || scan_segments_ws_floats(a.T, a.nseq, a.heads, a.dim, a.vdim) > a.par_ws_floats || a.vdim % 4 ||
      (reinterpret_cast<uintptr_t>(a.par_ws) | reinterpret_cast<uintptr_t>(a.states)) % 16) return false;
  return force == 1 || rules::segments_pay(a.T, a.nseq, a.max_rows, a.heads, (a.vdim + kCols - 1) / kCols, slots, sm_count());
}
template <int NK>
int launch(const GlaArgs& a, cudaStream_t st) {
  const int cb = (a.vdim + kCols - 1) / kCols;
  Segments sg = {nullptr, nullptr};
  static std::atomic<unsigned long long> attr{0};
  int per_sm = 0;
  if (!ensure_dynamic_smem(scalar_decay_chunk_kernel<NK, PART_ALL>, static_cast<int>(chunk_smem(16 * NK, PART_ALL)), &attr) ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, scalar_decay_chunk_kernel<NK, PART_ALL>, kThreads, chunk_smem(a.dim, PART_ALL)) != cudaSuccess) return -2;
  if (!cut_into_segments(a, std::max(1, per_sm) * sm_count())) return launch_part<NK, PART_ALL>(a, sg, dim3(cb, a.heads, a.nseq), st);
  const int segs = a.T / kSegment + a.nseq;
  sg.s = a.par_ws;
  sg.d = sg.s + static_cast<size_t>(segs) * a.heads * a.dim * a.vdim;
  if (const int rc = launch_part<NK, PART_SUMS>(a, sg, dim3(segs, a.heads, cb), st)) return rc;
  segment_states_kernel<<<dim3((a.dim * a.vdim / 4 + 255) / 256, a.heads, a.nseq), 256, 0, st>>>(a, sg);
  return launch_part<NK, PART_OUT>(a, sg, dim3(segs, a.heads, cb), st);
}

}  // namespace

size_t scan_segments_ws_floats(int tokens, int seqs, int heads, int dim, int vdim) {
  return (static_cast<size_t>(tokens) / kSegment + seqs) * heads * (static_cast<size_t>(dim) * vdim + 1);
}

bool scan_chunk_fits(const GlaArgs& a) {
  auto al = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  return a.dt_pre && a.t == DT_BF16 && a.act == GLA_ACT_NONE && !a.rope && a.q_scale == 1.f && a.k_scale == 1.f && a.dim % 16 == 0 && a.dim <= 128 &&
         a.vdim % 8 == 0 && a.ld % 8 == 0 && a.q_off % 8 == 0 && a.k_off % 8 == 0 && a.v_off % 8 == 0 && al(a.qkv);
}

int scan_chunk(const GlaArgs& a, cudaStream_t st) {
  if (!scan_chunk_fits(a)) return -1;
  if (a.dim <= 32) return launch<2>(a, st);
  return a.dim <= 64 ? launch<4>(a, st) : launch<8>(a, st);
}

}  // namespace b200
