// Rules that choose between two kernels with the same result by the sizes of a call alone, as plain host functions: the kernels'
// launchers use them, and b200_rule_query answers from them without a GPU.
#pragma once
#include <math.h>

namespace b200 {
namespace rules {

// Rows that pick their own matrix (linear.cu, linear_picked_rows_kernel): behind its predecessor instead of overlapping it.  The products
// around it hold some 200 KB of shared memory an SM, and an SM that never runs empty keeps that split of its memory: the stream of
// weights then runs with 28 KB of L1 instead of about 200.  What that costs grows with the stream, the launch's gap does not.
// us a decode step of 4 layers, overlapped / behind: 2 pairs of 17 MB 304 / 310, 16 of them 508 / 475; 32 of 67 MB 3028 / 2478,
// 64 of 67 MB 5335 / 4222 (4980 before those products held so much); 16 pairs of 8 MB 359 / 367, 24 of 8 MB 425 / 422.
inline bool picked_rows_alone(long long rows, long long N, long long K, int bytes) { return rows * N * K * bytes > 160000000; }

// Attention of single tokens (window_attention.cu): sixteen lanes a key (window_attn_rows_kernel), or a lane a key
// (window_attn_kernel).  The sixteen have one key in flight for the whole group of heads, but repeat its exponential (and the
// cap's tanh) on every lane, use width / 8 of their loads and merge sixteen partial results however few keys there are.
// units: tokens times query heads; width: the larger of the head's two dimensions; keys: the most any token sees.
// Up to 1024 units the other kernel spreads a token's keys over 16 warps, and what counts is the length of a chain.  us a launch,
// sixteen lanes / one: 128 wide, 1 token: 16 keys 11 / 19, 16000 302 / 375; 72 wide 4000 keys 114 / 117, 8000 154 / 147; 64 wide 600 keys
// 20 / 22, 2000 49 / 40, 8000 156 / 115; 32 wide 30 keys 12 / 16, 250 15.6 / 14.0; 8 wide 30 keys 11 / 14, 300 15.7 / 14.9, 16000 294 / 124; with
// a cap 96 wide 1000 keys 0.9 of the other, 2000 1.12 of it.
// Beyond, what counts is instructions a key.  128 wide, up to 10 keys: 100 tokens of 16 heads 24 / 26, 64 of 32 heads 29 / 27, 100 of them 39 / 36
// (with keys kept in front of the window 43 / 36); 112 tokens of up to 40 keys, 32 heads 46 / 52; 128 x 250 keys 51 / 100; 72 wide 128 x 20 30 / 28, 128 x 250
// 62 / 72; 64 wide 640 tokens of 250 253 / 245; 32 wide 257 / 214; with a cap, 128 wide: up to 10 keys 58 / 36, 40 63 / 52, 100 0.89 of the
// other, 250 64 / 108; 96 wide 0.96 to 1.14 of it from 250 keys on.
inline bool sixteen_lanes_a_key(long long units, int width, long long keys, bool cap) {
  if (units <= 1024) return width >= 120 || keys <= (width > 64 ? (cap ? 1024 : 4096) : width > 32 ? 512 : 128);
  if (width >= 120) return cap ? keys >= 96 : units < 2048 || keys >= 16;
  return width > 64 && !cap && keys >= 64;
}

// Products of few rows that have a whole-tile form too: where the passes over the weights (linear_stream.cu) and the clusters
// (linear_cluster.cu) are still ahead of it.  Both read all of X in every CTA, T * K values through each SM's port, and a long K makes
// that the larger part.  Ratio of their time to the whole tiles', weights from HBM; N rows of W, passes:
//   K 4096   40 tokens, N 1024 .. 4736 0.67 .. 0.82     K 8192   N 64 .. 4736 0.82 .. 1.0      K 14336  N 64 .. 3168 1.06 .. 1.18, 4096 0.95
//   K 14336  32 tokens, N 64 .. 3168 0.77 .. 0.93       K 28672  N 64 .. 1536 1.06 .. 1.20, 2048 0.95     16 tokens, N 64 .. 3168 0.80 .. 1.0
// In a design's step (ff_down, us, whole tiles / here): 1024 x 28672 40 tokens 33 / 51, 200 tokens 57 / 71; 2048 x 14336 24 tokens 29 / 20, 100 tokens 35 / 32.
//   pairs of rows (against the kernel of a decode step's pairs), 7168 x 16384: 24 tokens 46.4 / 49.9 us, 32 tokens 53.0 / 50.0
// Llama-3-8B's down projection (4096 x 14336) and the norm behind it, 33 to 48 tokens: a step of 4 layers 530 .. 537 us, fused 580 .. 584.
inline bool stream_pays(int T, int N, int K, bool pairs) {
  if (K <= 8192) return true;
  if (pairs) return T <= 24;
  return T <= 16 || (T <= 32 ? K <= 16384 || N >= 2048 : N >= 4096);
}
// clusters, 49 .. 256 tokens, over tiles as large as can be.  tiles_ahead below leaves them less than these lines do, which so decide only for outputs that are no
// whole 16-byte pieces:
//   K 4096   N 1024 .. 2112 0.67 .. 0.83, 2560 .. 3168 0.77 .. 0.91     K 8192   0.73 .. 0.93, 0.93 .. 1.08
//   K 14336  0.83 .. 1.08 (to 128 tokens), 1.0 .. 1.12 (129 on); 1.08 .. 1.19     K 28672  1.12 .. 1.52, 1.28 .. 1.42
inline bool cluster_pays(int T, int N, int K) { return K <= (N > 2112 ? 6144 : T <= 128 ? 16384 : 10240); }

// Both of them against tiles whose rows are chosen for the call (whole_tiles below), where there is a plan for those.  us a launch, weights from
// memory, few rows / tiles:
//   passes    T 40: 2048 x 4096 9.8 / 11.7, 1024 x 8192 15.3 / 12.6, 3168 x 8192 17.4 / 17.4, 4096 x 8192 18.2 / 20.2, 2048 x 14336 24.3 / 18.6, 4096 x 14336 28.1 / 28.6
//             T 32: 1024 x 8192 11.3 / 12.7, 2048 x 8192 12.1 / 14.1, 1024 x 14336 17.4 / 14.9, 2048 x 14336 17.9 / 18.2, 3168 x 14336 21.8 / 23.5
//   clusters  T 64: 2048 x 2048 8.0 / 9.5, 2048 x 4096 11.1 / 12.1, 2048 x 8192 15.6 / 14.8, 1024 x 14336 21.0 / 15.7, 3072 x 1024 8.0 / 7.5, 3072 x 4096 13.1 / 13.3
//             T 128: 2048 x 2048 9.1 / 9.6, 2048 x 512 6.8 / 6.4, 3072 x 2048 11.1 / 9.8      T 129 .. 256: 1024 x 2048 9.5 .. 11.2 / 9.6, 2048 x 8192 20.8 .. 24.3 / 16.7 .. 19.2
inline bool tiles_ahead(int T, int N, int K) {
  if (T <= 32) return T > 24 && K > 12288 && N <= 2112;
  if (T <= 48) return K > 6144 && N < (K > 12288 ? 4096 : 3168);
  return T > 128 || K > 6144 || N > 2112;
}

// Mamba-2 prompts (scan_chunk.cu): sequences cut into segments of 256 tokens, or one chain of 64-token chunks each.  Times in chunks
// of a chain's CTA with a second one on its SM (9.2 us at 128 state rows, 6.5 at 64, 5.1 at 32; alone on its SM 0.83 of that).  A chain takes its
// longest sequence, and where not all CTAs (heads, column blocks) run at once as many rounds of equal ones, or the sum of unequal ones and a part of the
// longest, which comes last at worst; the segments' three launches take about 4 and then 4.6 for every time that all of them fill the device twice over,
// with any number of state rows.  us, segments / chains, 64 columns, 128 state rows:
//   8 heads   1 x 4096 67 / 481    6 x 682 71 / 90         64 heads   1 x 512 71 / 70    1 x 4096 202 / 485    3 x 1365 216 / 206
//   32 heads  4 x 512 87 / 70      6 x 682 126 / 109                  4 x 512 128 / 84   4 x 1024 208 / 155    6 x 682 214 / 195
//   128 heads 1 x 1024 124 / 131   2 x 512 128 / 84        256 heads  1 x 512 128 / 84   1 x 4096 744 / 586    3 x 1365 800 / 614
//   unequal: 64 heads 455 + 1365 + 2275 214 / 330; 128 heads 300 + 700 + 1100 + 2000 407 / 392; 256 heads 300 + 2000 456 / 347
// 64 state rows: 64 heads 1 x 4096 146 / 338, 4 x 1024 144 / 111, 128 heads 2 x 2048 253 / 211; 32: 64 heads 1 x 4096 118 / 268, 4 x 1024 120 / 88.
// longest 0: not known, all taken as equal.  From seven sequences on, or with a mean below 512, chains.
inline bool segments_pay(long long T, int nseq, int longest, int heads, int blocks, int slots, int sms) {
  if (nseq < 1 || nseq > 6 || T < 512LL * nseq) return false;
  const double mean = T / 64.0 / nseq, most = ceil(longest > 0 ? longest / 64.0 : mean), per_slot = static_cast<double>(heads) * blocks / slots, rounds = ceil(nseq * per_slot);
  const double chain = rounds <= 1 ? (nseq * heads * blocks <= sms ? 0.83 : 1.0) * most : most <= 1.1 * mean + 1 ? rounds * most : fmax(most, T / 64.0 * per_slot + 0.7 * fmax(0.0, 1.0 - per_slot) * most);
  return 4.1 + 4.6 * (T / 256.0 + nseq / 2.0) * heads * blocks / (2.0 * sms) < chain;
}

// Chunks of the delta rule (delta_chunk.cu): four more warps a CTA form the next chunk's scores, one CTA an SM, or two CTAs of four warps share an SM.  A
// chain gains what waits left of its SM's tensor pipe; where the SMs' work outlasts the longest chain, two CTAs hide each other's waits as well and without the
// rest.  us, by itself / ahead, 128 x 128 (CTAs a sequence: twice the heads): 16 heads, 63 to 959 tokens in 8 sequences (work 14.7 chunks an SM, longest 15)
// 229 / 162, 4 x 1000 and 500 (15.7, 16) 238 / 172, 5 x 777 (13.7, 13) 217 / 244, 8 x 200 (6.3, 4) 82 / 98; 32 heads, the 8 sequences (29.4, 15) 256 / 305,
// 100 to 2000 in six (20, 32) 440 / 307; 2 x 1000: 4 heads 213 / 148, 37 (148 CTAs) 223 / 172, 40 (17.4, 16) 264 / 299, 74 (32, 16) 283 / 330.  64 and 32 rows
// the same.  Sequences of one chunk have nothing ahead (40 of 17 tokens, 4 heads of 128 x 64 27 / 40).  longest 0: not known.
inline bool delta_scores_ahead(int ctas, int nseq, int tokens, int longest, int sms) {
  return (longest > 0 ? longest : tokens) > 64 && (static_cast<long long>(ctas) * nseq <= sms || (tokens / 64.0 + nseq / 2.0) * ctas / sms <= (longest + 63) / 64);
}

// Norms between sublayers (hyper.cu): a row of 256 threads times `pieces` of four columns in registers through both sums, or read from
// memory again behind each.  Three and four pieces leave an SM two rows at a time: ahead while that holds all rows there are (steps), behind
// where many follow.  us of 9 launches, again / registers, 4096 wide: 1 row 55 / 42, 148 rows 51 / 41, 444 52 / 52, 900 69 / 74, 4000 196 / 232;
// 2560 wide: 148 48 / 39, 444 49 / 50, 600 51 / 58, 4000 144 / 183.  More than four would spill.
inline bool row_in_registers(int pieces, int rows, int sms) { return pieces <= 2 || (pieces <= 4 && rows <= 3 * sms); }

// Products per head of 17 to 128 rows (linear.cu): blocks of 16 rows that read the weights from L2 again, or tiles of 64 rows that walk K in
// a chain.  What the blocks cost is those bytes, what the tiles cost is K.  us, tiles / blocks: 128 x 512 (rows of W 512, bf16 rows of X)
// 16 heads 64 rows 12.1 / 11.1, 128 rows 12.7 / 14.5; 32 heads 32 rows 12.5 / 12.6, 100 rows 14.9 / 18.8; 64 heads 128 rows 23.9 / 31.2; K 64,
// 32 heads 100 rows 10.0 / 13.1, 64 heads 48 rows 9.7 / 10.9, 128 rows 13.7 / 17.4.  Rows of X in fp32, K 512 to 128 columns: 16 heads 21 / 11, 64 heads 64 rows 23.5 / 17.2, 100 rows
// 25.1 / 24.7, 128 rows 25.5 / 27.6; K 256, 64 heads 128 rows 15.3 / 13.0.
inline bool row_blocks_pay(int rows, long long batch, long long N, long long K, bool fp32_rows) {
  return (rows + 15) / 16 * batch * N * K * 2 <= (fp32_rows ? 60000000 : K >= 128 ? 8500000 : 3000000);
}

// Single tokens of the recurrences (gla.cu, delta.cu): a pass over the states, CTAs of 64 value columns and up to 16, 128 or 256 rows a lane
// group, or the scan that walks tokens, a column a thread.  The pass idles where a state fills little of that.  Ratio of its time to the
// scan's, 16 heads, 32 or 128 sequences: GLA, mLSTM, HGRN2, Mamba-2 0.42 .. 1.0 up to 128 rows and from 32 columns on, 256 rows of 4 to 16
// columns 0.82 .. 1.11; delta rule 64 rows 0.74 .. 0.99, 128 and 256 rows of 32 to 256 columns 0.40 .. 1.0, of 4 to 16 columns 0.92 .. 1.22; 4 to 32
// rows of 4 to 64 columns 0.74 .. 0.95, of 96 to 256 columns 0.99 .. 1.40.  4 sequences: 0.5 .. 1.0 everywhere.
inline bool single_step_pays(long long heads_times_sequences, int dim, int vdim, bool delta, int sms) {
  if (heads_times_sequences * ((vdim + 63) / 64) <= sms) return true;
  if (!delta) return dim <= 128 || vdim >= 32;
  return dim > 64 ? vdim >= 32 : dim > 32 || vdim <= 64;
}

// Whole tiles (gemm_grouped.cu): the rows of a tile of 256 rows of W, and the parts its K is cut into, for `rows` rows of X on `pairs` CTA pairs.
// A 64-wide step of K takes a pair 0.036 + 0.00105 us a row of the tile, at least 0.16 (what a step costs besides its products), a tile
// 1.2 us besides, the weights what they take from memory; the exchange between parts 3 + rows * (0.016 + 0.009 parts) us.  So the tiles are as
// large as they can be with as few rows to work through as there are: rows of the tile times tiles of the busiest pair.  (All tiles had up to
// 256 rows while a step took 0.3 us whatever they had.)  us a launch, weights from memory, tiles as large as can be / these; over N 1024 to 28672, K 2048 to
// 14336 and 129 to 3000 rows 0.84 of the time, and within 2.5 % of the best of all tiles and parts in the mean:
//   2048 x 2048   256 rows 16.2 / 10.5   1000 rows 17.0 / 12.1   3000 rows 27.0 / 22.0 (176)    2048 x 8192   512 31.8 / 23.6   3000 97.9 / 74.0
//   4096 x 14336  256 rows 60.6 / 44.8   700 rows 77.1 / 63.2    2048 rows 190 / 178 (240)      6144 x 4096  1000 49.0 / 38.6   2048 83.7 / 78.4
//   28672 x 4096  512 rows 123 / 109     1400 rows 271 / 259     8192 x 2048  700 rows 26.3 / 22.5, 1400 rows 35.9 / 37.3
// split: whether K may be cut at all.  (Many rows never want the smallest tiles, which are not tried then.)  Of choices within 2 % the fewest tiles, which read the
// weights less often (fewest / best by the count of steps alone, us: 700 rows 11008 x 8192 92.0 / 101.3, 11008 x 14336 160 / 178, 19456 x 2048 44.5 / 49.7; 1000 rows
// 19456 x 14336 401 / 432; 22016 x 2048 52.3 / 50.4); short K and up to 320 rows gain nothing (14336 x 1024, 600 rows 19.5 / 18.1; 28672 x 14336, 300 rows 278 / 240).
inline void whole_tiles(int rows, int N, int K, int pairs, bool split, int* tile, int* parts) {
  const int KB = (K + 63) / 64, slabs = (N + 255) / 256;
  const double memory = 2.0 * N * K / 6.3e6;
  double best = 0;
  *tile = 0;
  for (int n = (rows + 255) / 256, last = 0; n <= (rows + 31) / 32; ++n) {
    const int t = ((rows + n - 1) / n + 15) & ~15;
    if (t == last) continue;
    if (rows > 1024 && t < 96) break;
    last = t;
    const long long tiles = static_cast<long long>(slabs) * ((rows + t - 1) / t);
    const double step = fmax(0.16, 0.036 + 0.00105 * t);
    const bool fewer = rows > 320 && KB >= 32 && tiles > pairs;
    for (int p = 1; p == 1 || (split && tiles * p <= pairs && p * 8 <= KB); ++p) {
      const long long waves = (tiles * p + pairs - 1) / pairs;
      const double us = fmax(waves * ((KB + p - 1) / p * step + 1.2), memory) + (p > 1 ? 3.0 + t * (0.016 + 0.009 * p) : 0.0);
      if (!*tile || us < best * (fewer ? 0.98 : 1.0) - 1e-9) { best = us; *tile = t; *parts = p; }
    }
  }
}

// Gate and up of up to 128 rows: whole tiles, or gemm3's pairs that share out the tiles' steps of K evenly.  Tiles are ahead by 10 to 30 % (28672 x 4096, 64 rows
// 44.2 us in pairs / 41.7, 14336 x 4096 27.4 / 24.0) unless a few of them are left for a second round: those stream their K on few SMs, at 0.16 us a step, under
// which the memory idles.  Tiles' time over the pairs', 74 pairs, 64 rows: 19456 x 8192 (76 tiles, 66.1 us over 61.2) 1.08, x 5120 1.07, x 3072 1.03, x 2048 0.82; 20480 x 5120
// (80) 1.04; 22016 x 8192 (86) 1.06, x 5120 0.99, x 4096 0.95; 24576 x 8192 (96) 0.98; from the second full round on tiles again (38912 x 8192, 152 tiles, 0.96).
inline bool gate_up_tiles(int N, int K, int pairs) {
  const int left = (N + 255) / 256 - pairs;
  return left <= 0 || left >= pairs || (K + 63) / 64 * 0.16 + 1.2 - left * 512.0 * K / 6.3e6 <= 8.0;
}

// Llama steps of 9 to 128 tokens (engine.cu forward_fused): projections that are no passes over the weights as whole tiles with a norm or the rotation behind
// them, or gemm3 with those in its epilogue.  What tiles cost is the weights and a launch each, where gemm3's exchange and its wait for all other clusters cost as much
// again.  A step of 4 layers, gemm3 / tiles, us: Llama-3-8B sizes 9 tokens 401 / 391, 48 479 / 474, 49 506 / 487, 96 539 / 524, 128 579 / 537; 2048 wide 33 tokens
// 266 / 251, 128 330 / 299; 1024 wide 49 to 64 tokens 204 / 209, 128 223 / 206.  The rotation apart pays from 65 tokens on.
inline bool step_tiles(int tokens, int hidden) { return hidden >= 2048 || tokens <= 48 || tokens > 64; }
inline bool rotation_apart(int tokens) { return tokens > 64; }

// Latent rows (latent_attention.cu): in registers between their sum and their norm, or read again.  Registers for 1024 numbers a CTA cost room on
// an SM, which short rows and many of them feel; longer rows do not fit.  rank: the longest row asked for, 0 where only queries are rotated.
// us of two layers, again / held: ranks 1024 and 512, 8 tokens 21 / 17, 4096 43 / 38; 512 and 256, 8 18 / 16, 2400 27.8 / 26.4, 4096 34.3 / 36.3; 128 and
// 64, 600 tokens 18 / 19, 4096 33 / 38.  One kernel that could do both: 1500 and 1100, 4096 tokens 63 / 73, 2048 60 / 73.
inline bool latent_rows_held(int rank, int tokens) { return rank <= 1024 && (rank > 512 || tokens <= 4 * (rank > 128 ? rank : 128)); }

}  // namespace rules
}  // namespace b200
