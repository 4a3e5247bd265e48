// Rules that choose between two kernels with the same result by the sizes of a call alone, as plain host functions: the kernels'
// launchers use them, and b200_rule_query answers from them without a GPU.
#pragma once

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

}  // namespace rules
}  // namespace b200
