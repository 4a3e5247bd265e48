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

}  // namespace rules
}  // namespace b200
