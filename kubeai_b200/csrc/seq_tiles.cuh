// Which (sequence, tile of its rows) CTA `idx` of a step has, when every sequence's rows are cut into tiles of TQ and the tiles are
// numbered through: the lanes of a warp look at 32 sequences at a time (one after the other, a step of 128 sequences spent 40
// us on it).  All lanes of the warp call it and get the same answer; false past the last tile.
#pragma once

namespace b200 {

__device__ __forceinline__ bool find_tile(const int* seqs, int nseq, int TQ, int idx, int* seq, int* tile) {
  const int lane = threadIdx.x & 31;
  for (int s0 = 0; s0 < nseq; s0 += 32) {
    const int s = s0 + lane, own = s < nseq ? (seqs[s * 8 + 1] + TQ - 1) / TQ : 0;
    int upto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned past = __ballot_sync(0xffffffffu, idx < upto);
    if (past) {
      const int at = __ffs(past) - 1;
      *seq = s0 + at;
      *tile = idx - __shfl_sync(0xffffffffu, upto - own, at);
      return true;
    }
    idx -= __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

}  // namespace b200
