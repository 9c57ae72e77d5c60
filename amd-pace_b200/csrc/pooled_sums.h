// Where the prompt kernel of pooled attention (attn_pooled_umma.cu) keeps the sums of a unit between the KV heads of its keys.
#pragma once

#ifdef __CUDACC__
#define PACE_SUMS_FN __host__ __device__ __forceinline__
#else
#define PACE_SUMS_FN inline
#endif

namespace pace {

// A unit's part of the workspace, in float4: [KV heads of values][16-column pieces][rounds][4][rows].  A group of softmax warps has the
// pieces d = group, group + groups, ... of every head, one after the other; -1: no sums (the group has no piece, or no further one).
struct PooledSums {
  static constexpr int kGroups = 4, kRows = 128;
  int heads, pieces, rounds;
  PACE_SUMS_FN int size() const { return heads * pieces * rounds * 4 * kRows; }
  PACE_SUMS_FN int at(int head, int piece, int round) const { return ((head * pieces + piece) * rounds + round) * 4 * kRows; }
  PACE_SUMS_FN int first(int group) const { return group < pieces ? at(0, group, 0) : -1; }
  PACE_SUMS_FN int next(int group, int head, int piece, int round) const {
    if (round + 1 < rounds) return at(head, piece, round + 1);
    if (piece + kGroups < pieces) return at(head, piece + kGroups, 0);
    return head + 1 < heads ? at(head + 1, group, 0) : -1;
  }
};

}  // namespace pace
