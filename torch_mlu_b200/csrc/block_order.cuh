// The order in which a kernel's row blocks run: heads in groups whose streamed tensors stay in L2 together, a group's blocks by rank, the
// heaviest first, across its heads. Under a causal mask the lightest ranks of all heads may come behind all groups, again heaviest first: a
// launch whose last group begins with heavy blocks ends on them, wherever the CTAs that took them stand (tail_ranks() in kernels.h).
#pragma once

#include <cuda_runtime.h>

namespace sdpa_b200 {

struct BlockOrder {
  int heads;            // (batch, head) pairs
  int ranks;            // row blocks per head, at the longest length
  int heads_per_group;
  int front_ranks;      // ranks that go group by group; the others come behind all groups
  int front_slots;      // slots of those (the last group may have slots without a head)
  int slots;
};

inline BlockOrder block_order(int heads, int ranks, int heads_per_group, int tail_ranks = 0) {
  BlockOrder o;
  o.heads = heads;
  o.ranks = ranks;
  o.heads_per_group = heads_per_group;
  o.front_ranks = ranks - tail_ranks;
  o.front_slots = (heads + heads_per_group - 1) / heads_per_group * heads_per_group * o.front_ranks;
  o.slots = o.front_slots + heads * tail_ranks;
  return o;
}

// False for a slot without a block.
__host__ __device__ __forceinline__ bool block_of_slot(const BlockOrder& o, int slot, int& rank, int& head) {
  if (slot >= o.front_slots) {
    const int w = slot - o.front_slots;
    rank = w / o.heads;
    head = w - rank * o.heads;
    rank += o.front_ranks;
    return true;
  }
  const int per_group = o.heads_per_group * o.front_ranks;
  const int grp = slot / per_group;
  const int w = slot - grp * per_group;
  const int size = min(o.heads_per_group, o.heads - grp * o.heads_per_group);
  rank = w / size;
  head = grp * o.heads_per_group + (w - rank * size);
  return rank < o.front_ranks;
}

}  // namespace sdpa_b200
