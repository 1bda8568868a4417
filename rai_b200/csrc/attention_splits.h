// Into how many blocks the keys of a sequence are split at a single-token step (host code without CUDA in it: the rule is tested
// against the table of measured times in tests/test_attention_splits.py).
#pragma once
#include <algorithm>

namespace rb {

// Microseconds of one launch's parts, fitted to steps of ten models (heads of 64 to 256, latents, mixed heads; batches of 1, 4
// and 32; 2 to 17 tiles of 64 keys; every split).  A step is at most 2.4 % longer with the rule's choice than with the best one, and at
// most 3.2 % at batches of 2, 8 and 16 and 4 to 33 tiles, which the fit did not see.  A number of tiles cannot stand for the hand-over:
// with six tiles, 1 x 7 tiles took 128.9 us a layer instead of 94.0 (8 mixed heads of 128, 7.2 us a tile), with 1.5 tiles
// 1 x 5 tiles took 31.4 instead of 29.0 (2 heads of 64, 0.5 us a tile), with either 1 x 17 tiles 89.5 instead of 76.7 (one head of 256).
struct SplitCost {
  double start;   // a block before and after its tiles
  double tile;    // a tile of 64 keys in one block, which waits for copies rather than for bandwidth
  double hand;    // handing parts over to the block that comes last, and its merge:
  double part;    //   for each part
  int slots;      // blocks resident at once
};

// attention_kernel, one block per (sequence, key/value head): column blocks of 64, and `group` heads' sums to merge.
inline SplitCost attention_split_cost(int head_dim, int group, int sm_count) {
  const double sums = group * head_dim / 1024.0;
  return {7.4, 0.33 + 0.16 * ((head_dim + 63) / 64), 2.9 + 1.3 * sums, 0.1 + 0.25 * sums, (head_dim <= 128 ? 2 : 1) * sm_count};
}

// attention_joint.cuh, one block per sequence (or tile of its rows): the bytes of 64 keys of all heads, and the sums of all rows.
inline SplitCost joint_split_cost(int tile_bytes, int sums, int sm_count) {
  return {4.3, 0.027 * tile_bytes / 1024.0, 1.6 + 0.23 * sums / 1024.0, 0.5 + 0.035 * sums / 1024.0, sm_count};
}

// One block per pair keeps its copies coming and hands nothing over; splitting pays where pairs are few and their tiles take longer
// than the hand-over.  Blocks run in rounds of `slots`; each round that splitting adds costs a start.  Gains below 1 % are left alone:
// of many pairs they are no more than the end of the last round, which is not as even as this.
inline double key_split_cost(const SplitCost& c, int pairs, int tiles, int s) {
  const int rounds = (pairs * s + c.slots - 1) / c.slots;
  double cost = rounds * (c.start + c.tile * ((tiles + s - 1) / s));
  if (s > 1) cost += (c.hand + c.part * s) * std::max(1.0, (double)pairs / c.slots);
  return cost;
}
inline int pick_key_splits(const SplitCost& c, int pairs, int tiles) {
  int best = 1;
  double best_cost = 1e30;
  for (int s = 1; s <= std::min(tiles, 32); ++s) {
    const double cost = key_split_cost(c, pairs, tiles, s);
    if (cost < best_cost) {
      best_cost = s == 1 ? 0.99 * cost : cost;
      best = s;
    }
  }
  return best;
}

}  // namespace rb
