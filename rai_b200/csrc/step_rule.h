// Which single-token steps run as one kernel (step.cu), as far as their cached keys and values decide it (host code without CUDA in it: the
// rule is tested against a table of measured times in tests/test_step_rule.py).
#pragma once
#include <algorithm>

#include "attention_splits.h"

namespace rb {

// How step_kernel shares the keys out: it takes the cheapest of 16 ways by the same account (a tile 4, a piece 35, cut pairs 25).
struct StepPieces {
  int each, widest;   // pieces of a CTA; tiles of a piece, at most
  bool cut;
};
inline StepPieces step_pieces(const int* lens, int batch, int kv_heads, int ctas, int most_pieces) {
  int most = 0;
  for (int b = 0; b < batch; ++b) most = std::max(most, (lens[b] + 63) / 64);
  StepPieces best{0, 0, false};
  int best_cost = 1 << 24;
  for (int ways = 0; ways < 16; ++ways) {
    const int q = std::max(1, (most + ways) / (ways + 1));
    int line = 0, widest = 0;
    for (int b = 0; b < batch; ++b) {
      const int t = (lens[b] + 63) / 64, n = (t + q - 1) / q;
      line += n * kv_heads;
      if (n) widest = std::max(widest, (t + n - 1) / n);
    }
    const StepPieces w{(line + ctas - 1) / ctas, widest, q < most};
    const int cost = w.each * (w.widest * 4 + 35) + (w.cut ? 25 : 0);
    if (line <= most_pieces && cost < best_cost) { best_cost = cost; best = w; }
  }
  return best;
}

// Steps as separate launches spend about 8.2 us a layer more between their kernels, but their attention is shorter where the CTAs' pieces
// come out uneven or walk their tiles alone: 5 sequences of 32 heads are 160 pairs for 148 CTAs, so 80 CTAs walk two each.
// Microseconds of both: here the busiest CTA's pieces (3.5 each, 2.5 where pairs are cut, 0.5 a tile, 0.72 where several query heads of 128
// multiply it), there the account of attention_splits.h, but not below the bytes at 6 TB/s.  us a layer, launches -> one kernel:
// phi3-mini 5 x 1500 84.7 -> 82.8, 5 x 2000 90.8 -> 91.9, 5 x 2700 99.0 -> 101.6, 8 x 1700 90.1 -> 88.0, 4 x 3400 91.6 -> 84.1; phi2 5 x 1500
// 75.7 -> 74.0, 5 x 2000 81.3 -> 83.6; qwen2-7b 8 x 16000 142.8 -> 140.7, 1 x 90000 148.0 -> 155.6.  Not
// caught: qwen2-7b 8 x 20000 152.1 -> 159.0 (288 pieces of 35 tiles, two a CTA, run into the bytes' time).
inline bool step_attention_pays(const int* lens, int batch, int kv_heads, int group, int head_dim, int ctas, int most_pieces) {
  const StepPieces w = step_pieces(lens, batch, kv_heads, ctas, most_pieces);
  const double tile = head_dim > 96 && group > 1 ? 0.72 : 0.5;
  const double one = w.each * (w.widest * tile + 3.5) + (w.cut ? 2.5 : 0.0);
  int most = 0;
  double keys = 0.0;
  for (int b = 0; b < batch; ++b) { most = std::max(most, lens[b]); keys += lens[b]; }
  const SplitCost c = attention_split_cost(head_dim, group, ctas);
  const int pairs = batch * kv_heads, tiles = (most + 63) / 64;
  const double many = std::max(key_split_cost(c, pairs, tiles, pick_key_splits(c, pairs, tiles)), keys * 4.0 * kv_heads * head_dim / 6e6);
  return one - many <= 8.2;
}

}  // namespace rb
