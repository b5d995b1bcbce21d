// Length of a work item of the MXFP8 streaming kernel, decided on the host.
#pragma once
#include <stdint.h>

namespace es_b200 {

constexpr int kDefaultItemKSteps = 16;   // tunable mm_item_k_steps
constexpr int kMaxItemTiles = 8;

// Consecutive weight tiles of one work item: as many as span item_k_steps K steps, at most eight.  Where item_k_steps is
// left at its default, a call also gets as many items as half the SMs while there are the tiles for it (`tiles`: weight
// tiles of the call, an upper bound known on the host): a call of few tiles is a matter of latency, and up to half the SMs
// the CTAs of both streaming shapes are on an SM at once.  Measured without the rule -> with it (one item per SM, per
// three SMs): 24 experts, 3000 rows, n = 896, k = 384: 32.0 -> 25.7 us (29.1, 25.4); 20, 600, 1024, 256: 22.5 -> 17.3
// (22.0, 17.7); 16, 100, 4096, 256: 14.5 -> 13.6 (15.0, 14.6); 8, 729, 640, 384: 23.8 -> 15.7.
inline int weight_tiles_per_item(int item_k_steps, int k_steps_per_tile, int64_t tiles, int sm_count) {
  const int steps = item_k_steps < 1 ? 1 : item_k_steps;
  int group = (steps + k_steps_per_tile - 1) / k_steps_per_tile;
  if (group > kMaxItemTiles) group = kMaxItemTiles;
  if (item_k_steps == kDefaultItemKSteps)
    while (group > 1 && tiles / group < sm_count / 2) --group;
  return group;
}

}  // namespace es_b200
