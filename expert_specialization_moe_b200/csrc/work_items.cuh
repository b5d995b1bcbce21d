// Work list of the MXFP8 grouped GEMM: what the host decides about it.
#pragma once
#include <stdint.h>

namespace es_b200 {

constexpr int kDefaultItemKSteps = 16;   // tunable mm_item_k_steps
constexpr int kMaxItemTiles = 8;
// Experts with at least this many rows are the heavy ones of the work list: bound by the tensor pipe rather than by HBM.
constexpr int kHeavyMinRows = 113;       // tunable mm_heavy_min_rows

// Consecutive weight tiles (for the CTA-pair kernel: of 256 weight rows) of one work item of an expert with few rows: as many
// as span item_k_steps K steps, at most eight.  Where item_k_steps is left at its default, a call also gets as many items as
// half the SMs, one per CTA pair, while there are the tiles for it (`tiles`: weight tiles of the call, an upper bound known
// on the host): a call of few tiles is a matter of latency.  Measured without the rule -> with it: 3 rows on 8
// experts, n = k = 1024: 8.7 -> 7.3 us; 8, 400 rows, n = 2048, k = 1024: 9.9 -> 8.6; 64, 300 rows, n = 896, k = 512: 11.1 ->
// 12.5 (it cannot see which experts have rows; 11.1 since an expert's tiles are divided evenly).  Heavy experts get a quarter of it (their K steps take longer,
// and an item must not be long at the end of a call).
inline int weight_tiles_per_item(int item_k_steps, int k_steps_per_tile, int64_t tiles, int sm_count) {
  const int steps = item_k_steps < 1 ? 1 : item_k_steps;
  int group = (steps + k_steps_per_tile - 1) / k_steps_per_tile;
  if (group > kMaxItemTiles) group = kMaxItemTiles;
  if (item_k_steps == kDefaultItemKSteps)
    while (group > 1 && tiles / group < sm_count / 2) --group;
  return group;
}

}  // namespace es_b200
