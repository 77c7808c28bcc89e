// Host build of the split block solve's rule (oco_internal.h) for tests/test_split_rule_host.py.
#include <algorithm>

#include "oco_internal.h"

extern "C" int split_rule(int grey, int64_t ncol, int nw, int nz, int num_sms, int max_blocks) {
  return oco::solve_is_split(grey, ncol, nw, nz, num_sms, max_blocks) ? 1 : 0;
}
// Blocks of the larger of its two grids.
extern "C" int64_t split_grid(int64_t ncol, int nw, int nz) {
  const int64_t tiles = oco::split_tiles(ncol, nw);
  return std::max(tiles, oco::split_row_blocks(tiles, nz));
}
