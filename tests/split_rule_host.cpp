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
// The other rules by size of the block solves.
extern "C" int items_few(int mixed, int64_t items, int num_sms) {
  return mixed ? oco::mixed_items_few(items, num_sms) : oco::solve_items_few(items, num_sms);
}
extern "C" int mixed_mode(int arrays, int layout, int64_t items, int nz) {
  const void *p = &items;
  return oco::mixed_store_mode(arrays > 0 ? p : nullptr, arrays > 1 ? p : nullptr, arrays > 2 ? p : nullptr, layout, items, nz);
}
