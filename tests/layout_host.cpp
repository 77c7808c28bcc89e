// Host build of the kernels' data layouts (oco_internal.h) for tests/test_layout_host.py.
#include "oco_internal.h"

extern "C" int layout_record_alignment() { return (int)alignof(oco::PillarRecord); }
extern "C" int layout_record_doubles() { return (int)(sizeof(oco::PillarRecord) / sizeof(double)); }
extern "C" int layout_record_fields() { return (int)oco::NF; }
extern "C" int64_t layout_tile_level(int z) { return oco::tile_level(z); }
extern "C" uint64_t layout_split_doubles(int64_t tiles, int nz) { return oco::split_scratch_doubles(tiles, nz); }
