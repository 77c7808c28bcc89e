// Host build of the kernels' data layouts (oco_internal.h) for tests/test_layout_host.py.
#include "oco_internal.h"

extern "C" int layout_record_alignment() { return (int)alignof(oco::PillarRecord); }
extern "C" int layout_record_doubles() { return (int)(sizeof(oco::PillarRecord) / sizeof(double)); }
extern "C" int layout_record_fields() { return (int)oco::NF; }
