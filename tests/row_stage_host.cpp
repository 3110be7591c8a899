// Host build of the row staging rules (nalu-wind_gb300/csrc/row_stage.h) for
// tests/test_row_stage.py.
#include <cstdint>

#include "row_stage.h"

extern "C" int row_staged(int64_t first, int64_t last, int smem_bytes) {
  return nw::stage_fits(nw::stage_count(first, last), int(first & 1), smem_bytes);
}
