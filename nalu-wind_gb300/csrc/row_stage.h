// Staging of a group of CSR rows in a warp's shared memory (row3_groups,
// assemble.cu). Host-callable: the CPU test checks it at sizes that no test
// mesh reaches.
#pragma once

#include <cstdint>

#include "dd.h"  // NW_HD

namespace nw {

// CSR entries of a group, [first, last). A group of ten node rows holds more
// than 2^31 only where nodes have about 24 million neighbours; the count is
// then cut to 2^31 - 1, which stages nowhere.
NW_HD int32_t stage_count(int64_t first, int64_t last) {
  return last - first < INT32_MAX ? int32_t(last - first) : INT32_MAX;
}
// Whether `cnt` entries behind `odd` (0 or 1) unused ones fit in smem_bytes.
// Compared in entries: the bytes of 2^28 entries are beyond 32 bits.
NW_HD bool stage_fits(int32_t cnt, int odd, int smem_bytes) { return cnt <= smem_bytes / 8 - odd; }

}  // namespace nw
