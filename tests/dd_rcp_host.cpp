// Host build of the float-pair reciprocals (nalu-wind_gb300/csrc/dd.h) for
// tests/test_dd_rcp.py. The device takes its seed from an approximate
// instruction; here the caller gives it.
#include <cstdint>

#include "dd.h"

extern "C" void dd_rcp_seeded(int64_t n, const float* hi, const float* lo, const float* seed, float* rh, float* rl) {
  for (int64_t i = 0; i < n; ++i) {
    const nw::dd r = nw::dd_rcp_seed(nw::fast_two_sum(hi[i], lo[i]), seed[i]);
    rh[i] = r.hi;
    rl[i] = r.lo;
  }
}
