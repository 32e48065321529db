// Host build of the four-child records' box conversion, for the CPU test that compares it with exact
// arithmetic (test infrastructure; compiled by tests/test_box_centre_half.py).
#include <cstdint>

#include "layout.h"

extern "C" void centre_half(const float* lo, const float* hi, float* c, float* h, int64_t n) {
  for (int64_t i = 0; i < n; ++i) bvhc::box_centre_half(lo[i], hi[i], c[i], h[i]);
}
