// Host build of reciprocal_near (sdtfe_b200/csrc/walk64.cuh) for
// tests/test_reciprocal.py.  Test scaffolding only.
#include "walk64.cuh"

extern "C" void reciprocals(const double* s, const double* near, int n, double* out) {
  for (int i = 0; i < n; ++i) out[i] = sdtfe::reciprocal_near(s[i], 1.0 / near[i]);
}
