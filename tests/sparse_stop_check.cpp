// sp_stop (csrc/sparse_stop.hpp) over a sequence of sweeps for test_sparse_stop.py:
// the sweep at which it stops, negative where a norm is not finite, 0 if it never does.
#include "sparse_stop.hpp"

extern "C" int sparse_stop_check(int mixed, int n, const double* c, const double* y, const double* r, const double* a, int nrow) {
  double last[3] = {0.0, 0.0, 0.0};
  for (int k = 0; k < n; ++k) {
    const int s = mgpu::sp_stop(mixed != 0, k + 1, c[k], y[k], r[k], a[k], nrow, last);
    if (s != mgpu::SP_GO_ON) return s == mgpu::SP_CONVERGED ? k + 1 : -(k + 1);
  }
  return 0;
}
