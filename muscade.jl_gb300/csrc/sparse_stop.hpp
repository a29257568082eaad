// When the sweeps around the multifrontal factors stop (sparse_lu.cu; host-compilable).
//
// A sweep corrects the scaled solution y by c = M⁻¹ r, r the residual of y itself.
// The factors M are FP32 ones as a rule, and the corrections shrink by their error,
// |I − M⁻¹A|, until they are the rounding of r seen through M⁻¹: the accuracy that FP64
// attains, 1e-14 to 1e-10 of y as the matrix is conditioned.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define SP_HD __host__ __device__ inline
#else
#define SP_HD inline
#endif

namespace mgpu {

constexpr double kRefineTol = 1e-14;    // correction / solution: converged
constexpr double kRefineNear = 1e-11;   // ... or below this with the next one 0.1 kRefineTol
constexpr double kRefineStall = 1e-10;  // ... or no longer shrinking below this

enum SpStop : int { SP_GO_ON = 0, SP_CONVERGED = 1, SP_NOT_FINITE = 2 };

// The largest entries of a sweep's correction (c) and of the solution with it (y), the
// largest residual that the correction came from (r) and the largest of its rows'
// |A||y| + |b| (a), all scaled; nrow: most entries in a row.  sweep counts from 1;
// last[3] keeps the last correction, the worst rate of the sweeps so far and whether the
// last one had stopped shrinking.
// Converged:
//  * c <= 1e-14 y;
//  * from the third sweep on, c <= 1e-11 y and the next correction below 1e-15 y at the
//    worst rate so far (not the last: the rate may worsen again, the method lessens
//    |M⁻¹r|₂ over the sweeps so far, not its largest entry; a rate a thousand times the
//    worst still leaves 1e-12);
//  * c <= 1e-10 y and no better than half the last one: after plain sweeps at once; after
//    mixed ones with r down at its own rounding, (nrow + 4) 2⁻⁵³ a, or for the second time
//    in a row: with neither it may be a plateau of the method instead of the accuracy
//    attained.  (Factors of raised pivots add rounding of their own, and r stays a
//    hundred times higher.)
// Without the second rule a sweep or two at the rounding level follow where the matrix
// is conditioned well: 12 x 12 x 6 lattice 44.6 -> 51.7 ms for its three load steps;
// 60 x 60 x 20 takes 9 sweeps a solve either way (491 ms).
SP_HD SpStop sp_stop(bool mixed, int sweep, double c, double y, double r, double a, int nrow, double last[3]) {
  if (!(c <= 1.7e308) || !(y <= 1.7e308)) return SP_NOT_FINITE;
  const bool again = sweep > 1;
  const double prev = last[0], rate = again ? fmax(last[1], c / prev) : 0.0;
  const bool still = again && c >= 0.5 * prev, before = again && last[2] != 0.0;
  last[0] = c;
  last[1] = rate;
  last[2] = still ? 1.0 : 0.0;
  if (c <= kRefineTol * y) return SP_CONVERGED;
  if (sweep >= 3 && c <= kRefineNear * y && c * rate <= 0.1 * kRefineTol * y) return SP_CONVERGED;
  if (still && c <= kRefineStall * y && (!mixed || before || r <= (nrow + 4) * 0x1p-53 * a)) return SP_CONVERGED;
  return SP_GO_ON;
}

}  // namespace mgpu
