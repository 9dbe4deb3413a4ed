// The eight basis functions of the TaylorF2 phase to more than float64's digits,
// for the fixed-point tables of gwl_wide.cu (host and device).
#pragma once

#include <cmath>
#include <cstdint>

#include <cuda_runtime.h>

#include "gwl_internal.h"

namespace gwl {

// The basis functions at frequency f (wide_lnref subtracted from ln f) as
// float64 pairs hi + lo; lo = 0 for the last four, whose coefficients stay
// within tens of cycles.
__host__ __device__ inline void wide_basis(double f, double lnref, double* hi, double* lo) {
  const double y = cbrt(f), p = y * y, pe = fma(y, y, -p), t = p * y, te = fma(p, y, -t) + pe * y;
  const double yl = ((f - t) - te) / (3.0 * p);
  const double h3 = 1.0 / y, l3 = (fma(-h3, y, 1.0) - h3 * yl) * h3;
  const double h2 = h3 * h3, l2 = fma(h3, h3, -h2) + 2.0 * h3 * l3;
  const double h1 = 1.0 / f, l1 = fma(-h1, f, 1.0) * h1;
  hi[0] = h1 * h2;
  lo[0] = fma(h1, h2, -hi[0]) + (h1 * l2 + l1 * h2);
  hi[1] = h1;
  lo[1] = l1;
  hi[2] = h2;
  lo[2] = l2;
  hi[3] = h3;
  lo[3] = l3;
  const double ln = log(f) - lnref;
  hi[4] = ln > 0 ? ln : 0.0;
  hi[5] = y;
  hi[6] = y * hi[4];
  hi[7] = p;
  for (int b = 4; b < kNumBasis; ++b) lo[b] = 0.0;
}

}  // namespace gwl
