// dustb_div.cuh -- a correctly rounded FP64 quotient from the divisor's reciprocal.  Plain C++ on
// the host: its test runs there (multiplications and fused multiply-adds round alike on both).
#pragma once

#ifdef __CUDACC__
#define DUSTB_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define DUSTB_HD inline
#endif

namespace dustb {

DUSTB_HD double fused(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return ::fma(a, b, c);
#endif
}

// n / d, correctly rounded, from y = 1 / d correctly rounded: two steps of Markstein's
// quotient iteration (P. Markstein, IBM J. Res. Dev. 34 (1990) 111): the first brings the
// quotient within an ulp, the second rounds it correctly.  For d and n of 1e-150 to 1e150 in
// magnitude, or n = 0 (the sign of a zero quotient is not kept): the residuals are exact there.
// The operands are cell widths and weights times distances
DUSTB_HD double div_by(double n, double d, double y) {
  double q = n * y;
  q = fused(fused(-q, d, n), y, q);
  return fused(fused(-q, d, n), y, q);
}

}  // namespace dustb
