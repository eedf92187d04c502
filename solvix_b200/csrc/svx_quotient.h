// svx_quotient.h - a division off the critical path (device code of
// svx_resident.cu; also compiles for the host, where its test runs).
#ifndef SVX_QUOTIENT_H
#define SVX_QUOTIENT_H

#include <cmath>

#ifdef __CUDACC__
#define SVX_QUOTIENT_FN __device__ __forceinline__
#else
#define SVX_QUOTIENT_FN inline
#endif

namespace svx {

// x / y from y's reciprocal: one residual correction brings the product to
// within an ulp of the quotient (Markstein 1990); operands outside the range
// where the residual is exact take the division.
SVX_QUOTIENT_FN double quotient(double x, double y, double y_inv) {
    const double ay = fabs(y), ax = fabs(x);
    if (!(ay > 1e-140 && ay < 1e140 && ax > 1e-140 && ax < 1e140)) return x / y;
    const double q = x * y_inv;
    return fma(fma(-y, q, x), y_inv, q);
}

}  // namespace svx

#endif  // SVX_QUOTIENT_H
