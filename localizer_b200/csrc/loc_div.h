// Division by a value whose reciprocal is at hand, rounded as the division
// itself. Plain C++ for the host too, where it is tested.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define LOC_HD __host__ __device__ __forceinline__
#else
#define LOC_HD inline
#endif

namespace locb {

// a / b rounded correctly, with inv = RN(1 / b): Markstein's two residual
// corrections ("Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990). The first brings the
// quotient within one ulp, the second rounds it correctly; both residuals
// are exact while no intermediate leaves the normal range, which the caller
// ensures (in_range, div_fast).
LOC_HD double div_by(double a, double b, double inv)
{
    double q = a * inv;
    q = fma(fma(-b, q, a), inv, q);
    return fma(fma(-b, q, a), inv, q);
}
// dividends, and divisors, for which that holds over two divisions in a row
LOC_HD bool in_range(double a) { return fabs(a) > 0x1p-300 && fabs(a) < 0x1p300; }
LOC_HD bool div_fast(double b) { return fabs(b) > 0x1p-100 && fabs(b) < 0x1p100; }

}  // namespace locb
