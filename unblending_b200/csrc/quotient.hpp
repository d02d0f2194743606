// Correctly rounded division by a shared reciprocal.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define UNB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define UNB_HOST_DEVICE inline
#endif

namespace unb {

// a / b from y = RN(1/b), correctly rounded (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990): two
// residual corrections of a*y; the first leaves a faithful quotient, the
// second rounds it correctly given that y is the correctly rounded
// reciprocal. It holds while the residuals are exact: |a| >= 2^-960 or a = 0
// (a negative zero gives a positive one), a normal quotient (below either
// bound the quotient can be off by its last bit), and nothing overflows. Five operations
// without a branch, so that the three channels' (and the gradient's twelve)
// divisions by one composite alpha overlap, where the compiler's division
// branches to its slow path after each. In the solver b is a composite alpha or
// a blend denominator in (1e-12, 2^240) and a is built from values in [0, 1]
// and such quotients, at most 2^600 over eight layers.
UNB_HOST_DEVICE double quotient(double a, double b, double y) {
    double q = a * y;
    double r = fma(-b, q, a);
    q = fma(r, y, q);
    r = fma(-b, q, a);
    return fma(r, y, q);
}

}  // namespace unb
