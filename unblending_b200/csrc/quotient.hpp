// Correctly rounded division by a shared reciprocal.
#pragma once
#include <cmath>
#include <cstdint>

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

// RN(1/b) from an approximation y of relative error below 2^-16, for b and
// 1/b well inside the exponent range: Newton's iteration with fused residuals
// (Markstein, as above). The last step rounds correctly from a reciprocal
// within one unit in the last place, except where b's significand is all
// ones: the result there is the number above a power of two, and the
// iteration ends on either of the two.
UNB_HOST_DEVICE double refine_reciprocal(double b, double y) {
    y = fma(y, fma(-b, y, 1.0), y);
    y = fma(y, fma(-b, y, 1.0), y);
    return fma(y, fma(-b, y, 1.0), y);
}

#ifdef __CUDACC__
// RN(1/b) from the hardware's approximation, without the branch to a slow path
// that __drcp_rn takes, so that it overlaps the code around it (with
// __drcp_rn the two passes of the 1024x1024 five-layer image took 1.03 times as
// long).
__device__ __forceinline__ double reciprocal(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = refine_reciprocal(b, y);
    const bool ones = (uint32_t(__double2hiint(b)) | 0xfff00000u) == 0xffffffffu && __double2loint(b) == -1;
    return __hiloint2double(__double2hiint(y), ones ? 1 : __double2loint(y));
}
#endif

}  // namespace unb
