// Division by a divisor whose reciprocal is known, for host and device code.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define MI_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define MI_HOST_DEVICE inline
#endif

namespace mi {

// a / b with y = 1 / b rounded to double, both computed once: the correctly rounded quotient by P. Markstein's theorem ("Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990): a quotient within one ulp, corrected with its exact remainder
// times y, rounds correctly.  a * y may be a little further off than that, hence two corrections.  Five multiply-adds in a row
// where the general division takes some 360 cycles in the middle of every norm.  b is finite and positive; a finite a is zero or far from the
// ends of the exponent range (the sum of squares of fp32 values is).  An infinite a has no remainder and is its own quotient, a NaN stays one.
MI_HOST_DEVICE double div_known(double a, double b, double y) {
    double q = a * y;                               // (not contracted: the product is used as a factor only)
    q = fma(fma(-q, b, a), y, q);
    q = fma(fma(-q, b, a), y, q);
    return fabs(a) < HUGE_VAL ? q : a;
}

}  // namespace mi
