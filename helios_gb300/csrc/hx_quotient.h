// Division by a denominator whose reciprocal is stored (host and device).
#pragma once
#include <cmath>
#include <cstring>

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

// a / d for r = 1 / d: q = a r and one correction q + (a - q d) r (Markstein's
// division: three FP64 operations instead of a division's dozen). Where d is
// zero or infinite, or a infinite, the correction is inf - inf or 0 inf and q
// already the quotient; that shows in its exponent (an integer test, as
// the FP64 pipe is what the caller has least of).
__host__ __device__ __forceinline__ double stored_quotient(double a, double d, double r)
{
    const double q = a * r, x = fma(fma(-q, d, a), r, q);
#ifdef __CUDA_ARCH__
    const unsigned high = (unsigned)__double2hiint(x);
#else
    unsigned long long bits;
    memcpy(&bits, &x, sizeof bits);
    const unsigned high = (unsigned)(bits >> 32);
#endif
    return (high & 0x7FF00000u) != 0x7FF00000u ? x : q;
}
