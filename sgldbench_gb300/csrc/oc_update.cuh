// The optimality-criteria update of one element, for device code and (checked there over
// all kinds of operands) for the host.
#pragma once
#include <math.h>
#include <string.h>

#ifdef __CUDACC__
#define SGLD_HD __host__ __device__ __forceinline__
#else
#define SGLD_HD inline
#endif

namespace sgld {

SGLD_HD double oc_new(double xe, double qe, double rs, double move) {
    // max(0, max(x - move, min(1, min(x + move, x sqrt(-dc/dv/lmid)))))   (:87)
    return fmax(0.0, fmax(xe - move, fmin(1.0, fmin(xe + move, qe * rs))));
}

SGLD_HD unsigned long long oc_bits(double a) {
#ifdef __CUDA_ARCH__
    return (unsigned long long)__double_as_longlong(a);
#else
    unsigned long long b;
    memcpy(&b, &a, sizeof b);
    return b;
#endif
}

// Whether oc_new_bits may take this element at any rs >= 0: x finite and >= +0, q >= +0 or a NaN
// whose sign bit is clear, the move limit >= 0.  Nothing else makes sure of it: the first
// iteration's x and the move limit are the caller's, and where nothing strains the
// elements in the filter's reach, sqrt(-dc/dv) may be -0.
SGLD_HD bool oc_ordered(double xe, double qe, double move) {
    return oc_bits(xe) < 0x7ff0000000000000ull && (long long)oc_bits(qe) >= 0 && move >= 0.0;
}

// oc_new with the comparisons on the bit patterns, as FP64 operations bound the bisection.
// With oc_ordered, x + move and q rs are +0 or more, or a NaN, whose pattern is above every
// number's whatever its sign: the order of the unsigned patterns is fmin's.  x - move is
// a number, and a negative one is below all others as a signed pattern.
SGLD_HD double oc_min_bits(double a, double b) { return oc_bits(a) < oc_bits(b) ? a : b; }
SGLD_HD double oc_max_bits(double a, double b) { return (long long)oc_bits(a) > (long long)oc_bits(b) ? a : b; }
SGLD_HD double oc_new_bits(double xe, double qe, double rs, double move) {
    return oc_max_bits(0.0, oc_max_bits(xe - move, oc_min_bits(1.0, oc_min_bits(xe + move, qe * rs))));
}

}  // namespace sgld
