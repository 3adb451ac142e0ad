#pragma once
#include <math.h>

#include "df_arith.cuh"

namespace sgld {

// Sums of the coarse apply's blocks of 32 columns (kernels_asm.cu): in FP64, or for FP32 in
// three FP32 words, as an FP64 operation holds a warp's scheduler for 64 clocks (96 x 48 x 48: a
// V-cycle of 31.2 us, 33.4 with FP64 sums).  Every step adds a word exactly and hands its
// error to the next, and only the third is rounded: some 70 bits, where FP64 has 53.  What
// is left is the rounding within a block, 8 products in a row.
template <typename T>
struct WideSum;
template <>
struct WideSum<double> {
    double v;
    __device__ __forceinline__ void add(double a) { v += a; }
    __device__ __forceinline__ WideSum operator+(const WideSum &b) const { return {v + b.v}; }
    __device__ __forceinline__ double value() const { return v; }
};
template <>
struct WideSum<float> {
    float s, e, f;
    __device__ __forceinline__ void add(float a) {
        const df t = two_sum(s, a), u = two_sum(e, t.lo);
        s = t.hi;
        e = u.hi;
        f = __fadd_rn(f, u.lo);
    }
    __device__ __forceinline__ WideSum operator+(const WideSum &b) const {
        const df t = two_sum(s, b.s), u = two_sum(e, b.e), w = two_sum(u.hi, t.lo);
        return {t.hi, w.hi, __fadd_rn(__fadd_rn(f, b.f), __fadd_rn(u.lo, w.lo))};
    }
    // an infinite sum has no error terms
    __device__ __forceinline__ float value() const { return isinf(s) ? s : __fadd_rn(s, __fadd_rn(e, f)); }
};

}  // namespace sgld
