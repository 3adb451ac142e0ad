"""The sums of the FP32 coarse apply (csrc/wide_sum.cuh) hold at least as much as FP64 ones.

Compiled for the host with the device's rounded operations as plain FP32 ones, which
round the same way.  Words of many magnitudes and both signs are added one by one into
8 sums, which are added in pairs as the kernel does it.  The exact sum is known from rational
arithmetic; a chain of N additions in FP64 is allowed N 2^-53 of the sum of magnitudes, so
the sum in words (before its rounding to FP32) has to be within one 2^-53 of it.
"""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sgldbench_gb300", "csrc")
SRC = r"""
#define __device__
#define __forceinline__ inline
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return __builtin_fmaf(a, b, c); }
static inline float __double2float_rn(double a) { return (float)a; }
static inline float __shfl_sync(unsigned, float v, int, int) { return v; }
struct float2 { float x, y; };
#include "wide_sum.cuh"
using W = sgld::WideSum<float>;
static_assert(sizeof(W) % sizeof(float) == 0, "words");
extern "C" int add_up(long n, const float *x, float *words, float *value) {
    W t[8] = {};
    for (long i = 0; i < n; ++i) t[i & 7].add(x[i]);
    const W s = ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
    __builtin_memcpy(words, &s, sizeof s);
    *value = s.value();
    return (int)(sizeof s / sizeof(float));
}
"""


def test_sum_of_many_magnitudes(tmp_path):
    (tmp_path / "w.cpp").write_text(SRC)
    so = str(tmp_path / "w.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, str(tmp_path / "w.cpp"),
                    "-o", so], check=True)
    lib = ctypes.CDLL(so)
    rng = np.random.default_rng(0)
    for trial in range(300):
        n = int(rng.integers(1, 400))
        x = (rng.standard_normal(n) * np.exp2(rng.uniform(-18, 18, n))).astype(np.float32)
        if trial % 3 == 0:
            x = np.abs(x)
        words, value = np.zeros(4, np.float32), ctypes.c_float()
        k = lib.add_up(ctypes.c_long(n), x.ctypes.data_as(ctypes.c_void_p), words.ctypes.data_as(ctypes.c_void_p),
                       ctypes.byref(value))
        exact = sum(Fraction(float(v)) for v in x)
        size = sum(abs(Fraction(float(v))) for v in x)
        held = sum(Fraction(float(v)) for v in words[:k])
        assert abs(held - exact) <= size / 2 ** 53, trial
        assert abs(Fraction(value.value) - exact) <= abs(exact) / 2 ** 24 + size / 2 ** 48


def test_infinite_sum(tmp_path):
    (tmp_path / "w.cpp").write_text(SRC)
    so = str(tmp_path / "w.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, str(tmp_path / "w.cpp"),
                    "-o", so], check=True)
    lib = ctypes.CDLL(so)
    for x, want in (([1.0, np.inf, 2.0], np.inf), ([-np.inf] + [3.0] * 9, -np.inf), ([np.inf, -np.inf], np.nan)):
        x = np.array(x, np.float32)
        words, value = np.zeros(4, np.float32), ctypes.c_float()
        lib.add_up(ctypes.c_long(x.size), x.ctypes.data_as(ctypes.c_void_p), words.ctypes.data_as(ctypes.c_void_p),
                   ctypes.byref(value))
        assert np.array_equal([value.value], [want], equal_nan=True)
