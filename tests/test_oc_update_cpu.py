"""The OC update by comparisons of bit patterns (csrc/oc_update.cuh, what the bisection
sums) against the one by fmin and fmax (what is applied to the design), compiled for the
host: over zeros of both signs, denormals, numbers past 1 and below 0, infinities and NaNs
of both signs in every operand, and random numbers.  Wherever oc_ordered lets it be
taken it is equal (the update is a choice between its operands; a zero's sign does not
count), and oc_ordered turns down no design of [0, 1] with a sensitivity of either zero.
"""
import ctypes
import os
import subprocess

import numpy as np

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sgldbench_gb300", "csrc")
SRC = r"""
#include "oc_update.cuh"
extern "C" void both(long n, const double *x, const double *q, const double *rs, const double *m, double *a, double *b,
                     double *ok) {
    for (long i = 0; i < n; ++i) {
        a[i] = sgld::oc_new(x[i], q[i], rs[i], m[i]);
        b[i] = sgld::oc_new_bits(x[i], q[i], rs[i], m[i]);
        ok[i] = sgld::oc_ordered(x[i], q[i], m[i]);
    }
}
"""


def _both(tmp_path, x, q, rs, m):
    (tmp_path / "both.cpp").write_text(SRC)
    so = str(tmp_path / "both.so")
    # -ffp-contract=off: x - move and q rs are rounded in both forms
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
                    str(tmp_path / "both.cpp"), "-o", so], check=True)
    arg = [np.ascontiguousarray(v, dtype=np.float64) for v in (x, q, rs, m)]
    out = [np.empty(arg[0].size) for _ in range(3)]
    ptr = [a.ctypes.data_as(ctypes.c_void_p) for a in arg + out]
    ctypes.CDLL(so).both(ctypes.c_long(arg[0].size), *ptr)
    return out[0], out[1], out[2] != 0.0


def _equal(a, b):
    return (a == b) | (np.isnan(a) & np.isnan(b))


def test_special_values(tmp_path):
    nan = np.float64(np.nan)
    v = np.array([0.0, -0.0, 5e-324, -5e-324, 1e-300, 0.1, 0.25, 0.5, 1.0, 1.5, 7.0, -0.1, -0.5, -1.0, -3.0, 1e308, -1e308,
                  np.inf, -np.inf, nan, np.copysign(nan, -1.0)])
    g = [a.reshape(-1) for a in np.meshgrid(v, v, np.array([0.0, 1e-5, 0.5, 1.0, 1e34, np.inf]), v, indexing="ij")]
    a, b, ok = _both(tmp_path, *g)
    bad = np.flatnonzero(ok & ~_equal(a, b))
    assert not bad.size, [[w[i] for w in g] + [a[i], b[i]] for i in bad[:5]]
    assert not _equal(a, b).all()   # and it is needed


def test_random_values(tmp_path):
    rng = np.random.default_rng(0)
    n = 200000
    x, m = rng.random(n), rng.choice([0.05, 0.1, 0.2, 1.0], n)
    q = x * np.exp(rng.uniform(-30, 30, n)) * rng.choice([1.0, 0.0, -0.0], n, p=[0.8, 0.1, 0.1]) + 0.0
    a, b, ok = _both(tmp_path, x, q, np.exp(rng.uniform(-12, 30, n)), m)
    assert ok.all() and _equal(a, b).all()
    # a design that nothing strains goes down by the move limit
    assert np.array_equal(b[q == 0], np.maximum(0.0, x - m)[q == 0])
