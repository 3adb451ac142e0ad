"""GPU: the events of an FP64 solve go with it when it ends early.

A shim between the library and the CUDA runtime (loaded before it, in a process of its own)
counts events made and destroyed and gives one call an error code of its own instead of
making it.  The call is refused on the host; what was launched before it finishes.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include <dlfcn.h>
static void *next(const char *name) { return dlsym(dlopen(CUDART, RTLD_LAZY), name); }
typedef void *ev;
static int live, refuse;   // refuse: which of the next cudaStreamWaitEvent calls fails (1 the next), 0 none
int live_events(void) { return live; }
void refuse_wait(int n) { refuse = n; }
int cudaEventCreate(ev *e) {
    int (*f)(ev *) = (int (*)(ev *))next("cudaEventCreate");
    int r = f(e);
    live += r == 0;
    return r;
}
int cudaEventCreateWithFlags(ev *e, unsigned flags) {
    int (*f)(ev *, unsigned) = (int (*)(ev *, unsigned))next("cudaEventCreateWithFlags");
    int r = f(e, flags);
    live += r == 0;
    return r;
}
int cudaEventDestroy(ev e) {
    int (*f)(ev) = (int (*)(ev))next("cudaEventDestroy");
    live -= 1;
    return f(e);
}
int cudaStreamWaitEvent(void *s, ev e, unsigned flags) {
    int (*f)(void *, ev, unsigned) = (int (*)(void *, ev, unsigned))next("cudaStreamWaitEvent");
    if (refuse && --refuse == 0) return 2;   // cudaErrorMemoryAllocation
    return f(s, e, flags);
}
"""
CODE = r"""
import ctypes, sys
import numpy as np
from sgldbench_gb300 import VoxelSolver, domains
shim = ctypes.CDLL(sys.argv[1])
s = VoxelSolver(np.ones((8, 16, 8), bool), omega=0.6)
F, fixed = domains.cantilever3(s.voxels, s.nodMapBack(1), nelx=16)
s.set_fixed_dofs(fixed)
s.set_modulus(np.ones(s.numElements))
s.Solving_AssembleFEAstencil()
ref, _ = s.pcg(F, tol=1e-8, maxIT=500)
before = shim.live_events()
for n in (1, 2, 5):
    shim.refuse_wait(n)
    try:
        s.pcg(F, tol=1e-8, maxIT=500)
        print("no error")
    except Exception as e:
        print("error", type(e).__name__)
print("left", shim.live_events() - before)
U, info = s.pcg(F, tol=1e-8, maxIT=500)   # the context is as good as before
print("same", bool(np.array_equal(U, ref)))
"""


def test_no_event_outlives_a_solve_that_fails(built_lib, tmp_path):
    (tmp_path / "shim.c").write_text(SHIM)
    (tmp_path / "run.py").write_text(CODE)
    so = str(tmp_path / "shim.so")
    needed = subprocess.run(["ldd", built_lib], capture_output=True, text=True, check=True).stdout.split()
    cudart = [w for w in needed if w.startswith("/") and "libcudart" in w][0]
    subprocess.run(["gcc", "-O1", "-w", "-shared", "-fPIC", f'-DCUDART="{cudart}"', str(tmp_path / "shim.c"), "-o", so,
                    "-ldl"], check=True)
    r = subprocess.run([sys.executable, str(tmp_path / "run.py"), so], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "LD_PRELOAD": so, "PYTHONPATH": ROOT})
    out = r.stdout.split("\n")
    assert r.returncode == 0, r.stderr[-2000:]
    assert [l.split()[0] for l in out if l[:5] in ("error", "no er")] == ["error"] * 3, r.stdout
    assert "left 0" in out and "same True" in out, r.stdout
