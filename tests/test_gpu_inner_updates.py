"""GPU: the inner CG's vector updates over the shapes at which they change form:
flat vectors or active runs (heads and tails off the 16-byte boundaries, runs shorter
than a group, runs longer than a lane's batch), alpha and beta summed by the update or,
past 1024 partials, by a launch of their own.

An update that skips or repeats a word, or a wrong alpha or beta, leaves s different
from r - K e, so that CG converges to something else and the outer FP64 iteration has to
make up for it.  Checked: the FP64 residual of the answer by the tested FP64 K*u
(the tolerance asked for, 1e-8, with 1 % for the recurrence's own drift), no fallback, and
inner iterations of at most three times the FP64 solve's (FP32 CG restarted about 3 times
on the way to 1e-8 repeats its early iterations).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def carved(shape, cut=None):
    vox = np.ones(shape, dtype=bool)
    if cut:
        vox[cut] = False
    return vox


SHAPES = [("tiny", carved((3, 7, 2))),
          ("flat", carved((13, 31, 11))),
          ("runs_short", carved((5, 40, 9), np.s_[1:4, 3:37, 2:9])),
          ("runs_odd", carved((37, 45, 21), np.s_[5:30, 7:40, 3:18])),
          ("runs_long", carved((190, 30, 20), np.s_[3:187, 4:20, 5:18])),
          ("flat_many_partials", carved((96, 160, 96))),
          ("runs_many_partials", carved((96, 160, 96), np.s_[11:90, 20:150, 7:80]))]


@pytest.mark.parametrize("vox", [v for _, v in SHAPES], ids=[n for n, _ in SHAPES])
def test_mixed_solve_residual_and_iterations(built_lib, vox):
    from sgldbench_gb300 import VoxelSolver
    from sgldbench_gb300 import domains as D

    s = VoxelSolver(vox, num_levels=2 if vox.size < 10000 else 4, non_dyadic=0, omega=0.6)
    F, fixed = D.cantilever3(s.voxels, s.nodMapBack(1), nelx=vox.shape[1])
    s.set_fixed_dofs(fixed)
    s.set_modulus(np.random.default_rng(vox.shape[1]).uniform(0.2, 1.0, s.numElements))
    s.Solving_AssembleFEAstencil()
    _, i64 = s.pcg(F, tol=1e-8, maxIT=2000, precision="fp64")
    assert i64["converged"]
    b = np.where(fixed, 0.0, F)
    for prec in ("mixed", "mixed_df"):
        U, info = s.pcg(F, tol=1e-8, maxIT=500, precision=prec)
        assert info["converged"] and not info["fallback"], info
        r = np.where(fixed, 0.0, b - s.Solving_KbyU_MatrixFree(U))
        assert np.linalg.norm(r) <= 1.01e-8 * np.linalg.norm(b)
        assert info["inner_its"] <= 3 * i64["its"] + 16, (info, i64)
    s.close()
