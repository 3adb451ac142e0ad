"""GPU: K*u of every precision on grids that are mostly void in large pieces, with the
tiles' activity maps (made by the assembly): CTAs that own no active node write
zeros and take no part in the sum u . K u.

A solid slab is moved through the grid node plane by node plane along each axis, so that
it starts and ends at, one before and one after every tile border, whatever tile the
grid gets.  Reference: the element product in plain numpy FP64.  Tolerances as in
test_gpu_kbyu_tiles and test_gpu_parity: FP64 1e-13, double-float 1e-12, FP32 1e-5 of the
largest entry; the sum u . K u 1e-12 of the sum of magnitudes, as in test_zz_no_alloc.
"""
import ctypes

import numpy as np
import pytest

from test_gpu_kbyu_tiles import numpy_kbyu
from test_gpu_parity import _rel

pytestmark = pytest.mark.gpu

SHAPE = (64, 48, 56)


@pytest.mark.parametrize("thickness", [1, 6])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_slab_moved_through_a_void_grid(built_lib, axis, thickness):
    import torch

    from sgldbench_gb300 import VoxelSolver

    for at in range(0, 27):
        rng = np.random.default_rng(100 * axis + at)
        vox = np.zeros(SHAPE, dtype=bool)
        cut = [slice(5, 27), slice(9, 20), slice(3, 22)]
        cut[axis] = slice(at, at + thickness)
        vox[tuple(cut)] = True
        vox[-1, -1, -1] = True
        s = VoxelSolver(vox, num_levels=3, non_dyadic=0, omega=0.6, pad=False)
        fixed = rng.random(s.numDOFs) < 0.3
        fixed[-24:] = True   # the single element of the far corner
        E = rng.uniform(0.1, 1.0, s.numElements)
        s.set_fixed_dofs(fixed)
        s.set_modulus(E)
        s.Solving_AssembleFEAstencil()
        u = rng.standard_normal(s.numDOFs)
        ref = numpy_kbyu(s, u, E, fixed)
        assert _rel(s.Solving_KbyU_MatrixFree(u), ref) <= 1e-13, at
        assert _rel(s.kbyu_double_float(u), ref) <= 1e-12, at
        assert _rel(s.Solving_KbyU_MatrixFree(u, "mixed"), ref) <= 1e-5, at
        # the sum, by the call on full-grid vectors, whose void nodes are zero
        full = torch.zeros(3 * (SHAPE[0] + 1) * (SHAPE[1] + 1) * (SHAPE[2] + 1), dtype=torch.float64)
        where = (3 * (s.nodMapBack() - 1)[:, None] + np.arange(3)).reshape(-1)
        full[torch.from_numpy(where)] = torch.from_numpy(u)
        full = full.cuda()
        y = torch.full_like(full, np.nan)
        dot = torch.full((1,), np.nan, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert s.lib.sgld_kbyu_dot_noalloc(s.ctx, *(ctypes.c_void_p(t.data_ptr()) for t in (full, y, dot)), None) == 0
        torch.cuda.synchronize()
        got = y.cpu().numpy()
        assert _rel(got[where], ref) <= 1e-13, at
        got[where] = 0.0
        assert not got.any(), at   # zeros at every void node, in empty tiles and others
        assert abs(float(dot) - u @ ref) <= 1e-12 * (np.abs(u) @ np.abs(ref)), at
        s.close()
