"""GPU: the FP32 V-cycle whose small levels are chained into single launches, against the
oracle's level-by-level cycle: two to four levels below the finest, base levels
within and past the size where the chain starts, solid and sparse, coarse grids of a
few nodes.

Tolerance as in test_gpu_transfers: 1e-4 of the largest entry (FP32 sums on every
level and an FP32 coarsest inverse of condition ~1e3).
"""
import numpy as np
import pytest

from oracle import glue as G
from test_gpu_parity import _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,levels,fill", [((4, 12, 8), 3, 1.0), ((8, 40, 16), 4, 0.7), ((24, 8, 56), 4, 1.0),
                                               ((32, 64, 48), 5, 0.5), ((32, 96, 32), 6, 0.8), ((64, 96, 64), 4, 0.4)])
def test_vcycle_fp32_chained_levels(built_lib, shape, levels, fill):
    from sgldbench_gb300 import VoxelSolver

    rng = np.random.default_rng(sum(shape) + levels)
    vox = rng.random(shape) < fill
    vox[:, 0, :] = True   # the clamped face
    m = G.build_model(vox, non_dyadic=0, omega=0.6, num_levels=levels)
    s = VoxelSolver(vox, num_levels=levels, non_dyadic=0, omega=0.6, pad=False)
    E = rng.uniform(0.05, 1.0, s.numElements)
    G.set_modulus(m, E)
    s.set_fixed_dofs(m.levels[0].fixedDOFs)
    s.set_modulus(E)
    G.assemble_stencil(m)
    s.Solving_AssembleFEAstencil()
    assert m.numLevels == levels
    r = rng.standard_normal(m.levels[0].numDOFs)
    r[m.levels[0].fixedDOFs] = 0.0
    z = s.Solving_Vcycle(r, "mixed")
    assert _rel(z, G.vcycle(m, r)) <= 1e-4
    # scratch vectors keep zeros at inactive nodes from one cycle to the next
    assert np.array_equal(z, s.Solving_Vcycle(r, "mixed"))
    s.close()


@pytest.mark.parametrize("shape,levels,fill", [((8, 40, 24), 4, 1.0), ((16, 48, 32), 5, 0.6), ((32, 64, 32), 6, 1.0)])
def test_vcycle_fp32_chained_levels_non_dyadic(built_lib, shape, levels, fill):
    """The first level 4 times coarser: one to three levels below it."""
    from sgldbench_gb300 import VoxelSolver

    rng = np.random.default_rng(sum(shape) + levels)
    vox = rng.random(shape) < fill
    vox[:, 0, :] = True
    m = G.build_model(vox, non_dyadic=1, omega=0.6, num_levels=levels)
    s = VoxelSolver(vox, num_levels=levels, non_dyadic=1, omega=0.6, pad=False)
    E = rng.uniform(0.05, 1.0, s.numElements)
    G.set_modulus(m, E)
    s.set_fixed_dofs(m.levels[0].fixedDOFs)
    s.set_modulus(E)
    G.assemble_stencil(m)
    s.Solving_AssembleFEAstencil()
    r = rng.standard_normal(m.levels[0].numDOFs)
    r[m.levels[0].fixedDOFs] = 0.0
    z = s.Solving_Vcycle(r, "mixed")
    assert _rel(z, G.vcycle(m, r)) <= 1e-4
    assert np.array_equal(z, s.Solving_Vcycle(r, "mixed"))
    s.close()
