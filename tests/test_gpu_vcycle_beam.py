"""GPU: both V-cycles over a slender beam clamped along its long side's end plane only, whose coarsest
system is badly conditioned, with bounds that scale with its condition number kappa (2-norm,
from the oracle's factor).

The device factors the coarsest matrix in double-float arithmetic (u = 2^-48) and applies
M' M with M = L^-1, so the solution's relative error is a small multiple of u kappa; 16 is
allowed.  The FP32 cycle applies M from a sweep in FP32 (v = 2^-24), off by a small
multiple of v |M| |L|, so that y = M r is off by that of v kappa(L) |y| and x = M' y by that of
v sqrt(kappa) |M| |y|; 16 again.  Both are measured against the largest entry, and the rest of
the cycle adds the other tests' 1e-12 and 1e-6.
"""
import numpy as np
import pytest
from scipy.linalg import solve_triangular

from oracle import glue as G
from test_gpu_parity import _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 66, 4), (4, 96, 8), (8, 48, 4)])
def test_vcycle_of_a_beam(built_lib, shape):
    from sgldbench_gb300 import VoxelSolver

    rng = np.random.default_rng(sum(shape))
    vox = np.ones(shape, bool)
    m = G.build_model(vox, non_dyadic=0, omega=0.6, num_levels=2)
    s = VoxelSolver(vox, num_levels=2, non_dyadic=0, omega=0.6, pad=False)
    E = rng.uniform(0.05, 1.0, s.numElements)
    G.set_modulus(m, E)
    s.set_fixed_dofs(m.levels[0].fixedDOFs)
    s.set_modulus(E)
    G.assemble_stencil(m)
    s.Solving_AssembleFEAstencil()
    r = rng.standard_normal(m.levels[0].numDOFs)
    r[m.levels[0].fixedDOFs] = 0.0
    ref = G.vcycle(m, r)
    factor = np.tril(m.chol[0])
    sv = np.linalg.svd(factor, compute_uv=False)
    kappa = (sv[0] / sv[-1]) ** 2
    rc = G.restrict(m.levels, r, 2)[m.levels[1].freeDOFs]
    y = solve_triangular(factor, rc, lower=True)
    reach = np.linalg.norm(y) / sv[-1] / np.abs(ref).max()   # |M| |y| over the largest entry
    assert _rel(s.Solving_Vcycle(r), ref) <= 16 * 2.0 ** -48 * kappa + 1e-12
    bound32 = 16 * 2.0 ** -24 * np.sqrt(kappa) * reach + 1e-6
    assert bound32 < 0.1   # it says something
    assert _rel(s.Solving_Vcycle(r, "mixed"), ref) <= bound32
    s.close()
