"""K*u of every precision over the grid shapes at which its tiles change:
one tile, ragged last tiles, grids thinner than a tile, one layer per CTA.

The reference is the element product in plain numpy FP64 with the context's
own element matrix.  FP64 tolerance 1e-13 of the largest entry: a node sums 8
x 24 products, each rounded a few times at 1.1e-16.
"""
import numpy as np
import pytest

from test_gpu_parity import _hadamard_to_ke, _rel

pytestmark = pytest.mark.gpu

# reference corner order, offsets (dy, dx, dz)
CORNERS = [(1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 0), (1, 0, 1), (1, 1, 1), (0, 1, 1), (0, 0, 1)]


def numpy_kbyu(s, u, E, fixed):
    ny, nx, nz = s.voxels.shape
    full = np.full((ny + 1) * (nx + 1) * (nz + 1), -1)
    full[s.nodMapBack() - 1] = np.arange(s.numNodes)
    e = s.eleMapBack() - 1
    y, x, z = e % ny, (e // ny) % nx, e // (ny * nx)
    nod = np.stack([full[(y + a) + (ny + 1) * ((x + b) + (nx + 1) * (z + c))] for a, b, c in CORNERS], 1)
    f = (u.reshape(-1, 3)[nod].reshape(-1, 24) @ s.Ke.T) * E[:, None]
    out = np.zeros((s.numNodes, 3))
    np.add.at(out, nod.reshape(-1), f.reshape(-1, 3))
    out = out.reshape(-1)
    out[fixed] = 0.0
    return out


@pytest.mark.parametrize("general", [False, True], ids=["cubic", "general"])
@pytest.mark.parametrize("shape,fill", [((2, 2, 2), 1.0), ((6, 34, 2), 0.6), ((46, 10, 62), 0.7), ((130, 4, 8), 0.5),
                                        ((10, 194, 6), 0.9), ((32, 64, 32), 1.0), ((70, 38, 26), 0.08)])
def test_kbyu_tiles(built_lib, shape, fill, general):
    from sgldbench_gb300 import VoxelSolver

    rng = np.random.default_rng(sum(shape))
    vox = rng.random(shape) < fill
    vox[0, 0, 0] = True
    s = VoxelSolver(vox, num_levels=2, non_dyadic=0, pad=False)
    if general:
        s.set_ke(_hadamard_to_ke(s.Ke, [([9, 20], 1.2), ([11, 16, 18], 0.9)]))
    fixed = rng.random(s.numDOFs) < 0.1
    E = rng.uniform(0.0, 1.0, s.numElements) ** 3
    s.set_fixed_dofs(fixed)
    s.set_modulus(E)
    if fill == 1.0 and not general:
        s.Solving_AssembleFEAstencil()   # makes the tiles' activity maps
    u = rng.standard_normal(s.numDOFs)
    ref = numpy_kbyu(s, u, E, fixed)
    assert _rel(s.Solving_KbyU_MatrixFree(u), ref) <= 1e-13
    assert _rel(s.kbyu_double_float(u), ref) <= 1e-12
    # a void element reads nothing: infinite values at its nodes do not reach it
    inf = np.full(s.numDOFs, np.inf)
    s.set_modulus(np.zeros(s.numElements))
    assert not s.Solving_KbyU_MatrixFree(inf).any()
    s.close()

