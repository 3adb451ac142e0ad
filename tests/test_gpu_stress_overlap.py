"""GPU: stress recovery whose output buffers overlap the displacements, in page-locked
memory (whose copy to the device runs on its own) and in ordinary memory: the same
numbers as with buffers of their own, bit for bit.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [True, False], ids=["pinned", "pageable"])
@pytest.mark.parametrize("fill", [1.0, 0.5])
def test_outputs_over_the_input(built_lib, fill, pinned):
    import torch

    from sgldbench_gb300 import VoxelSolver

    rng = np.random.default_rng(5)
    vox = rng.random((64, 128, 64)) < fill
    vox[0, 0, 0] = True
    s = VoxelSolver(vox, num_levels=3, non_dyadic=0, pad=False)
    fixed = np.zeros(s.numDOFs, bool)
    fixed[:3] = True
    s.set_fixed_dofs(fixed)
    s.set_modulus(rng.uniform(0.1, 1.0, s.numElements))
    u = rng.standard_normal(s.numDOFs)
    nn, ne = s.numNodes, s.numElements

    def buffer(n):
        t = torch.zeros(n, dtype=torch.float64)
        return (t.pin_memory() if pinned else t).numpy()

    def p(a):
        return a.ctypes.data_as(ctypes.c_void_p)

    def recover(U, nodal=None, vmn=None, vme=None):
        assert s.lib.sgld_stress(s.ctx, p(U), *(p(a) if a is not None else None for a in (nodal, vmn, vme))) == 0

    own = [buffer(6 * nn), buffer(nn), buffer(ne), buffer(12 * nn), buffer(3 * ne)]
    recover(u, *own[:3])
    assert s.lib.sgld_principal_stress(s.ctx, p(u), p(own[3]), None) == 0
    assert s.lib.sgld_principal_stress(s.ctx, p(u), None, p(own[4])) == 0
    buf = buffer(12 * nn)
    for k, ref in enumerate(own):
        for at in (0, 1000) if ref.size >= u.size + 1000 else (0,):   # the input inside the output, or over its start
            buf[:] = 0.0
            U, out = buf[at:at + u.size], buf[:ref.size]
            U[:] = u
            if k < 3:
                recover(U, *[out if i == k else None for i in range(3)])
            else:
                assert s.lib.sgld_principal_stress(s.ctx, p(U), *((p(out), None) if k == 3 else (None, p(out)))) == 0
            assert np.array_equal(out, ref), (k, at)
    s.close()
