"""GPU: K*u on device vectors, which runs on the caller's vectors where it can (every
node active, device memory, no overlap) and through the grid's own where it cannot.
Both apply the same kernel to the same numbers, so each must equal the call on host
arrays bit for bit.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["apart", "same", "shifted", "pinned_u"])
@pytest.mark.parametrize("fill", [1.0, 0.6])
def test_kbyu_device_forms(built_lib, fill, form):
    import torch

    from sgldbench_gb300 import VoxelSolver

    rng = np.random.default_rng(3)
    vox = rng.random((10, 22, 14)) < fill
    vox[0, 0, 0] = True
    s = VoxelSolver(vox, num_levels=2, non_dyadic=0, pad=False)
    s.set_fixed_dofs(rng.random(s.numDOFs) < 0.1)
    s.set_modulus(rng.uniform(0.1, 1.0, s.numElements))
    u = rng.standard_normal(s.numDOFs)
    ref = s.Solving_KbyU_MatrixFree(u)
    n = s.numDOFs
    buf = torch.full((2 * n + 8,), np.nan, dtype=torch.float64, device="cuda")
    du = buf[1:n + 1]   # 8-byte alignment only
    if form == "pinned_u":
        du = torch.from_numpy(u.copy()).pin_memory()
    else:
        du.copy_(torch.from_numpy(u))
    dy = {"apart": buf[n + 2:2 * n + 2], "same": du, "shifted": buf[4:n + 4], "pinned_u": buf[n + 2:2 * n + 2]}[form]
    torch.cuda.synchronize()
    rc = s.lib.sgld_kbyu_device(s.ctx, ctypes.c_void_p(du.data_ptr()), ctypes.c_void_p(dy.data_ptr()))
    assert rc == 0
    assert np.array_equal(dy.cpu().numpy(), ref)
    if form == "apart":   # nothing past either vector is touched, u is not written
        assert torch.isnan(buf[0]) and torch.isnan(buf[n + 1]) and torch.isnan(buf[2 * n + 2:]).all()
        assert np.array_equal(du.cpu().numpy(), u)
    s.close()
