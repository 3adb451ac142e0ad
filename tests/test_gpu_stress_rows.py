"""GPU: the stress outputs of a model that fills its grid (rows copied as they are) and of one
with a single element missing, all nodes active (node rows copied, element rows
gathered) or not (both gathered): against the oracle, both principal outputs in one call
and one at a time.

Tolerances as in test_gpu_parity: stresses 1e-12, principal values 1e-10 of the largest.
"""
import ctypes

import numpy as np
import pytest

from oracle import glue as G
from test_gpu_parity import _rel, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("missing", [None, (3, 7, 4), (0, 15, 0)], ids=["none", "inside", "corner"])
def test_rows(built_lib, missing):
    vox = np.ones((8, 16, 8), bool)
    if missing:
        vox[missing] = False
    m, s = make_pair(vox, non_dyadic=0, seed=2)
    full = (s.resY + 1) * (s.resX + 1) * (s.resZ + 1)
    assert (s.numNodes == full) == (missing != (0, 15, 0))
    u = np.random.default_rng(9).standard_normal(s.numDOFs)
    s6_o, vmn_o = G.stress_analysis(m, u)
    s6, vmn, vme = s.FEA_StressAnalysis(u)
    assert _rel(s6, s6_o) <= 1e-12 and _rel(vmn, vmn_o) <= 1e-12
    assert _rel(vme, G.per_element_von_mises(m, s6_o)) <= 1e-12
    ps, dirs = s.FEA_ComputePrincipalStress(u)
    ref = G.principal_stress(s6_o)
    for k in (0, 4, 8):
        assert np.abs(ps[:, k] - ref[:, k]).max() <= 1e-10 * np.abs(ref[:, [0, 4, 8]]).max()
    p1, d1 = np.zeros_like(ps), np.zeros_like(dirs)

    def p(a):
        return a.ctypes.data_as(ctypes.c_void_p)

    assert s.lib.sgld_principal_stress(s.ctx, p(u), p(p1), None) == 0
    assert s.lib.sgld_principal_stress(s.ctx, p(u), None, p(d1)) == 0
    assert np.array_equal(p1, ps) and np.array_equal(d1, dirs)
    assert np.allclose(np.linalg.norm(dirs, axis=1), 1.0, atol=1e-12)
    s.close()
