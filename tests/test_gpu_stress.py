"""Stress recovery over sparse, ragged and thin models, and with displacements
that are not finite, against the oracle's product with the corner stress
matrix.  1e-12 of the largest entry, as in test_gpu_parity."""
import numpy as np
import pytest

from oracle import glue as G
from test_gpu_parity import _rel, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,fill", [((8, 16, 8), 0.3), ((40, 8, 12), 0.8), ((8, 8, 72), 0.5), ((24, 40, 8), 1.0)])
def test_stress(built_lib, shape, fill):
    rng = np.random.default_rng(sum(shape))
    vox = rng.random(shape) < fill
    vox[:, 0, :] = True
    m, s = make_pair(vox, non_dyadic=0, seed=1)
    u = rng.standard_normal(s.numDOFs)
    s6_o, vmn_o = G.stress_analysis(m, u)
    s6, vmn, vme = s.FEA_StressAnalysis(u)
    assert _rel(s6, s6_o) <= 1e-12 and _rel(vmn, vmn_o) <= 1e-12
    assert _rel(vme, G.per_element_von_mises(m, s6_o)) <= 1e-12
    vme2, vmn2 = s.vonmises(u)
    assert np.array_equal(vme2, vme) and np.array_equal(vmn2, vmn)
    # a displacement that is not finite spoils every node of its elements, and no other
    for bad in (np.nan, np.inf):
        w = u.copy()
        w[3 * (s.numNodes // 2)] = bad
        with np.errstate(invalid="ignore"):
            s6_o, _ = G.stress_analysis(m, w)
        s6, _, _ = s.FEA_StressAnalysis(w)
        ok = np.isfinite(s6_o).all(axis=1)
        assert not ok.all()
        assert np.array_equal(np.isfinite(s6).all(axis=1), ok)
        assert _rel(s6[ok], s6_o[ok]) <= 1e-12
    s.close()
