"""GPU: the OC update where whole regions carry no strain energy, against the oracle.

Every node of the lowest element layers is fixed (the benchmark's clamping,
domains.fix_bottom_layers), so that within the filter's reach of them the filtered
sensitivity is a zero, whose sign the filter's sum decides, and the update's
x sqrt(-dc/dv/lmid) a zero of either sign: the design there goes down by the move limit
and the bisection has to count it so.

Tolerances as in test_gpu_topopt: every solve to 1e-10 on both sides, compliance
within 1e-6 relative, volume within 1e-9, change within 1e-5, xPhys within 1e-5.
"""
import numpy as np
import pytest

from oracle import glue as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers,rmin", [(4, 1.5), (6, 2.6)])
def test_oc_with_a_clamped_block_thicker_than_the_filter(built_lib, layers, rmin):
    from sgldbench_gb300 import VoxelSolver, domains

    vox = np.ones((8, 16, 16), bool)
    s = VoxelSolver(vox, omega=0.6)
    fixed = domains.fix_bottom_layers(s.voxels, s.nodMapBack(), layers)
    m = G.build_model_fixed(vox, fixed, omega=0.6)
    _, _, iz = domains.node_coords(s.nodMapBack(), *s.voxels.shape[:2])
    top = np.flatnonzero(iz == iz.max())
    m.F = np.zeros(s.numDOFs)
    m.F[3 * top + 2] = -1.0 / top.size
    m.F[3 * top[: top.size // 2]] = 0.5 / top.size
    s.set_fixed_dofs(fixed)
    opt = G.TopOptOptions(n_loop=4, rmin=rmin, tol=1e-10, maxit=2000, Emin=1e-9)
    xp_o, hist_o = G.topopt_global_volume(m, opt)
    xp, hist = s.TopOpti_GlobalVolumeConstraint(m.F, volfrac=0.3, rMin=rmin, nLoop=4, tol=1e-10, maxIT=2000, Emin=1e-9)
    assert len(hist) == len(hist_o) == 4
    for a, b in zip(hist, hist_o):
        assert abs(a["compliance"] - b["c"]) <= 1e-6 * abs(b["c"])
        assert abs(a["volume"] - b["vol"]) <= 1e-9
        assert abs(a["change"] - b["change"]) <= 1e-5
    assert np.abs(xp - xp_o).max() <= 1e-5 * np.abs(xp_o).max()
    assert abs(xp.mean() - 0.3) <= 1e-3   # the update meets the volume constraint
    s.close()


def test_oc_with_a_design_that_takes_the_other_comparison(built_lib):
    """-0 in the first design sends its elements' CTAs to fmin and fmax: the same designs, bit for
    bit, as +0 there."""
    from sgldbench_gb300 import VoxelSolver

    s = VoxelSolver(np.ones((8, 24, 16), bool), omega=0.6)
    m = G.build_model(np.ones((8, 24, 16), bool), omega=0.6)
    s.set_fixed_dofs(m.levels[0].fixedDOFs)
    x0 = np.full(s.numElements, 0.4)
    zero = np.random.default_rng(0).random(s.numElements) < 0.05
    runs = []
    for z in (0.0, -0.0):
        x0[zero] = z
        runs.append(s.TopOpti_GlobalVolumeConstraint(m.F, volfrac=0.35, nLoop=3, tol=1e-8, maxIT=2000, x0=x0))
    (xa, ha), (xb, hb) = runs
    assert np.array_equal(xa, xb)
    assert [h["change"] for h in ha] == [h["change"] for h in hb]
    s.close()
