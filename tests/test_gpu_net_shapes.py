"""GPU: the U-Net's tensor-core convolutions at the shapes where their copies and
tiles change form, against the oracle restatement (oracle/net.py).

Channel counts that are multiples of 8 and only of 4 (asynchronous 16-byte copies or
element loads, padded rows of K and N), outputs that are not multiples of 4 (element
epilogue), from 1 to 15 taps per weight-gradient CTA (127 // ceil8(channels)); grids
smaller than one tile of 128 voxels, one voxel short of or past a tile, and spanning
two voxel ranges.  The tolerances are those of the oracle comparison for the ordinary
shapes: it rounds where the device rounds, so that only FP32 order and the BF16
flips it causes differ (one BF16 ulp is 3.9e-3): 2e-2 relative L2, 5e-2 for the
gradient of a single convolution.
"""
import numpy as np
import pytest

from oracle.net import UNet as OracleNet

pytestmark = pytest.mark.gpu

SHAPES = [((5, 4, 3), 4, 2, 1, [4]),             # 60 voxels, element loads, 15 taps per CTA
          ((127, 1, 1), 8, 3, 1, [8]),           # one short of a tile, flat in two directions
          ((43, 3, 1), 12, 1, 1, [12]),          # one past a tile
          ((11, 6, 9), 20, 3, 2, [4, 20]),
          ((17, 16, 8), 4, 3, 3, [12, 24, 40]),  # 2176 voxels: two ranges
          ((8, 16, 17), 16, 4, 2, [64, 64])]     # the widest: one tap per CTA


def _rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a, float) - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("dims,cin,cout,levels,widths", SHAPES, ids=[f"{s[0]}-{s[1]}-{s[4]}" for s in SHAPES])
def test_forward_and_gradient_match_oracle(built_lib, dims, cin, cout, levels, widths):
    from sgldbench_gb300.net import UNet

    net = UNet(dims, cin, cout, levels, widths, seed=11)
    orc = OracleNet(dims, cin, cout, levels, widths, emulate=True)
    rng = np.random.default_rng(12)
    V = int(np.prod(dims))
    x = rng.standard_normal((V, cin)).astype(np.float32)
    t = rng.standard_normal((V, cout)).astype(np.float32)
    m = (rng.random(V) > 0.25).astype(np.float32)
    p = net.get_params()
    p[orc.conv[-1][4]:] *= 10.0   # a head of ordinary size
    net.set_params(p)
    y_ref, _ = orc.forward(p.astype(np.float64), x)
    assert _rel_l2(net.forward(x), y_ref) <= 2e-2
    loss, g = net.grad(x, t, m)
    loss_ref, g_ref, _ = orc.value_and_grad(p.astype(np.float64), x, t, m)
    assert abs(loss - loss_ref) <= 1e-2 * loss_ref
    for ci, co, taps, _, wo, bo in orc.conv:
        assert _rel_l2(g[wo:bo + co], g_ref[wo:bo + co]) <= 5e-2
    net.close()
