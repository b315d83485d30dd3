"""The weight-gradient kernel where a CTA takes many voxel chunks, the last
one partly filled, and where a grid line is longer than a chunk, against the
CPU network oracle.  Tolerance: one BF16 rounding that flips on one side is
2^-8 of that value; through the six layers' stored gradients these add to at
most 6 * 2^-8 in the relative L2 norm."""
import numpy as np
import pytest

from netcases import net_case, random_params

pytestmark = pytest.mark.gpu

LAYERS = [(4, 16), (16, 32), (32, 64), (64, 32), (32, 16), (16, 1)]


@pytest.mark.parametrize("shape", [(34, 30, 52), (10, 6, 130)])
def test_weight_gradient_over_many_chunks(lhi, oracle_mod, shape):
    from liquidhairinteration_b200.net import LearnedNet
    r, t, s = net_case(shape, seed=23)
    params = random_params(oracle_mod.net_num_params(), seed=24)
    dz = np.random.default_rng(25).standard_normal(shape).astype(np.float32)
    net = LearnedNet(seed=7)
    net.set_params(params)
    net.set_relu(False)
    oracle_mod.net_set_relu(False)
    g = net.backward(r, t, s, dz)
    net.close()
    g_o = oracle_mod.net_backward(params, r, t, s, dz)
    off = 0
    for cin, cout in LAYERS:
        nw = 27 * cout * cin
        a, b = g[off:off + nw].astype(np.float64), g_o[off:off + nw]
        err = np.linalg.norm(a - b) / np.linalg.norm(b)
        assert err < 6 / 256, (cin, cout, err)
        off += nw + cout
