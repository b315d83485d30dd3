"""One network on grids of equal volume and different shape: the sparse
plan's buffers follow the shape (tests/test_cpu_net_buffers.py checks their
sizes), so a call gives the same bits as on a new network."""
import numpy as np
import pytest

from netcases import net_case, random_params

pytestmark = pytest.mark.gpu

SHAPES = [(17, 16, 16), (16, 17, 16), (16, 16, 17), (16, 16, 16), (64, 8, 8), (8, 64, 8)]


def test_equal_volumes(lhi, oracle_mod):
    from liquidhairinteration_b200.net import LearnedNet
    params = random_params(oracle_mod.net_num_params(), seed=51)
    kept = LearnedNet(seed=7)
    kept.set_params(params)
    for i, shape in enumerate(SHAPES):
        r, t, s = net_case(shape, seed=52 + i)
        new = LearnedNet(seed=7)
        new.set_params(params)
        assert np.array_equal(kept.forward(r, t, s), new.forward(r, t, s)), shape
        new.close()
    kept.close()
