"""The network's host entry points keep their device copies between calls: a
call gives the same bits on a network that has seen other grids -- larger,
smaller, with and without solid flags -- as on a new one."""
import numpy as np
import pytest

from netcases import net_case, random_params

pytestmark = pytest.mark.gpu

CALLS = [((16, 16, 16), True), ((24, 20, 36), True), ((9, 6, 10), True), ((24, 20, 36), False), ((8, 8, 8), True)]


def test_calls_do_not_see_earlier_ones(lhi, oracle_mod):
    from liquidhairinteration_b200.net import LearnedNet
    params = random_params(oracle_mod.net_num_params(), seed=41)
    kept = LearnedNet(seed=7)
    kept.set_params(params)
    for i, (shape, with_solid) in enumerate(CALLS):
        r, t, s = net_case(shape, seed=42 + i)
        s = s if with_solid else None
        dz = np.random.default_rng(43 + i).standard_normal(shape).astype(np.float32)
        new = LearnedNet(seed=7)
        new.set_params(params)
        assert np.array_equal(kept.forward(r, t, s), new.forward(r, t, s)), (shape, with_solid)
        # the gradient's sums meet in atomic additions: equal to their rounding
        a, b = kept.backward(r, t, s, dz), new.backward(r, t, s, dz)
        new.close()
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b), (shape, with_solid)
    kept.close()
