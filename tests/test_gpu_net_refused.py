"""A network call whose grid does not fit the device's memory is refused
before anything of it is copied, holds no memory afterwards, and does not
fail the next call.

The grid's first layer alone (32 bytes a cell) is larger than the device, so
nothing is allocated either; the host arrays are never touched, so they stay
unmapped pages."""
import numpy as np
import pytest

from netcases import net_case, random_params

pytestmark = pytest.mark.gpu


def _refused(call, *args):
    from liquidhairinteration_b200 import _lib, abi
    with pytest.raises(_lib.LhiError) as e:
        call(*args)
    assert e.value.code == abi.LHI_E_OOM, e.value


def test_grid_beyond_the_device(lhi, oracle_mod):
    import torch
    from liquidhairinteration_b200.net import LearnedNet
    n = 64
    while 32 * n ** 3 <= torch.cuda.get_device_properties(0).total_memory:
        n += 64
    net = LearnedNet(seed=7)
    net.set_params(random_params(oracle_mod.net_num_params(), seed=61))
    r, t = np.zeros((n, n, n), np.float32), np.zeros((n, n, n), np.uint8)
    free = torch.cuda.mem_get_info(0)[0]
    for _ in range(2):
        _refused(net.forward, r, t)
        _refused(net.backward, r, t, None, r)
        assert torch.cuda.mem_get_info(0)[0] >= free - (64 << 20)
    net.close()


def test_next_call_after_a_refused_one(lhi, oracle_mod):
    from liquidhairinteration_b200.net import LearnedNet
    params = random_params(oracle_mod.net_num_params(), seed=62)
    net, new = LearnedNet(seed=7), LearnedNet(seed=7)
    net.set_params(params)
    new.set_params(params)
    r, t, s = net_case((16, 12, 20), seed=63)
    expected = new.forward(r, t, s)
    new.close()
    n = 2048  # 275 GB of first-layer activations
    _refused(net.forward, np.zeros((n, n, n), np.float32), np.zeros((n, n, n), np.uint8))
    assert np.array_equal(net.forward(r, t, s), expected)
    net.close()
