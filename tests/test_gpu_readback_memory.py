"""A read-back allocates no device memory, the first one of a network neither."""
import numpy as np
import pytest

from netgen import random_net

pytestmark = pytest.mark.gpu


def free_bytes():
    torch = pytest.importorskip("torch")
    return torch.cuda.mem_get_info(0)[0]


def read_all(net):
    return [net.weights(), net.potentials(), net.potAct, net.lastFire(), net.stats(), net.delays(), net.inhibitory(), net.raster()]


def make(nc, mode, device_built):
    if device_built:
        return nc.NeuCor.knn(30000, 80, 8.0, seed=2, params=nc.default_params(seed=2, step_mode=mode))
    xyz, pre, post, w = random_net(30000, 2400000, 3)
    return nc.NeuCor.from_arrays(xyz, pre, post, w, params=nc.default_params(seed=2, step_mode=mode))


@pytest.mark.parametrize("mode,device_built", [(0, False), (1, False), (2, False), (0, True)],
                         ids=["dense", "event", "auto", "device-built"])
def test_reads_hold_no_memory(nc, mode, device_built):
    for first in (True, False):  # (a network before it loads the kernels)
        net = make(nc, mode, device_built)
        net.record_raster(8)
        net.run(8)
        net.sync()
        before = free_bytes()
        out = read_all(net)
        after = free_bytes()
        assert np.isfinite(out[1]).all()
        net.close()
    assert after >= before  # (host tables of a device-built network give some back)


def test_batch_reads_hold_no_memory(nc):
    for first in (True, False):
        nets = []
        for q in range(3):
            xyz, pre, post, w = random_net(20000, 1500000, q)
            nets.append(dict(xyz=xyz, pre=pre, post=post, weight=w, horizon=100, params=nc.default_params(seed=q)))
        b = nc.Batch(nets)
        b.run(8)
        b.potentials(0)
        before = free_bytes()
        for q in range(3):
            b.weights(q), b.lastFire(q), b.stats(q)
        after = free_bytes()
        b.close()
    assert after == before
