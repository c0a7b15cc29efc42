"""The event form at the sizes where its warps take fewer neurons (8, 16 or 32 in the
neuron step, 1 to 8 in the spike launch), with tiles cut at odd remainders, against the
oracle, bit for bit."""
import numpy as np
import pytest

from netgen import random_net

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


@pytest.mark.parametrize("n,s,steps", [(1, 2, 80), (31, 400, 150), (9725, 60000, 40), (9733, 60000, 40),
                                       (19501, 90000, 30), (38925, 120000, 24)])
def test_event_rows_match_the_oracle(nc, oracle_mod, n, s, steps):
    xyz, pre, post, w = random_net(n, s, 40 + n % 7)
    groups = [dict(first=0, count=max(1, n // 3), rate_hz=150.0, correlated=0, jitter=0)]
    net = nc.NeuCor.from_arrays(xyz, pre, post, w, params=nc.default_params(seed=6, step_mode=1))
    net.set_input_groups(groups)
    o = oracle_mod.OracleS(xyz, pre, post, w, params=oracle_mod.default_params(seed=6), groups=groups)
    net.record_raster(steps)
    net.run(steps)
    assert np.array_equal(net.raster(), o.run(steps, raster=True)[0])
    assert np.array_equal(bits(net.weights()), bits(o.weights()))
    assert np.array_equal(bits(net.potentials()), bits(o.potentials()))
    st, so = net.stats(), o.stats()
    assert (st["fires"], st["launched"], st["dropped"]) == (so["fires"], so["launched"], so["dropped"])
    assert st["launched"] > 0 or n == 1
