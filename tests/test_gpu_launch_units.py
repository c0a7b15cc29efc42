"""The spike launch with several units a warp, looked at a lane each: units on both sides of one
and of two rounds of 32, of one network and of several, and a network large enough to take that
way by itself, against the oracle, bit for bit."""
import numpy as np
import pytest

from netgen import random_net

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


def check(nc, oracle_mod, sizes, launch, steps):
    nets = []
    for q, n in enumerate(sizes):
        xyz, pre, post, w = random_net(n, 12 * n, 50 + q)
        nets.append(dict(xyz=xyz, pre=pre, post=post, weight=w, horizon=steps,
                         groups=[dict(first=0, count=n, rate_hz=60.0, correlated=0, jitter=0)],
                         params=nc.default_params(seed=q, step_mode=1)))
    b = nc.Batch(nets)
    b.set_launch(**launch)
    b.run_to_end()
    for q, d in enumerate(nets):
        o = oracle_mod.OracleS(d["xyz"], d["pre"], d["post"], d["weight"], groups=d["groups"],
                               params=oracle_mod.default_params(seed=q))
        o.run(steps)
        st, so = b.stats(q), o.stats()
        assert (st["fires"], st["launched"], st["dropped"]) == (so["fires"], so["launched"], so["dropped"]), q
        assert st["launched"] > 0
        assert np.array_equal(bits(b.weights(q)), bits(o.weights())), q
        assert np.array_equal(bits(b.potentials(q)), bits(o.potentials())), q


# one warp, one neuron a unit: 32 units to a tile of 32 neurons
@pytest.mark.parametrize("sizes", [(3,), (33,), (64,), (65,), (9, 40, 1, 30)])
def test_one_warp(nc, oracle_mod, sizes):
    check(nc, oracle_mod, sizes, dict(launch_blocks=1, launch_block=32), 60)


@pytest.mark.parametrize("blocks,threads", [(1, 96), (2, 64), (3, 32)])
def test_few_warps(nc, oracle_mod, blocks, threads):
    check(nc, oracle_mod, (500, 31, 129), dict(launch_blocks=blocks, launch_block=threads), 40)


@pytest.mark.parametrize("n", [155648, 155649, 330001])
def test_large_network(nc, oracle_mod, n):
    xyz, pre, post, w = random_net(n, 2 * n, 7)
    groups = [dict(first=0, count=n, rate_hz=20.0, correlated=0, jitter=0)]
    net = nc.NeuCor.from_arrays(xyz, pre, post, w, params=nc.default_params(seed=6, step_mode=1))
    net.set_input_groups(groups)
    o = oracle_mod.OracleS(xyz, pre, post, w, params=oracle_mod.default_params(seed=6), groups=groups)
    net.run(8)
    o.run(8)
    assert np.array_equal(bits(net.weights()), bits(o.weights()))
    assert np.array_equal(bits(net.potentials()), bits(o.potentials()))
    st, so = net.stats(), o.stats()
    assert (st["fires"], st["launched"], st["dropped"]) == (so["fires"], so["launched"], so["dropped"])
