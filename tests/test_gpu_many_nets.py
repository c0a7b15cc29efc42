"""More networks in one engine than a warp moves on at once, at the sizes where the way changes,
against the oracle, bit for bit, with horizons that end at different steps."""
import numpy as np
import pytest

from netgen import random_net

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


@pytest.mark.parametrize("per_launch", [0, 5])
@pytest.mark.parametrize("mode", [0, 1], ids=["dense", "event"])
@pytest.mark.parametrize("count", [32, 33, 256, 257, 300])
def test_many_networks_match_the_oracle(nc, oracle_mod, count, mode, per_launch):
    if mode == 1 and per_launch:
        pytest.skip("the event form has no launch of several steps")
    nets = []
    for q in range(count):
        xyz, pre, post, w = random_net(1 + q % 9, 3 * (q % 7), 100 + q, duplicates=False)
        nets.append(dict(xyz=xyz, pre=pre, post=post, weight=w, horizon=3 + q % 5,
                         params=nc.default_params(seed=q, step_mode=mode, run_speed=[1.0, 0.5, 2.0][q % 3])))
    b = nc.Batch(nets)
    b.set_launch(steps_per_launch=per_launch)
    b.run(4)
    b.weights(0)  # a flush between them
    b.run_to_end()
    for q, d in enumerate(nets):
        o = oracle_mod.OracleS(d["xyz"], d["pre"], d["post"], d["weight"],
                               params=oracle_mod.default_params(seed=q, run_speed=float(d["params"].run_speed)))
        o.run(d["horizon"])
        st = b.stats(q)
        assert (st["steps"], st["fires"]) == (d["horizon"], o.stats()["fires"]), q
        assert np.array_equal(bits(b.potentials(q)), bits(o.potentials())), q
        assert np.array_equal(bits(b.weights(q)), bits(o.weights())), q
