"""The dense step with its charges staged in shared memory (networks with inhibitory synapses,
a tile to a block) at the edges of that rule, against the oracle, bit for bit: tiles of just
as many quads as fit and of one more, one row or eight, sparse windows and full ones, and whole
step counters."""
import numpy as np
import pytest

from netgen import random_net

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


def heavy_tile(fans, n, seed):
    """Neurons 0 .. 7 have `fans` in-synapses, from distinct sources; each drives others."""
    rng = np.random.default_rng(seed)
    pre, post = [], []
    for j, fan in enumerate(fans):
        pre.append(np.sort(rng.permutation(np.delete(np.arange(n), j))[:fan]))
        post.append(np.full(fan, j))
    pre, post = np.concatenate(pre).astype(np.int32), np.concatenate(post).astype(np.int32)
    xyz = (rng.random((n, 3)) * 2).astype(np.float32)
    w = rng.random(len(pre)).astype(np.float32)
    w[rng.random(len(w)) < 0.3] *= np.float32(-1.0)
    return xyz, pre, post, w


NETS = {  # quads of the heavy tile: rows end on 4 positions, the eighth on 32
    "640_quads": (lambda: heavy_tile([320] * 8, 400, 1), {}),
    "641_quads": (lambda: heavy_tile([321] + [320] * 7, 400, 2), {}),
    "one_row": (lambda: heavy_tile([391] + [0] * 6 + [1], 400, 3), {}),
    "odd_rows": (lambda: heavy_tile([1, 2, 3, 5, 31, 33, 63, 65], 100, 4), {}),
    "whole_counters": (lambda: heavy_tile([200] * 8, 300, 5), dict(presynaptic_trace_decay=0.9995)),
    "half_step": (lambda: random_net(90, 2000, 6), dict(run_speed=0.5)),
    "three_neurons": (lambda: random_net(3, 6, 7), dict(run_speed=0.02)),
}


@pytest.mark.parametrize("name", NETS)
@pytest.mark.parametrize("fire", [10.0, 500.0], ids=["sparse", "busy"])
def test_staged_sums_match_the_oracle(nc, oracle_mod, name, fire):
    make, extra = NETS[name]
    xyz, pre, post, w = make()
    pkw = dict(seed=3, inhibitory_rule=1, **extra)
    groups = [dict(first=0, count=min(len(xyz), 400), rate_hz=fire, correlated=0, jitter=0)]
    net = nc.NeuCor.from_arrays(xyz, pre, post, w.astype(np.float32), params=nc.default_params(storage_order=1, **pkw))
    net.set_input_groups(groups)
    o = oracle_mod.OracleS(xyz, pre, post, w.astype(np.float32), params=oracle_mod.default_params(**pkw), groups=groups)
    steps = 60
    net.record_raster(steps)
    rows = []
    for part in (1, 20, 39):  # a flush between them: the next step finds its plasticity done
        net.run(part)
        rows.append(o.run(part, raster=True)[0])
        assert np.array_equal(bits(net.weights()), bits(o.weights()))
        assert np.array_equal(bits(net.potentials()), bits(o.potentials()))
    assert np.array_equal(net.raster(), np.concatenate(rows))
    assert net.stats()["fires"] == o.stats()["fires"]
