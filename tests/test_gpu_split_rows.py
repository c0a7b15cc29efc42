"""The dense step with rows of so many in-synapses that they are split over blocks, against the
oracle, bit for bit: runs just below and above the rule's size, several long rows in one run of 8,
in the first and the last one, sparse and full windows, whole step counters, batches in every
launch shape, and a served network, rows of even length and of one long one."""
import numpy as np
import pytest

from netgen import random_net

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


def long_rows(n, fans, extra, seed, negative=0.0):
    """Neuron j has fans[j] in-synapses from distinct sources; `extra` random ones besides."""
    rng = np.random.default_rng(seed)
    pre, post = [rng.integers(0, n, extra)], [rng.integers(0, n, extra)]
    for j, fan in fans.items():
        pre.append(rng.permutation(np.delete(np.arange(n), j))[:fan])
        post.append(np.full(fan, j))
    xyz = (rng.random((n, 3)) * 2).astype(np.float32)
    pre, post = np.concatenate(pre).astype(np.int32), np.concatenate(post).astype(np.int32)
    w = (rng.random(len(pre)) * 0.1).astype(np.float32)
    w[rng.random(len(w)) < negative] *= np.float32(-1.0)
    return xyz, pre, post, w


NETS = {
    "1536_quads": (lambda s: long_rows(6500, {3: 6144}, 0, 1, s), {}),
    "1537_quads": (lambda s: long_rows(6500, {3: 6145}, 0, 2, s), {}),
    "one_long_row": (lambda s: long_rows(7000, {1234: 6999}, 8000, 3, s), {}),
    "run_of_long_rows": (lambda s: long_rows(3000, {j: 1500 + 101 * (j - 16) for j in range(16, 24)}, 6000, 4, s), {}),
    "first_and_last": (lambda s: long_rows(6501, {0: 4000, 7: 3000, 6500: 6500}, 3000, 5, s), {}),
    "many": (lambda s: long_rows(6600, {j: 6400 for j in range(0, 6600, 597)}, 4000, 6, s), {}),
    "even_rows": (lambda s: long_rows(1397, {j: 1396 - j % 5 for j in range(1397)}, 0, 9, s), {}),
    "whole_counters": (lambda s: long_rows(6500, {5: 6499}, 3000, 7, s), dict(presynaptic_trace_decay=0.9995)),
    "half_step": (lambda s: long_rows(4000, {5: 3999, 6: 3000}, 3000, 8, s), dict(run_speed=0.5)),
}


def make_oracle(oracle_mod, net, pkw, groups):
    return oracle_mod.OracleS(*net, params=oracle_mod.default_params(**pkw), groups=groups)


@pytest.mark.parametrize("rate", [4.0, 400.0], ids=["sparse", "busy"])
@pytest.mark.parametrize("negative", [0.0, 0.2], ids=["positive", "negative"])
@pytest.mark.parametrize("name", NETS)
def test_split_rows_match_the_oracle(nc, oracle_mod, name, negative, rate):
    make, extra = NETS[name]
    net_arrays = make(negative)
    pkw = dict(seed=3, inhibitory_rule=1, **extra)
    groups = [dict(first=0, count=len(net_arrays[0]), rate_hz=rate, correlated=0, jitter=0)]
    net = nc.NeuCor.from_arrays(*net_arrays, params=nc.default_params(storage_order=1, **pkw))
    net.set_input_groups(groups)
    o = make_oracle(oracle_mod, net_arrays, pkw, groups)
    net.record_raster(50)
    rows = []
    for part in (1, 16, 33):  # a flush between them: the next step finds its plasticity done
        net.run(part)
        rows.append(o.run(part, raster=True)[0])
        assert np.array_equal(bits(net.weights()), bits(o.weights()))
        assert np.array_equal(bits(net.potentials()), bits(o.potentials()))
    assert np.array_equal(net.raster(), np.concatenate(rows))
    st, so = net.stats(), o.stats()
    assert (st["fires"], st["launched"], st["dropped"]) == (so["fires"], so["launched"], so["dropped"])


def mixed():
    return [long_rows(6500, {9: 6499}, 2000, 11, 0.2), random_net(40, 300, 12), long_rows(1500, {j: 1499 for j in range(7)}, 0, 13),
            random_net(700, 9000, 14)]


@pytest.mark.parametrize("blocks,threads,per_launch", [(0, 96, 0), (0, 256, 0), (3, 64, 0), (1, 96, 7), (0, 128, 5)])
def test_batches_with_split_rows(nc, oracle_mod, blocks, threads, per_launch):
    nets = []
    for q, (xyz, pre, post, w) in enumerate(mixed()):
        nets.append(dict(xyz=xyz, pre=pre, post=post, weight=w, horizon=40 + 9 * q,
                         groups=[dict(first=0, count=len(xyz), rate_hz=60.0, correlated=0, jitter=0)],
                         params=nc.default_params(seed=q, run_speed=[1.0, 0.5, 1.0, 2.0][q])))
    b = nc.Batch(nets)
    b.set_launch(neuron_block=threads, dense_blocks=blocks, steps_per_launch=per_launch)
    b.run_to_end()
    for q, d in enumerate(nets):
        o = oracle_mod.OracleS(d["xyz"], d["pre"], d["post"], d["weight"], groups=d["groups"],
                               params=oracle_mod.default_params(seed=q, run_speed=float(d["params"].run_speed)))
        o.run(d["horizon"])
        assert np.array_equal(bits(b.potentials(q)), bits(o.potentials())), q
        assert np.array_equal(bits(b.weights(q)), bits(o.weights())), q
        assert b.stats(q)["launched"] == o.stats()["launched"], q


def test_served_with_split_rows(nc, oracle_mod):
    server = nc.Server(1 << 28, max_networks=8, steps_per_batch=8, build_threads=2, keep_results=True)
    jobs = []
    for q, (xyz, pre, post, w) in enumerate(mixed() * 2):
        d = dict(xyz=xyz, pre=pre, post=post, weight=w, horizon=20 + 13 * q, params=nc.default_params(seed=q),
                 groups=[dict(first=0, count=len(xyz), rate_hz=60.0, correlated=0, jitter=0)])
        jobs.append((server.submit(d), d))
    server.drain()
    for rid, d in jobs:
        w, pot = server.fetch(rid)
        o = oracle_mod.OracleS(d["xyz"], d["pre"], d["post"], d["weight"], groups=d["groups"],
                               params=oracle_mod.default_params(seed=int(d["params"].seed)))
        o.run(d["horizon"])
        assert np.array_equal(bits(w), bits(o.weights()))
        assert np.array_equal(bits(pot), bits(o.potentials()))
    server.close()
