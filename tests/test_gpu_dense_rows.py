"""The dense step's row layout at its edges, against the oracle, bit for bit: rows whose
window bits do not fit in shared memory, tiles and blocks cut at every remainder, empty
rows, networks that keep whole step counters (a long trace, a long fold window), ages set
back on synapses idle for more than 2^15 and 2^16 steps, and in-flight synapses across
flushes and form switches."""
import numpy as np
import pytest

from netgen import knn_net, random_net

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


def hub_net(n, extra, seed):
    """Every neuron drives neuron 5 (a row of n - 1 synapses); `extra` random synapses."""
    rng = np.random.default_rng(seed)
    xyz = (rng.random((n, 3)) * 2).astype(np.float32)
    pre = np.concatenate([np.delete(np.arange(n), 5), rng.integers(0, n, extra)]).astype(np.int32)
    post = np.concatenate([np.full(n - 1, 5), rng.integers(0, n, extra)]).astype(np.int32)
    return xyz, pre, post, (rng.random(len(pre)) * 0.3).astype(np.float32)


def one_target(n, seed):
    """Only the last neuron has in-synapses: every other row is empty."""
    xyz, pre, post, w = random_net(n, 5 * n, seed, inhibitory=0.0)
    return xyz, pre, np.full_like(post, n - 1), w


NETS = {
    "n1": (lambda: random_net(1, 3, 1), {}, 120),
    "n8_one_row_each": (lambda: random_net(8, 8, 2), {}, 200),
    "n9": (lambda: random_net(9, 60, 3), {}, 200),
    "n33_remainders": (lambda: random_net(33, 333, 4, inhibitory=0.0), {}, 200),
    "empty_rows": (lambda: one_target(70, 5), {}, 200),
    "hub_row": (lambda: hub_net(9001, 20000, 6), {}, 60),
    "hub_row_inhibitory": (lambda: (lambda x, a, b, w: (x, a, b, np.where(np.arange(len(w)) % 7 == 0, -w, w)))(
        *hub_net(8500, 9000, 7)), {}, 40),
    "long_trace": (lambda: knn_net(300, 10, 8), dict(presynaptic_trace_decay=0.9995), 300),
    "long_window": (lambda: knn_net(60, 6, 9, inhibitory=0.2), dict(run_speed=0.0005), 300),
    "delays_of_thousands": (lambda: (lambda x, a, b, w: (x * 900, a, b, w))(*random_net(200, 3000, 10)), {}, 900),
}


@pytest.mark.parametrize("mode", [0, 2], ids=["dense", "auto"])
@pytest.mark.parametrize("name", NETS)
def test_rows_match_the_oracle(nc, oracle_mod, name, mode):
    make, pkw, steps = NETS[name]
    xyz, pre, post, w = make()
    n = len(xyz)
    groups = [dict(first=0, count=min(n, 40), rate_hz=60.0 / pkw.get("run_speed", 1.0), correlated=1, jitter=1)]
    net = nc.NeuCor.from_arrays(xyz, pre, post, w, params=nc.default_params(seed=5, step_mode=mode, **pkw))
    o = oracle_mod.OracleS(xyz, pre, post, w, params=oracle_mod.default_params(seed=5, **pkw), groups=groups)
    net.set_input_groups(groups)
    net.record_raster(steps)
    rows = []
    part = max(1, steps // 7)
    for k in range(0, steps, part):
        m = min(part, steps - k)
        net.run(m)
        rows.append(o.run(m, raster=True)[0])
        assert np.array_equal(bits(net.weights()), bits(o.weights()))  # a flush with spikes in flight
        if mode == 2:  # the other form for the next part
            net.set_step_form(1 - net.step_form)
    assert np.array_equal(net.raster(), np.concatenate(rows))
    assert np.array_equal(bits(net.potentials()), bits(o.potentials()))
    st, so = net.stats(), o.stats()
    assert (st["fires"], st["launched"], st["dropped"]) == (so["fires"], so["launched"], so["dropped"])


def test_synapses_idle_past_sixteen_bits(nc, oracle_mod):
    """No input but a few forced fires, tens of thousands of steps apart."""
    xyz, pre, post, w = random_net(24, 200, 11)
    pkw = dict(seed=12, background_firing=0)
    net = nc.NeuCor.from_arrays(xyz, pre, post, w, params=nc.default_params(**pkw))
    o = oracle_mod.OracleS(xyz, pre, post, w, params=oracle_mod.default_params(**pkw))
    for gap in (3, 1020, 28900, 2100, 1, 33000, 65536, 4096):
        ids = [gap % 24, (gap * 7) % 24]
        net.schedule_fire(ids)
        o.schedule_fire(ids)
        net.run(gap)
        o.run(gap)
        assert np.array_equal(bits(net.weights()), bits(o.weights())), gap
        assert np.array_equal(bits(net.potentials()), bits(o.potentials())), gap
    assert net.stats()["launched"] == o.stats()["launched"] > 0


@pytest.mark.parametrize("blocks,threads,per_launch", [(0, 32, 0), (0, 256, 0), (3, 96, 0), (1, 64, 7), (0, 224, 5)])
def test_batches_cut_into_any_blocks(nc, oracle_mod, blocks, threads, per_launch):
    nets = []
    for q, (n, s) in enumerate([(1, 2), (40, 300), (131, 2500), (7, 0), (64, 64)]):
        xyz, pre, post, w = random_net(n, s, 20 + q)
        nets.append(dict(xyz=xyz, pre=pre, post=post, weight=w, horizon=60 + 17 * q,
                         params=nc.default_params(seed=q, run_speed=[1.0, 0.5, 1.0, 2.0, 0.0005][q])))
    b = nc.Batch(nets)
    b.set_launch(neuron_block=threads, dense_blocks=blocks, steps_per_launch=per_launch)
    b.run_to_end()
    for q, d in enumerate(nets):
        p = d["params"]
        o = oracle_mod.OracleS(d["xyz"], d["pre"], d["post"], d["weight"],
                               params=oracle_mod.default_params(seed=int(p.seed), run_speed=float(p.run_speed)))
        o.run(d["horizon"])
        assert np.array_equal(bits(b.potentials(q)), bits(o.potentials())), q
        assert np.array_equal(bits(b.weights(q)), bits(o.weights())), q
        assert b.stats(q)["launched"] == o.stats()["launched"], q


@pytest.mark.parametrize("how", ["built on the device", "served"])
def test_whole_step_counters_elsewhere(nc, oracle_mod, how):
    """A trace too long for 16-bit ages in a device-built network and in a served one."""
    n, k, steps = 500, 12, 200
    pkw = dict(seed=3, presynaptic_trace_decay=0.9995)
    xyz, pre, post, w = nc.build_knn(n, k, 8.0, seed=9)
    groups = [dict(first=0, count=30, rate_hz=50.0, correlated=1, jitter=2)]
    o = oracle_mod.OracleS(xyz, pre, post, w, params=oracle_mod.default_params(**pkw), groups=groups)
    o.run(steps)
    if how == "served":
        server = nc.Server(1 << 28, max_networks=32, steps_per_batch=16, build_threads=2, keep_results=True)
        rid = server.submit_knn(n, k, 8.0, 9, steps, params=nc.default_params(**pkw), groups=groups)
        server.drain()
        weights, potentials = server.fetch(rid)
        server.close()
    else:
        net = nc.NeuCor.knn(n, k, 8.0, seed=9, params=nc.default_params(**pkw))
        net.set_input_groups(groups)
        net.run(steps)
        weights, potentials = net.weights(), net.potentials()
        assert np.array_equal(net.delays(), o.delays())
    assert np.array_equal(bits(weights), bits(o.weights()))
    assert np.array_equal(bits(potentials), bits(o.potentials()))
