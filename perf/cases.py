"""The work users of the simulator have it do, as cases that can be timed and compared.

Six kinds of pass, each through the public Python binding of the C ABI:

  few      the reference's three-neuron STDP preset inside a render loop: one run() and the
           potentials and weights it draws, every frame;
  frame    the reference constructor's random sphere inside a render loop: the 16 steps of 1 ms
           of one 60 Hz frame, then what the frame draws;
  net      one network simulated for a stretch of its horizon, then its raster, its state and
           its weights read back;
  batch    several independent networks of uneven size advanced together;
  served   requests submitted to a server, all finished, each result fetched;
  request  one simulation request served from nothing: a network built on the device, run for
           its horizon, read back and dropped.

A pass continues the network where the last one left it, as a user's loop does.  Sizes are those of
the repository's workloads (1k x 50, 100k x 100, 2M x 200, mixes of 1k-64k and of 500-200k neurons
with fan-outs of 20-200) and odd sizes between them.
"""
import math

import numpy as np

import neurocorrelation_gb300 as G

FORMS = {"dense": G.NC_STEP_DENSE, "event": G.NC_STEP_EVENT, "auto": G.NC_STEP_AUTO}
DENSITY = 8.0  # the reference's spawn density, neurons per unit volume


def listed():
    return [
        # one frame of the three-neuron preset at its 0.02 ms step: the smallest call there is
        dict(name="few_frame", kind="few", n=3, dt=0.02, steps=1),
        # one frame of the sphere NeuCor(750) builds, a fifth of its synapses inhibitory
        dict(name="sphere_frame", kind="frame", n=750, dt=1.0, steps=16),
        # the 1k x 50 workload: correlated and control inputs, a second of simulated time
        dict(name="plain_1k", kind="net", n=1000, k=50, dt=1.0, steps=1000, form="dense", scale=1.0, inh=0.0, groups=2),
        # an odd mid-size network at half the step, so twice the fold window and longer delays
        dict(name="ragged_30k", kind="net", n=29989, k=73, dt=0.5, steps=200, form="dense", scale=1.0, inh=0.0, groups=5),
        # the 100k x 100 workload, a second of simulated time, saturated
        dict(name="plain_100k", kind="net", n=100000, k=100, dt=1.0, steps=1000, form="dense", scale=1.0, inh=0.0, groups=10),
        # the 2M x 200 workload, a prefix of its horizon (its weights are read once at the end of
        # 100,000 steps, so no pass reads them)
        dict(name="large_2m", kind="net", n=2000000, k=200, dt=1.0, steps=20, form="dense", scale=1.0, inh=0.0, groups=20),
        # inhibitory synapses: every arriving term is summed, in order
        dict(name="inhibitory_20k", kind="net", n=20000, k=100, dt=1.0, steps=200, form="dense", scale=1.0, inh=0.2, groups=4),
        # weak weights, activity near the inputs' own: the automatic choice settles on the event form
        dict(name="quiet_50k", kind="net", n=50000, k=80, dt=1.0, steps=512, form="auto", scale=0.05, inh=0.0, groups=8),
        # the event form pinned on a busy inhibitory network
        dict(name="event_8k", kind="net", n=8191, k=40, dt=1.0, steps=300, form="event", scale=1.0, inh=0.2, groups=3),
        # a mix of uneven networks in one engine
        dict(name="batch_12", kind="batch", n=8000, nets=12, dt=1.0, steps=256),
        # continuous batching of requests, built by the server's threads
        dict(name="served_12", kind="served", n=8000, nets=12, dt=1.0, steps=600),
        # one request from nothing to its results
        dict(name="request_20k", kind="request", n=20000, k=60, dt=1.0, steps=300),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "net", "net", "net", "net", "net", "batch", "request"])
    dt = rng.choice([0.25, 0.5, 1.0, 1.0, 1.0, 2.0])
    if kind == "frame":
        return dict(kind="frame", n=_log_int(rng, 30, 2000), dt=dt, steps=rng.randint(1, 32))
    if kind == "batch":
        return dict(kind="batch", n=_log_int(rng, 1500, 10000), nets=rng.randint(2, 16), dt=dt, steps=rng.randint(50, 400))
    if kind == "request":
        return dict(kind="request", n=_log_int(rng, 500, 60000), k=rng.randint(20, 150), dt=dt, steps=_log_int(rng, 100, 1000))
    form = rng.choice(["dense", "dense", "dense", "event", "auto"])
    inh = rng.choice([0.0, 0.0, 0.2])
    scale = rng.choice([1.0, 1.0, 0.05])
    on_device = form == "dense" and inh == 0.0 and scale == 1.0  # the others are laid out on the host
    n = _log_int(rng, 500, 400000 if on_device else 30000)
    k = rng.randint(20, min(200, n - 1))
    # at most the synapse updates of the largest listed case
    steps = max(8, min(1000, int(4e9 / (n * k)), _log_int(rng, 100, 1000)))
    return dict(kind="net", n=n, k=k, dt=dt, steps=steps, form=form, scale=scale, inh=inh, groups=rng.randint(1, 10))


# ------------------------------------------------------------------ networks
def _groups(case, n):
    """Correlated Poisson groups at 5-40 Hz on the first ids; of two, the second is the uncorrelated control."""
    size = max(1, min(20, n // (4 * case["groups"])))
    rates = np.linspace(5.0, 40.0, case["groups"]) if case["groups"] > 2 else [20.0] * case["groups"]
    return [dict(first=size * g, count=size, rate_hz=float(r), jitter=2, correlated=int(not (case["groups"] == 2 and g == 1)))
            for g, r in enumerate(rates)]


def _sphere(n, seed):
    """The reference constructor's network: uniform in a ball, every pair closer than 1 connected, weights
    U[0.2, 1) with a fifth of them negative.  Created in source order.  The places are the size's own, so
    that two seeds have as many synapses; the weights are the seed's."""
    rng = np.random.default_rng(n)
    radius = (n / (4.0 / 3.0 * math.pi * DENSITY)) ** (1.0 / 3.0)
    xyz = np.empty((0, 3))
    while len(xyz) < n:
        p = rng.uniform(-radius, radius, (2 * n + 8, 3))
        xyz = np.concatenate([xyz, p[(p * p).sum(1) <= radius * radius]])
    xyz = xyz[:n].astype(np.float32)
    d = np.sqrt(((xyz[:, None].astype(np.float64) - xyz[None]) ** 2).sum(-1))
    np.fill_diagonal(d, np.inf)
    pre, post = (a.astype(np.int32) for a in np.nonzero(d < 1.0))
    rng = np.random.default_rng(seed)
    w = rng.uniform(0.2, 1.0, len(pre)).astype(np.float32)
    w[rng.random(len(pre)) < 0.2] *= np.float32(-1.0)
    return xyz, pre, post, w


def _few(seed):
    """The three-neuron preset, its two weights and the rate of its inputs drawn from the seed."""
    rng = np.random.default_rng(seed)
    xyz = np.array([[0, 0, 0], [0.3, 0.3, 0], [0.3, -0.3, 0]], np.float32)
    w = rng.uniform(0.3, 0.7, 2).astype(np.float32)
    return xyz, np.zeros(2, np.int32), np.array([1, 2], np.int32), w, float(rng.uniform(15.0, 25.0))


def _mix(case, seed):
    """Sizes log-uniform between 500 or 1,000 neurons and the case's, fan-outs of 20-150 or 200, each
    with its own inputs and, when served, its own horizon.  The mix is the case's, its networks the seed's."""
    rng = np.random.default_rng(case["n"] + case["nets"])
    served = case["kind"] == "served"
    for q in range(case["nets"]):
        n = int(math.exp(rng.uniform(math.log(500 if served else 1000), math.log(case["n"]))))
        k = min(int(rng.integers(20, 151 if served else 201)), n - 1)
        groups = [dict(first=10 * g, count=10, rate_hz=float(rng.uniform(5.0, 50.0)), correlated=int(rng.integers(0, 2)),
                       jitter=int(rng.integers(0, 4))) for g in range(int(rng.integers(1, 9)))]
        horizon = int(math.exp(rng.uniform(math.log(case["steps"] / 6), math.log(case["steps"])))) if served else case["steps"]
        yield n, k, seed * 1009 + q, groups, horizon


def prepare(case, seed):
    kind, dt = case["kind"], case["dt"]
    if kind == "few":
        xyz, pre, post, w, rate = _few(seed)
        net = G.NeuCor.from_arrays(xyz, pre, post, w, params=G.default_params(seed=seed, run_speed=dt))
        net.setInputRateArray([rate] * 3, 3, xyz, [0.1] * 3)
        net.addInputOffset(1, 2.0)
        net.addInputOffset(2, -2.0)
        return dict(case=case, net=net)
    if kind == "frame":
        xyz, pre, post, w = _sphere(case["n"], seed)
        return dict(case=case, net=G.NeuCor.from_arrays(xyz, pre, post, w, params=G.default_params(seed=seed, run_speed=dt)))
    if kind == "net":
        n, k = case["n"], case["k"]
        params = G.default_params(seed=seed, run_speed=dt, step_mode=FORMS[case["form"]])
        if case["form"] == "dense" and case["scale"] == 1.0 and case["inh"] == 0.0:
            net = G.NeuCor.knn(n, k, DENSITY, seed=seed, params=params)
        else:
            xyz, pre, post, w = G.build_knn(n, k, DENSITY, seed=seed)
            w *= np.float32(case["scale"])
            w[np.random.default_rng(seed).random(len(w)) < case["inh"]] *= np.float32(-1.0)
            params.inhibitory_rule = 1  # the weight's sign
            net = G.NeuCor.from_arrays(xyz, pre, post, w, params=params)
        net.set_input_groups(_groups(case, n))
        return dict(case=case, net=net)
    if kind == "batch":
        nets = []
        for n, k, s, groups, _ in _mix(case, seed):
            xyz, pre, post, w = G.build_knn(n, k, DENSITY, seed=s)
            nets.append(dict(xyz=xyz, pre=pre, post=post, weight=w, groups=groups, params=G.default_params(seed=s, run_speed=dt)))
        return dict(case=case, batch=G.Batch(nets), nets=len(nets))
    if kind == "served":
        return dict(case=case, server=G.Server(2 << 30, max_networks=64, steps_per_batch=64, build_threads=8, keep_results=True),
                    requests=list(_mix(case, seed)))
    return dict(case=case, seed=seed)


def run(state):
    case = state["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "few":
        state["net"].run(steps)
        return dict(potact=state["net"].potAct, weights=state["net"].weights())
    if kind == "frame":
        net = state["net"]
        net.run(steps)
        return dict(potact=net.potAct, last_fire=net.lastFire(), weights=net.weights())
    if kind == "net":
        net = state["net"]
        net.record_raster(steps)
        net.run(steps)
        out = dict(raster=net.raster(), potact=net.potAct, last_fire=net.lastFire(), counts=np.array(list(net.stats().values())))
        if case["n"] * case["k"] <= 20_000_000:
            out["weights"] = net.weights()
        return out
    if kind == "batch":
        b = state["batch"]
        b.run(steps)
        return [dict(potentials=b.potentials(q), last_fire=b.lastFire(q), weights=b.weights(q)) for q in range(state["nets"])]
    if kind == "served":
        server = state["server"]
        ids = [server.submit_knn(n, k, DENSITY, s, horizon, params=G.default_params(seed=s, run_speed=case["dt"]), groups=groups)
               for n, k, s, groups, horizon in state["requests"]]
        server.drain()
        done = {d["request_id"]: d for d in server.poll()}
        return [[*server.fetch(i), np.array([done[i][f] for f in ("fires", "launched", "dropped", "steps")])] for i in ids]
    seed = state["seed"]
    net = G.NeuCor.knn(case["n"], case["k"], DENSITY, seed=seed, params=G.default_params(seed=seed, run_speed=case["dt"]))
    net.set_input_groups(_groups(dict(groups=4), case["n"]))
    net.run(steps)
    out = dict(weights=net.weights(), potentials=net.potentials(), counts=np.array(list(net.stats().values())))
    net.close()
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def _step_cost(n, synapses, dt, busy):
    """Bytes and operations of one step: 16 bytes a neuron, 14 a synaptic event.  A synapse launches again
    once its last spike is spent: every second refractory period of a saturated network."""
    kc = int(2.0 / dt) + 1
    events = synapses / (2.0 * kc) if busy else 0.002 * dt * synapses
    return 16.0 * n + 14.0 * events, 10.0 * n + 20.0 * events


def work(case):
    kind, dt, steps = case["kind"], case["dt"], case["steps"]
    if kind in ("few", "frame"):
        nets = [(case["n"], 2 if kind == "few" else 25 * case["n"], steps)]
    elif kind in ("net", "request"):
        nets = [(case["n"], case["n"] * case["k"], steps)]
    else:
        nets = [(n, n * k, h) for n, k, _, _, h in _mix(case, 1)]
    total = {"bytes": 0.0, "flops": 0.0}
    for n, s, h in nets:
        b, f = _step_cost(n, s, dt, case.get("scale", 1.0) == 1.0)
        total["bytes"] += h * b
        total["flops"] += h * f
        if kind == "net":
            total["bytes"] += h * n / 8  # the raster
        total["bytes"] += 12.0 * n + (4.0 * s if s <= 20_000_000 else 0.0)  # state and weights read back
    return total


# ------------------------------------------------------------------ 64 bits
def _philox(c0, c1, c2, seed):
    """Philox4x32-10, first two words of the draw of each counter (c0, c1, c2, 0)."""
    c = [np.asarray(v, np.uint64) * np.ones(len(c0), np.uint64) for v in (c0, c1, c2, 0)]
    k0, k1, low = seed & 0xffffffff, seed >> 32, np.uint64(0xffffffff)
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & low]
    return c[0], c[1]


def _simulate64(xyz, pre, post, w, inhibitory, dt, seed, steps):
    """The stepped model in 64 bits: potentials, activities, last fires (ms, NaN: none) and weights."""
    n, kc = len(xyz), int(2.0 / dt) + 1
    never = -(1 << 40)
    dist = np.sqrt(((xyz[pre].astype(np.float64) - xyz[post]) ** 2).sum(-1))
    delay = np.maximum(1, np.floor(dist * 2.0 / dt + 0.5)).astype(np.int64)
    after, before = (post > pre).astype(np.int64), post < pre
    lo, hi = np.where(inhibitory, -1.0, 0.0), np.where(inhibitory, 0.0, 1.0)
    w = w.astype(np.float64)
    leak, period = 0.5 ** dt, max(1, int(600.0 / dt))
    x = np.arange(kc) * dt
    ap = 100.0 * (np.exp(-(x - 1.0) ** 2 / (2 * 0.3 ** 2)) - np.exp(-(x - 2.16) ** 2 / (2 * 0.6 ** 2)) * 0.2) - 70.0 + 15.0 * np.maximum(1.0 - x, 0.0)
    pot, lf, firings = np.full(n, -70.0), np.full(n, never), np.zeros(n)
    la, seen, term = np.full(len(pre), never), np.full(len(pre), never), np.zeros(len(pre))

    def trace(decay, age):
        return np.where(age == 0, 0.0, decay ** (np.minimum(age, 1 << 20) * dt))

    def background(t):
        a, b = _philox(np.arange(n), t, 1, seed)
        forced = np.zeros(n, bool)
        forced[(b[a % np.uint64(period) == 0] % np.uint64(n)).astype(np.int64)] = True
        return forced

    forced = background(0)
    for t in range(1, steps + 1):
        arrives = (t - la >= 1) & (t - la <= kc)
        pot += np.bincount(post[arrives], term[arrives], n)
        pot = (pot + 70.0) * leak - 70.0
        fired = ((pot > -55.0) | forced) & (t - lf >= kc)
        lf[fired] = t
        firings += fired
        inside = t - lf < kc
        pot[inside] = ap[(t - lf)[inside]]
        forced = background(t)
        tf = fired[post]
        spiked = np.clip(w + 0.13 * trace(0.75, t - seen), lo, hi)
        launch = fired[pre] & (t - la >= kc + after)
        cap = np.where(tf & before, spiked, w)
        arrived = la == t
        w = np.where(tf, spiked, w)
        w = np.where(arrived, np.clip(w - 0.30 * trace(0.65, t - lf[post]), lo, hi), w)
        seen[arrived] = t
        term[launch] = dt * (0.2 * 52.0) * cap[launch] * 0.9943 * math.exp(0.3702 * dt)
        la[launch] = t + delay[launch]
    return pot, firings / (steps * dt / 10.0), np.where(lf == never, np.nan, lf * dt), w


def _kept_inhibitory(n, pre, w):
    """Synapse::inhibitory under the default rule: lost by the synapses that the growth of their source's
    vector copied (capacity 5, then doubled)."""
    out = np.zeros(len(w), bool)
    for i in range(n):
        mine = np.nonzero(pre == i)[0]
        for m, s in enumerate(mine):
            cap = 5
            while cap <= m:
                cap *= 2
            out[s] = w[s] < 0 and len(mine) <= cap
    return out


def exact(case, seed):
    # The frames are simulated from rest for a few steps.  Elsewhere a rounding decides a spike somewhere in
    # the thousands of steps and the spikes decide all that follows, so 64 bits say nothing about a pass: the
    # rasters and counts there are whole numbers, and those stay equal.
    if case["kind"] == "few":
        xyz, pre, post, w, _ = _few(seed)  # the inputs' first fire comes after 37 ms
    elif case["kind"] == "frame" and case["n"] <= 1000:
        xyz, pre, post, w = _sphere(case["n"], seed)
    else:
        return None
    pot, act, last, weights = _simulate64(xyz, pre, post, w, _kept_inhibitory(len(xyz), pre, w), case["dt"], seed, case["steps"])
    out = dict(potact=np.stack([pot, act], 1).reshape(-1), weights=weights)
    if case["kind"] == "frame":
        out["last_fire"] = last
    return out
