"""The work a user has the engine do, as cases that can be timed and compared.

Every case goes through the public entry points (``engine.Engine``,
``batch.BatchRunner``, ``serve.Server``).  A case's ``kind`` says what a pass
is:

* ``loop``       -- ``ms`` times one ``step(1)`` and the read of that step's
                    spikes: the real-time loop, and the bench's end-to-end form;
* ``round``      -- ``step(ms)``, then the spikes of those steps at once: a
                    simulation read back in rounds;
* ``stdp``       -- ``step(1000)`` with plasticity on, i.e. through one weight
                    update, then the weights and traces (the reference's
                    periodic synapse probe);
* ``sweep``      -- ``ms`` steps (a multiple of 80) of many networks as CUDA
                    graphs, then the last 80 steps' spikes of each;
* ``job``        -- a whole simulation: build, ``ms`` steps read back in
                    rounds of 40, final state, release;
* ``serve``      -- a stream of jobs through the server: build, step together,
                    digest, release;
* ``connectome`` -- build, then rank 0's synapse list and the bath parameters.

The networks are ``netconfig.cortical_grid``'s: cfx x cfy modules of n neurons
(two fifths + two fifths excitatory, the rest inhibitory), ``ranks`` emulated
reference ranks.  Passes on one state go on where the last one ended.

Spike and synapse lists come back whole, in arrays of one length per case: the
list, then zeros.
"""
import importlib
import math
import random

import numpy as np

E = importlib.import_module("201812realtimecortsim_b200.engine")
B = importlib.import_module("201812realtimecortsim_b200.batch")
S = importlib.import_module("201812realtimecortsim_b200.serve")
nc = importlib.import_module("201812realtimecortsim_b200.netconfig")

# steps a state has behind it before its first pass: past the onset burst and
# the silence after it, into the regime a long simulation spends its time in
SETTLED = 1000


def listed():
    return [
        # the smallest call: one module of the tests' size in a 1 ms loop
        dict(name="loop_1x1_n100", kind="loop", cfx=1, cfy=1, n=100, ranks=1, mu=0.6, ms=20),
        # a small ragged network with the reference Makefile's default delays
        dict(name="loop_3x5_n77_exp", kind="loop", cfx=3, cfy=5, n=77, ranks=5, mu=0.6, ms=10, exp=True),
        # a 2x2 grid on one rank, as the 2x2 benchmark has it
        dict(name="round_2x2_n400", kind="round", cfx=2, cfy=2, n=400, ranks=1, mu=0.42, ms=40),
        # a mid-size ragged grid: ranks of 2743 neurons
        dict(name="round_11x13_n211", kind="round", cfx=11, cfy=13, n=211, ranks=11, mu=0.5, ms=40),
        # the headline network of the bench (720 000 neurons, 192 ranks), read every ms
        dict(name="loop_24x24_n1250", kind="loop", cfx=24, cfy=24, n=1250, ranks=192, mu=0.3, ms=10),
        # weak adaptation: a network that stays busy, about eight events per neuron and ms
        dict(name="round_8x8_n250_busy", kind="round", cfx=8, cfy=8, n=250, ranks=64, mu=0.5, ms=40, g_c=0.2),
        # plasticity through a weight update, one rank
        dict(name="stdp_4x4_n150", kind="stdp", cfx=4, cfy=4, n=150, ranks=1, mu=0.5, ms=1000),
        # a parameter sweep stepped as graphs
        dict(name="sweep_16_n120", kind="sweep", count=16, n=120, mu=0.57, ms=80),
        # whole jobs: one module, and a grid over 12 ranks
        dict(name="job_1x1_n250", kind="job", cfx=1, cfy=1, n=250, ranks=1, mu=0.48, ms=200),
        dict(name="job_6x6_n150", kind="job", cfx=6, cfy=6, n=150, ranks=12, mu=0.5, ms=400),
        # a stream of small jobs, some with plasticity
        dict(name="serve_8_n100", kind="serve", count=8, n=100, mu=0.6, ms=300),
        # the connectome alone, read back as the reference dumps it
        dict(name="connectome_5x3_n150", kind="connectome", cfx=5, cfy=3, n=150, ranks=1, mu=0.5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop", "loop", "round", "round", "round", "stdp", "sweep", "job", "job", "serve", "connectome"])
    n = _log(rng, 50, 300 if kind in ("loop", "round") else 100 if kind in ("sweep", "serve") else 140)
    case = dict(kind=kind, n=n, mu=round(0.6 * min(1.0, (100 / n) ** 0.25), 4))
    if kind in ("sweep", "serve"):
        return dict(case, count=rng.randint(3, 16), ms=80 * rng.randint(1, 3) if kind == "sweep" else _log(rng, 60, 400))
    side = 6 if kind in ("stdp", "connectome") else 20
    cfx, cfy = _log(rng, 1, side), _log(rng, 1, side)
    mods = cfx * cfy
    # one reference rank simulates at most 32000 neurons
    ranks = rng.choice([p for p in range(1, mods + 1) if mods % p == 0 and mods // p * n <= 8000])
    case.update(cfx=cfx, cfy=cfy, ranks=ranks)
    if kind == "connectome":
        return dict(case, ranks=1, exp=rng.random() < 0.3)
    if kind == "stdp":
        return dict(case, ms=1000)
    case["ms"] = {"loop": lambda: rng.randint(4, 20), "round": lambda: rng.randint(20, 80), "job": lambda: _log(rng, 50, 600)}[kind]()
    if rng.random() < 0.3:
        case["exp"] = True
    if rng.random() < 0.25:
        case["g_c"] = round(rng.uniform(0.2, 1.0), 3)
    return case


def _network(case, rng, cfx, cfy, ranks, total_ms, stdp=False):
    """The case's network; the seed moves the global seed, the external rate
    and the adaptation strength (the sweep's parameters)."""
    n = case["n"]
    a = 2 * n // 5
    return nc.cortical_grid(
        cfx, cfy, n_exc_a=a, n_exc_b=a, n_inh=n - 2 * a, mu=case["mu"], g_c=case.get("g_c", 3.0),
        # the benchmark's lateral in-degree, at most the tests' probability on small modules
        p1=min(0.2, nc.lateral_p1_for_grid(cfx, cfy, neurons_per_module=n)),
        nu_ext_hz=3.0 * rng.uniform(0.95, 1.05), alpha_c=rng.uniform(0.9, 1.1), total_ms=total_ms,
        seed=rng.randrange(1, 1 << 30), glob_h=ranks, stdp=stdp, start_plasticity_ms=0,
        delay_exponential=bool(case.get("exp", False)), delay_range_subpop=True)


def _grids(case, rng):
    """The grid side of each network of a sweep or a stream."""
    sides = [1 + k % 4 for k in range(case["count"])]
    rng.shuffle(sides)
    return sides


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "sweep":
        cfgs = [_network(case, rng, g, g, g * g, 10 ** 8) for g in _grids(case, rng)]
        engines = B.build_all(cfgs)
        E.step_many(engines, 1)
        runner = B.BatchRunner(engines)
        runner.run(12 * B.GRAPH_STEPS)
        most = _most_spikes(case, sum(c.glob_n for c in cfgs), 80)
        return {"kind": kind, "ms": case["ms"], "engines": engines, "runner": runner, "spikes": most}
    if kind == "serve":
        nets = [_network(case, rng, g, g, g * g, case["ms"] + 1, stdp=k % 4 == 3)
                for k, g in enumerate(_grids(case, rng))]
        ms = [max(1, int(case["ms"] * rng.uniform(0.5, 1.0))) for _ in nets]
        return {"kind": kind, "nets": nets, "durations": ms}
    plastic = kind == "stdp"
    cfg = _network(case, rng, case["cfx"], case["cfy"], case["ranks"], 10 ** 8, stdp=plastic)
    state = {"kind": kind, "ms": case.get("ms", 0)}
    state["spikes"] = _most_spikes(case, cfg.glob_n, 80 if plastic else state["ms"])
    if kind in ("stdp", "connectome"):
        state["synapses"] = _most_synapses(cfg)
    if kind in ("job", "connectome"):
        return dict(state, cfg=cfg)
    eng = E.Engine(cfg)
    if not plastic:
        eng.step(SETTLED)
    eng.sync()
    return dict(state, eng=eng)


def _fixed(values, length):
    """The list in an array of the case's length."""
    out = np.zeros(length, values.dtype)
    k = min(len(values), length)
    out[:k] = values[:k]
    return out


def _most_spikes(case, neurons, ms):
    """More spikes than ``ms`` steps make: ten times the usual rate, and a
    quarter of the network at once."""
    return int(neurons * (0.25 + ms * (0.05 if case.get("g_c", 3.0) >= 1 else 0.25))) + 16


def _most_synapses(cfg):
    return int(1.1 * S.expected_synapses(cfg)) + 1000


def run(state):
    return {"loop": _loop, "round": _round, "stdp": _stdp, "sweep": _sweep, "job": _job, "serve": _serve,
            "connectome": _connectome}[state["kind"]](state)


def _loop(state):
    eng, ids, te = state["eng"], [], []
    for _ in range(state["ms"]):
        t = eng.time_ms
        eng.step(1)
        i, e = eng.spikes(t)
        ids.append(i)
        te.append(e)
    return _raster(state, np.concatenate(ids), np.concatenate(te), [len(i) for i in ids])


def _raster(state, ids, te, counts):
    return {"ids": _fixed(ids, state["spikes"]), "te": _fixed(te, state["spikes"]), "counts": np.array(counts)}


def _round(state):
    eng, n = state["eng"], state["ms"]
    t = eng.time_ms
    eng.step(n)
    ids, te, counts = eng.spikes_range(t, n)
    return dict(_raster(state, ids, te, counts), events=eng.events_delivered())


def _stdp(state):
    eng, n = state["eng"], state["ms"]
    eng.step(n)
    t = eng.time_ms
    ids, te, counts = eng.spikes_range(t - 80, 80)
    pre, post, delay, kind, w, td = eng.backward_synapses(0, with_tderiv=True)
    return dict(_raster(state, ids, te, counts), **_synapses(state, pre=pre, post=post, delay=delay, kind=kind, w=w, td=td))


def _synapses(state, **lists):
    return {k: _fixed(v, state["synapses"]) for k, v in lists.items()}


def _sweep(state):
    state["runner"].run(state["ms"])
    ids, te, counts = zip(*(e.spikes_range(e.time_ms - 80, 80) for e in state["engines"]))
    return _raster(state, np.concatenate(ids), np.concatenate(te), np.concatenate(counts))


def _job(state):
    eng, done, ids, te, counts = E.Engine(state["cfg"]), 0, [], [], []
    while done < state["ms"]:
        k = min(40, state["ms"] - done)
        eng.step(k)
        i, e, c = eng.spikes_range(done, k)
        ids.append(i)
        te.append(e)
        counts.append(c)
        done += k
    out = dict(_raster(state, np.concatenate(ids), np.concatenate(te), np.concatenate(counts)),
               events=eng.events_delivered(), **eng.state())
    eng.close()
    return out


def _serve(state):
    jobs = [S.Job(job_id=k, cfg=c, duration_ms=ms) for k, (c, ms) in enumerate(zip(state["nets"], state["durations"]))]
    S.Server(max_slots=6).run(jobs)
    digest = np.frombuffer(bytes.fromhex("".join(j.raster_sha256 for j in jobs)), np.uint8)
    return {"digest": digest.copy(), "events": np.array([j.events for j in jobs]),
            "spikes": np.array([j.spikes for j in jobs])}


def _connectome(state):
    eng = E.Engine(state["cfg"])
    pre, post, delay, kind, w = eng.backward_synapses(0)
    inv_nu, max_ext = eng.bath_params()
    eng.close()
    return dict(_synapses(state, pre=pre, post=post, delay=delay, kind=kind, w=w), inv_nu=inv_nu, max_ext=max_ext)


def _step_work(case, neurons, synapses, ms):
    """Bytes and operations of ``ms`` steps: the neurons' five fp64 variables
    in and out, 6 bytes per synapse of every spike, and about 30 operations
    per event.  Rates as these networks settle at: 5 Hz, 25 Hz with weak
    adaptation; 3 bath events per neuron and ms."""
    rate = 5e-3 if case.get("g_c", 3.0) >= 1 else 25e-3
    events = synapses * rate
    return {"bytes": ms * (80 * neurons + 6 * events + 12 * neurons * rate),
            "flops": ms * 30 * (events + 3 * neurons)}


def work(case):
    kind = case["kind"]
    if kind in ("sweep", "serve"):
        rng = random.Random(0)
        nets = [_network(case, rng, g, g, 1, 1) for g in _grids(case, rng)]
    else:
        nets = [_network(case, random.Random(0), case["cfx"], case["cfy"], 1, 1)]
    neurons, synapses = sum(c.glob_n for c in nets), sum(S.expected_synapses(c) for c in nets)
    ms = case.get("ms", 0)
    w = _step_work(case, neurons, synapses, 0.75 * ms if kind == "serve" else ms)
    if kind == "stdp":   # weights and traces once more, at the update and for the read
        w["bytes"] += 2 * 6 * synapses + 11 * synapses
    if kind in ("job", "serve", "connectome"):   # the connectome written, ten operations a synapse
        w["bytes"] += 6 * synapses + 42 * neurons
        w["flops"] += 10 * synapses
    if kind == "connectome":   # and read back
        w["bytes"] += (6 + 12) * synapses
    return w


def exact(case, seed):
    """None: the outputs are event lists of a chaotic network, whole numbers
    and times that follow from every earlier one; they are right when they
    are the same, and the tests pin them against the reference's."""
    return None
