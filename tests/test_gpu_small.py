"""The small networks' step (delivery with its compaction, update with its
sorts, tail) where its branches change, against the CPU restatement: light,
sorted, block-sorted and overflowing neurons (the bucket size moves the lines
between them), networks whose size is no multiple of a warp, with and without
plasticity, and the sizes on either side of the form's limits."""
import time

import numpy as np
import pytest

import dpsnn_oracle as O
from tests.conftest import engine_module, netconfig

pytestmark = pytest.mark.gpu
E = engine_module()
nc = netconfig()


def grid(cfx, cfy, n, ranks, **kw):
    a = 2 * n // 5
    kw.setdefault("p1", 0.1)
    return nc.cortical_grid(cfx, cfy, n_exc_a=a, n_exc_b=a, n_inh=n - 2 * a, glob_h=ranks, total_ms=100, seed=3,
                            delay_range_subpop=True, **kw)


CASES = {
    # an onset burst with hundreds of events per neuron and ms
    "burst": (lambda: grid(1, 1, 1250, 1, mu=0.3, g_c=0.2), 40),
    "ragged": (lambda: grid(3, 3, 77, 9, mu=0.6, g_c=0.3), 60),
    "plastic": (lambda: grid(3, 2, 85, 2, mu=0.6, g_c=0.3, stdp=True, start_plasticity_ms=0), 60),
}


@pytest.mark.parametrize("cap", [0, 64, 160])   # event slots per neuron: 1024, 64, 160
@pytest.mark.parametrize("name", sorted(CASES))
def test_small_step_matches_oracle(name, cap):
    make, steps = CASES[name]
    cfg = make()
    eng, orc = E.Engine(cfg, events_per_neuron=cap), O.OracleNet(cfg, 1)
    for t in range(steps):
        eng.step(1)
        ids, te = eng.spikes(t)
        oi, ot = orc.step()
        np.testing.assert_array_equal(ids, oi)
        np.testing.assert_array_equal(te, ot)
    st, so = eng.state(), orc.state()
    for k in st:
        np.testing.assert_array_equal(st[k], so[k], err_msg=k)
    eng.close()


# 30 x 17 modules of 32 neurons are half the form's limit less 64; one more
# row, or 2176 neurons per rank, change the rule; 32 x 32 are its limit and one
# more row is past it
@pytest.mark.parametrize("cfx, cfy, ranks", [(30, 17, 30), (30, 18, 30), (32, 17, 8), (32, 32, 32), (33, 32, 32)])
def test_forms_match_oracle(cfx, cfy, ranks):
    cfg = grid(cfx, cfy, 32, ranks, mu=0.8, g_c=0.5)
    eng, orc = E.Engine(cfg), O.OracleNet(cfg, 1)
    for t in range(30):
        eng.step(1)
        ids, te = eng.spikes(t)
        oi, ot = orc.step()
        np.testing.assert_array_equal(ids, oi)
        np.testing.assert_array_equal(te, ot)
    st, so = eng.state(), orc.state()
    for k in st:
        np.testing.assert_array_equal(st[k], so[k], err_msg=k)
    eng.close()


# requests below the smallest bucket (16) and odd ones are rounded; the burst in
# the small form, and the other form at its smallest network
@pytest.mark.parametrize("cap, slots", [(1, 16), (7, 16), (65, 66)])
@pytest.mark.parametrize("form", ["small", "large"])
def test_rounded_buckets_match_oracle(form, cap, slots):
    small = form == "small"
    cfg = CASES["burst"][0]() if small else grid(32, 17, 32, 8, mu=0.8, g_c=0.5)
    eng, even = E.Engine(cfg, events_per_neuron=cap), E.Engine(cfg, events_per_neuron=slots)
    assert eng.device_bytes == even.device_bytes
    even.close()
    orc = O.OracleNet(cfg, 1)
    for t in range(40 if small else 30):
        eng.step(1)
        ids, te = eng.spikes(t)
        oi, ot = orc.step()
        np.testing.assert_array_equal(ids, oi)
        np.testing.assert_array_equal(te, ot)
    st, so = eng.state(), orc.state()
    for k in st:
        np.testing.assert_array_equal(st[k], so[k], err_msg=k)
    eng.close()


def burst_seconds(cfg, steps, cap):
    best = np.inf
    for _ in range(3):
        eng = E.Engine(cfg, events_per_neuron=cap)
        eng.step(1)
        eng.sync()
        t = time.perf_counter()
        eng.step(steps)
        eng.sync()
        best = min(best, time.perf_counter() - t)
        eng.close()
    return best


# small buckets send most of a burst's neurons to the blocks' sort (with an
# overflow list to search): 5 times the default's time, 17 when it had a block
# per 32 neurons there too
def test_small_buckets_in_a_burst():
    cfg = CASES["burst"][0]()
    assert burst_seconds(cfg, 39, 64) < 11 * burst_seconds(cfg, 39, 0)


# so does a large in-degree with the default's buckets: as many blocks as buckets
# of nearly that size have, where a block per 32 neurons took twice the time
def test_large_in_degree_in_a_burst():
    cfg = grid(1, 1, 2000, 1, mu=0.3, g_c=0.2, p_intra=0.95)
    assert burst_seconds(cfg, 49, 0) < 1.5 * burst_seconds(cfg, 49, 1022)
