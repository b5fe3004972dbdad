"""The Poisson bath kernel at the sizes and rates where its rounds, segments
and caps have edges, against the CPU restatement: nextBath (the sum of every
lapse drawn) and the raster must be the same bits."""
import os

import numpy as np
import pytest

import dpsnn_oracle as O
from tests.conftest import engine_module, netconfig

pytestmark = pytest.mark.gpu
E = engine_module()
nc = netconfig()


@pytest.mark.parametrize("n_exc, n_inh, ranks", [
    (26, 13, 4),    # ranks of 65 neurons: segments of 16 and one neuron
    (51, 26, 4),    # 128: one round of 8 full segments
    (51, 27, 4),    # 129: a round and one neuron
    (130, 41, 1),   # 1204: several rounds, a ragged end
])
# mean events per ms; the cap is ceil(20 * rate): 0.01 and 0.06 reach it (1 and
# 2 events, then single draws that shift the pairs), 6.05 is the largest
# supported (121)
@pytest.mark.parametrize("rate", [0.01, 0.06, 0.5, 3.0, 6.05])
def test_next_bath_and_raster_match_oracle(n_exc, n_inh, ranks, rate):
    cfg = nc.cortical_grid(2, 2, n_exc_a=n_exc, n_exc_b=n_exc, n_inh=n_inh, p1=0.2, mu=0.6, nu_ext_hz=rate,
                           total_ms=40, seed=5, glob_h=ranks)
    eng, orc = E.Engine(cfg), O.OracleNet(cfg, 1)
    for t in range(40):
        eng.step(1)
        ids, te = eng.spikes(t)
        oi, ot = orc.step()
        np.testing.assert_array_equal(ids, oi)
        np.testing.assert_array_equal(te, ot)
    st, so = eng.state(), orc.state()
    for k in st:
        np.testing.assert_array_equal(st[k], so[k], err_msg=k)
    eng.close()


# caps below the sixteen events a mapper counts (rates below 0.75) are decided by
# the mappers too: fewer events take no longer, where a walk neuron by neuron took
# five times as long
def test_low_rates_cost_no_more():
    def bath_seconds(rate):
        cfg = nc.cortical_grid(1, 1, n_exc_a=640, n_exc_b=640, n_inh=320, p1=0.01, p_intra=0.02, mu=0.001,
                               nu_ext_hz=rate, total_ms=1000, seed=7)
        eng = E.Engine(cfg)
        eng.step(50)
        eng.sync()
        eng.set_timing(True)
        best = np.inf
        for _ in range(5):
            before = eng.kernel_times()[0][2]
            eng.step(50)
            eng.sync()
            best = min(best, eng.kernel_times()[0][2] - before)
        eng.close()
        return best

    at_3 = bath_seconds(3.0)
    for rate in (0.06, 0.25, 0.7):
        assert bath_seconds(rate) < 1.3 * at_3


# a rate of zero makes the interval infinite and the cap 0: the reference's loop
# still makes one event, which has no slot; refused, as a cap that is exceeded is
def test_rate_of_zero_is_refused():
    cfg = nc.cortical_grid(1, 1, n_exc_a=20, n_exc_b=20, n_inh=10, p1=0.2, mu=0.6, total_ms=10, seed=5)
    cfg.subpops[2].NuExt = 0.0
    eng = E.Engine(cfg)
    inv, cap = eng.bath_params()
    assert np.isinf(inv[40:]).all() and not cap[40:].any() and cap[:40].all()
    eng.step(2)
    with pytest.raises(E.EngineError, match="bath"):
        eng.sync()
    with pytest.raises(E.EngineError, match="bath"):
        eng.spikes(1)
    eng.close()


# a network's bath events hold no more memory than 9 bytes per event slot in two
# buffers did, a slot for every event that the neurons' caps allow
def test_events_hold_what_a_step_needs():
    def held(rate):
        cfg = nc.cortical_grid(4, 4, total_ms=10, seed=5, glob_h=16, p1=0.01, p_intra=0.02, nu_ext_hz=rate)
        eng = E.Engine(cfg)
        b, caps = eng.device_bytes, int(eng.bath_params()[1].astype(np.int64).sum())
        eng.close()
        return b, caps

    (low, low_caps), (high, high_caps) = held(0.5), held(5.0)
    assert high - low < 2 * 9 * (high_caps - low_caps)


def fixup_table():
    raw = np.fromfile(os.path.join(E.HERE, "logf_fixup.bin"), np.uint32)
    return raw[1:1 + raw[0]], raw[1 + raw[0]:1 + 2 * raw[0]]


# a table may hold any value: one that is not a neighbouring float (here of an
# input below 1e-9, which no draw makes) has the kernel search the table, with
# the same results; values moved by three floats are the ones that it uses
@pytest.mark.parametrize("moved", [False, True])
def test_fixup_table_of_another_library(moved, tmp_path, monkeypatch):
    keys, vals = fixup_table()
    vals = vals + np.uint32(3) if moved else vals
    first = np.array([0x30000001], np.uint32)
    path = tmp_path / "logf_fixup.bin"
    np.concatenate([np.array([len(keys) + 1], np.uint32), first, keys, np.array([0xC1A00000], np.uint32),
                    vals]).tofile(path)
    monkeypatch.setenv("DPSNN_LOGF_FIXUP", str(path))
    cfg = nc.cortical_grid(2, 2, n_exc_a=130, n_exc_b=130, n_inh=41, p1=0.02, p_intra=0.02, mu=0.001, nu_ext_hz=3.0,
                           total_ms=60, seed=5)
    eng, orc = E.Engine(cfg), O.OracleNet(cfg, 1)
    eng.step(60)
    for _ in range(60):
        orc.step()
    got, want = eng.state()["nb"], orc.state()["nb"]
    eng.close()
    if moved:
        assert np.any(got != want)
        np.testing.assert_allclose(got, want, rtol=1e-7)   # three floats of a few lapses
    else:
        np.testing.assert_array_equal(got, want)
