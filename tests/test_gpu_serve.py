"""The served form on the GPU: jobs of different sizes, durations and
plasticity, arriving while others run, give each the raster (SHA-256 of its
spikes, step by step) and the synaptic event count it gives alone."""
import importlib

import pytest

from tests.conftest import package

pytestmark = pytest.mark.gpu
S = importlib.import_module(package().__name__ + ".serve")
nc = importlib.import_module(package().__name__ + ".netconfig")


def jobs():
    specs = [  # side, ms, arrival s, seed, stdp
        (1, 180, 0.0, 3, False), (2, 120, 0.0, 4, True), (3, 90, 0.05, 5, False),
        (1, 60, 0.1, 6, True), (2, 150, 0.2, 7, False), (4, 70, 0.2, 8, False),
    ]
    out = []
    for i, (side, ms, arr, seed, stdp) in enumerate(specs):
        cfg = nc.cortical_grid(side, side, total_ms=ms + 1, seed=seed, glob_h=side * side, stdp=stdp,
                               start_plasticity_ms=0, **({"p1": 0.0376} if side == 2 else {}))
        out.append(S.Job(job_id=i, cfg=cfg, duration_ms=ms, arrival_s=arr))
    return out


def test_each_result_is_the_same_alone_and_in_the_mix():
    served = S.Server(device=0, hbm_budget=150e9, max_slots=4, round_ms=16).run(jobs())
    alone = S.run_one_at_a_time(jobs(), device=0, read_ms=40)
    for a, b in zip(served, alone):
        assert not a.error and not b.error
        assert a.steps_done == b.steps_done == a.duration_ms
        assert a.raster_sha256 == b.raster_sha256 and a.spikes == b.spikes and a.events == b.events
        assert a.latency_s >= a.real_time_factor * a.duration_ms * 1e-3 > 0
    # more jobs than slots: some waited for a slot, and ran while others ran
    starts = sorted(j.t_start for j in served)
    dones = sorted(j.t_done for j in served)
    assert starts[-1] >= dones[0]
    assert any(x.t_start < y.t_done and y.t_start < x.t_done for x in served for y in served if x is not y)


def network(name):
    if name == "by_warps":
        return nc.cortical_grid(4, 4, glob_h=4, p1=0.01)
    if name == "plastic":
        return nc.cortical_grid(3, 3, glob_h=9, p1=0.02, stdp=True, start_plasticity_ms=0)
    if name == "fast_bath":
        return nc.cortical_grid(4, 4, n_exc_a=400, n_exc_b=400, n_inh=200, glob_h=1, p1=0.005, nu_ext_hz=6.0)
    if name == "long_rows":
        return nc.cortical_grid(1, 1, n_exc_a=700, n_exc_b=700, n_inh=500, p_intra=0.95)
    cfg = nc.cortical_grid(16, 16, n_exc_a=10, n_exc_b=10, n_inh=5, glob_h=256, p1=0.1)   # by_threads
    cfg.conn = {k: (J, 0.2, lo, hi, probs) for k, (J, _, lo, hi, probs) in cfg.conn.items()}
    return cfg


@pytest.mark.parametrize("name", ["by_warps", "by_threads", "plastic", "fast_bath", "long_rows"])
def test_footprint_covers_the_build(name):
    """What the device's pool held at its highest while the engine was built."""
    from cuda.bindings import driver, runtime
    E = importlib.import_module(package().__name__ + ".engine")
    cfg = network(name)
    E.Engine(nc.cortical_grid(1, 1, n_exc_a=10, n_exc_b=10, n_inh=5, p1=0.1), device=0).close()   # the device is set up
    err, pool = runtime.cudaDeviceGetDefaultMemPool(0)
    assert int(err) == 0
    attr = runtime.cudaMemPoolAttr
    err, others = runtime.cudaMemPoolGetAttribute(pool, attr.cudaMemPoolAttrUsedMemCurrent)
    assert int(err) == 0
    high = attr.cudaMemPoolAttrUsedMemHigh
    err, = runtime.cudaMemPoolSetAttribute(pool, high, driver.cuuint64_t(0))
    assert int(err) == 0
    eng = E.Engine(cfg, device=0)
    err, used = runtime.cudaMemPoolGetAttribute(pool, high)
    assert int(err) == 0
    used, held = int(used) - int(others), eng.device_bytes
    eng.close()
    estimate = S.estimate_device_bytes(cfg)
    assert held <= used <= estimate < 1.3 * used
