"""Spike lists read back: one step, several at once (packed by one kernel, or
copied when they are longer than its buffer), across the ring's end, and by
threads at the same time."""
import ctypes as C
import threading

import numpy as np
import pytest

from tests.conftest import engine_module, netconfig

pytestmark = pytest.mark.gpu
E = engine_module()
nc = netconfig()


def network(n, **kw):
    a = 2 * n // 5
    return nc.cortical_grid(1, 1, n_exc_a=a, n_exc_b=a, n_inh=n - 2 * a, p1=0.1, total_ms=300, seed=11, **kw)


# a network's buffer holds 4 spikes per neuron, 1024 at least
CASES = {
    "quiet": (lambda: network(200, mu=0.5), True),
    "busy": (lambda: network(1250, mu=0.3, g_c=0.05), False),   # a list in most steps
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_ranges_are_the_steps_read_one_by_one(name):
    make, packed = CASES[name]
    eng = E.Engine(make())
    eng.step(30)
    one = [eng.spikes(t) for t in range(30)]
    for t in range(30, 133):   # the ring's end lies inside the last 80 steps
        eng.step(1)
        one.append(eng.spikes(t))
    total = sum(len(i) for i, _ in one[53:])
    assert total > 0 and (total <= max(1024, 4 * eng.glob_n)) == packed
    for t0, n in ((53, 80), (53, 1), (79, 2), (80, 53), (100, 0), (60, 71)):
        ids, te, counts = eng.spikes_range(t0, n)
        np.testing.assert_array_equal(counts, [len(i) for i, _ in one[t0:t0 + n]])
        np.testing.assert_array_equal(ids, np.concatenate([np.empty(0, np.uint32)] + [i for i, _ in one[t0:t0 + n]]))
        np.testing.assert_array_equal(te, np.concatenate([np.empty(0)] + [t for _, t in one[t0:t0 + n]]))
    with pytest.raises(E.EngineError, match="not among the last"):
        eng.spikes_range(52, 80)
    eng.close()


def test_threads_read_one_engine():
    eng = E.Engine(network(400, mu=0.5, g_c=0.3))
    eng.step(80)
    want = {(t0, n): eng.spikes_range(t0, n) for t0, n in ((0, 40), (40, 40), (10, 7), (77, 1))}
    wrong = []

    def read(t0, n):
        ids, te = np.empty(400 * n, np.uint32), np.empty(400 * n)
        counts = np.empty(n, np.uint32)
        lists = [a.ctypes.data_as(C.c_void_p) for a in (ids, te)]
        for _ in range(300):
            rc = eng._L.dpsnn_spikes_range(eng._h, t0, n, *lists, 400 * n, counts.ctypes.data_as(C.c_void_p))
            k = int(counts.sum())
            got = (ids[:k], te[:k], counts)
            if rc or any(not np.array_equal(a, b) for a, b in zip(got, want[t0, n])):
                wrong.append((t0, n))

    threads = [threading.Thread(target=read, args=k) for k in want]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not wrong
    eng.close()
