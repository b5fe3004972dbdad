"""The connectome build where its two forms and their steps have edges,
against the CPU restatement: every rank's synapse list (order, delays,
weights) and the external bath parameters."""
import numpy as np
import pytest

import dpsnn_oracle as O
from tests.conftest import engine_module, netconfig

pytestmark = pytest.mark.gpu
E = engine_module()
nc = netconfig()


def grid(cfx, cfy, a, b, i, ranks=1, dj=None, mean=None, **kw):
    kw.setdefault("mu", 0.3)
    cfg = nc.cortical_grid(cfx, cfy, n_exc_a=a, n_exc_b=b, n_inh=i, glob_h=ranks, total_ms=10, seed=9,
                           delay_range_subpop=True, **kw)
    if dj is not None:
        cfg.conn = {k: (J, dj, d0, d1, p) for k, (J, _, d0, d1, p) in cfg.conn.items()}
    if mean is not None:
        cfg.conn = {k: (mean, d, d0, d1, p) for k, (_, d, d0, d1, p) in cfg.conn.items()}
    return cfg


CASES = {
    # several modules per rank: NormDev's cached value crosses modules
    "cache_across_modules": lambda: grid(3, 4, 31, 30, 17, ranks=2, p1=0.2),
    "exponential_delays": lambda: grid(3, 2, 41, 23, 12, ranks=3, p1=0.15, delay_exponential=True),
    # every target taken; rows that end with the sub-population's last neuron
    "all_connected": lambda: grid(2, 2, 33, 32, 16, ranks=4, p_intra=1.0, p1=0.5),
    # rows of no or few targets, draws far in a table's tail
    "sparse": lambda: grid(3, 3, 130, 70, 40, ranks=1, p_intra=0.05, p1=0.002),
    # more synapses per neuron than the shared lists hold
    "long_rows": lambda: grid(1, 1, 700, 700, 500, p_intra=0.95),
    # weights far from their mean are drawn again: the thread form
    "rejected_weights": lambda: grid(2, 2, 40, 37, 20, ranks=2, p1=0.2, dj=0.6, mu=0.2),
    # means of five denormal units: a spread of 0.111 rounds to one unit, 0.2 of
    # the mean, and some weights are drawn again (all of them are stored as 0)
    "denormal_mean": lambda: grid(1, 1, 500, 500, 250, p_intra=0.95, dj=0.111, mean=7e-45),
    # one value per weight
    "no_spread": lambda: grid(2, 1, 40, 37, 20, ranks=1, p1=0.2, dj=0.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_connectome_matches_oracle(name):
    cfg = CASES[name]()
    eng, orc = E.Engine(cfg), O.OracleNet(cfg, 1)
    for h in range(cfg.glob_h):
        for g, o in zip(eng.backward_synapses(h), orc.synapses(h)):
            np.testing.assert_array_equal(g, o)
    gi, gm = eng.bath_params()
    oi, om = orc.bath_params()
    np.testing.assert_array_equal(gi, oi)
    np.testing.assert_array_equal(gm, om)
    # rank 0's dynamics continue its generation stream
    for _ in range(5):
        eng.step(1)
        orc.step()
    np.testing.assert_array_equal(eng.state()["nb"], orc.state()["nb"])
    eng.close()
