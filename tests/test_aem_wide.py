"""The all-events method over many nodes a group of lanes (k_aem_day looks
through the ordinary part of its queue a lane a node) against the oracle, bit
for bit: nodes mostly quiet, all quiet and all active, events on quiet nodes,
heavy nodes beside them, and a count that fills no warp."""
import numpy as np
import pytest

from siminf_gb300 import model as M
from test_aem_lanes import both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heavy_rate", [0, 2, -1])
@pytest.mark.parametrize("infected", [0.0, 0.02, 1.0])
@pytest.mark.parametrize("name,n", [("SEIR", 160001), ("SIS", 311307)])
def test_gpu_aem_many_nodes(gpu, oracle_lib, name, n, infected, heavy_rate):
    rng = np.random.default_rng(n)
    S = rng.poisson(40, n)
    I = rng.poisson(4, n) * (rng.random(n) < infected)
    I[::50001] = 60 if infected else 0
    k = 3000
    ev = M.make_events(rng.integers(0, 2, k), rng.integers(1, 5, k), rng.integers(1, n + 1, k),
                       np.zeros(k, int), np.ones(k, int), np.zeros(k), np.full(k, 1),
                       np.zeros(k, int))
    days = np.arange(1.0, 6.0)
    if name == "SEIR":
        m = M.SEIR(np.vstack([S + 5, 0 * S, I, 0 * S]), days, 0.3, 0.25, 0.1, events=ev)
    else:
        m = M.SIS(np.vstack([S + 5, I]), days, 0.3, 0.2, events=ev)
    co, ho, res, cg, hg, st = both(m, heavy_rate=heavy_rate)
    assert co == 0 and cg == 0
    assert np.array_equal(hg.U, ho.U)
    assert st.transitions == res.transitions
