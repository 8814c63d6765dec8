"""The particle filter's ordered sums (weights over nodes, weights, squares,
cumulative weights and resampling points over particles) against the
oracle, bit for bit, at node and particle counts beside the 32 and 128
additions a warp takes at once and beside its cluster's 4,096 threads;
weights that are all equal, floored, or carried by one particle."""
import numpy as np
import pytest

from oracle import oracle
from test_pfilter import small_case

pytestmark = pytest.mark.gpu


def check(m, P, t, obs, gdata=None, p=0.8, seed=5):
    from siminf_gb300.run import pfilter
    code, ll, ess, anc = oracle.pfilter(m, P, t, obs, 1, p, seed=seed, gdata=gdata, threads=4)
    r = pfilter(m, P, t, obs, 1, p, seed=seed, gdata=gdata)
    assert code == 0
    assert r.loglik == ll
    assert np.array_equal(r.ess, ess)
    assert np.array_equal(r.ancestors, anc)


@pytest.mark.parametrize("P", [1, 2, 31, 32, 33, 127, 128, 129, 1000, 4096, 4097])
def test_gpu_pfilter_particles(gpu, oracle_lib, P):
    m, gdata, t, obs = small_case(nodes=7, particles=P, weeks=4, seed=P)
    check(m, P, t, obs, gdata)


@pytest.mark.parametrize("nodes", [1, 31, 32, 33, 127, 128, 129, 300])
def test_gpu_pfilter_nodes(gpu, oracle_lib, nodes):
    m, gdata, t, obs = small_case(nodes=nodes, particles=40, weeks=3, seed=nodes)
    check(m, 40, t, obs, gdata)


@pytest.mark.parametrize("obs_value", [0, 1, 90])
def test_gpu_pfilter_weights_alike_and_floored(gpu, oracle_lib, obs_value):
    """No infected at all: every particle weighs the same (0 observed) or
    is impossible (1 observed); 90: impossible for most counts."""
    m, gdata, t, obs = small_case(nodes=12, particles=200, weeks=3)
    if obs_value < 2:
        m.u0[1, :] = 0
    obs[:] = obs_value
    check(m, 200, t, obs, gdata)
