"""The quiet test of a two-pass day (k_quick), which finds in single
precision the nodes whose first waiting time passes the day's end and takes
the quotient in double precision near a tie, against the oracle, bit for bit:
every node's waiting time set beside the day's end, from a unit in the last
place to 10^-4 of it, for start times up to 2^30 and rate sums up to 10^7."""
import numpy as np
import pytest

from siminf_gb300 import model as M
from test_lane_groups import check, with_transfer

pytestmark = pytest.mark.gpu

SEED = 42
OFF = np.array([0.0, 1.1e-16, 2.3e-16, 1e-15, 1e-13, 1e-10, 1e-8, 1e-7, 1e-6, 3e-6, 8e-6, 1e-5,
                1.3e-5, 3e-5, 1e-4])


def at_the_days_end(oracle_lib, tt0, n=4096):
    """n nodes of recoveries only whose first waiting time, from tt0, is
    the day's rest times 1 + an offset of either sign."""
    rng = np.random.default_rng(int(tt0) % 1000 + n)
    words = [oracle_lib.philox((0, 0, g, 0), (SEED, 0))[0] for g in range(n)]
    L = oracle_lib.neglog_u32(np.array(words, dtype=np.uint32))
    rest = np.floor(tt0) + 1.0 - tt0
    I = rng.integers(1, 40, n)
    off = 1.0 + rng.choice(OFF, n) * rng.choice([-1.0, 1.0], n)
    gamma = L / (rest * I) * off
    m = M.SIS(np.vstack([np.zeros(n, int), I]), np.concatenate([[tt0], np.floor(tt0) +
                                                                np.arange(2.0, 4.0)]),
              0.0, 0.1)
    m.ldata[1, :] = gamma
    return with_transfer(m, int(np.floor(tt0)) + 2, 2), L / (gamma * I) / rest


@pytest.mark.parametrize("tt0", [0.0, 1.0, 0.25, 1.0 - 2.0 ** -20, 1023.25, 1e6,
                                 1e6 + 1 - 2.0 ** -20,
                                 1e9, 1e9 + 0.75, 1e9 + 1 - 2.0 ** -18, 2.0 ** 30 - 1])
@pytest.mark.parametrize("heavy_rate", [-1, 0])
def test_gpu_quiet_nodes_at_the_days_end(gpu, oracle_lib, tt0, heavy_rate):
    m, ratio = at_the_days_end(oracle_lib, tt0)
    assert np.abs(ratio - 1.0).max() < 1.01e-4          # every node is beside the line
    assert 0.2 < np.mean(ratio > 1.0) < 0.8             # on both sides of it
    check(m, seed=SEED, two_pass=1, heavy_rate=heavy_rate)
