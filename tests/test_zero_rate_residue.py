"""A rate sum that is positive while every rate is zero (the residue of
rounded additions): the step that finds it sets the sum to zero and leaves
the node's time at that step, so that an event of the same day which brings
the rates back starts the next waiting time from there.  Whole horizons and
the day kernels against the oracle, bit for bit."""
import numpy as np
import pytest

from helpers import run_gpu
from oracle import oracle
from siminf_gb300 import abi, model as M, mparse

# c is 10^16: the rates 10^16 and 1.7 of one X and one Y add up to 10^16 + 2,
# and once both have gone 0.3 of that is left
DAYS, RATES = 12, {"c": 1e16, "d": 1.7}


def build(n, transfer):
    nodes, days = np.arange(1, n + 1), np.arange(1, DAYS)
    ev = {"event": np.ones(n * len(days), int), "time": np.repeat(days, n),
          "node": np.tile(nodes, len(days)), "dest": np.zeros(n * len(days), int)}
    if transfer:
        for k, x in zip(ev, (3, DAYS - 1, 1, 2)):
            ev[k] = np.append(ev[k], x)
    k = len(ev["event"])
    return mparse.mparse(["X -> c*X -> @", "Y -> d*Y -> @"], ["X", "Y"],
                         {"X": np.ones(n), "Y": np.ones(n)}, np.arange(1.0, DAYS + 1),
                         gdata=RATES, E=np.array([[0], [1]], dtype=float),
                         events=M.make_events(n=np.ones(k, int), proportion=np.zeros(k),
                                              select=np.ones(k, int), shift=np.zeros(k, int),
                                              **ev))


def expected(m):
    oracle.register_c_model(m.name, m.C_code, m.Nc, m.Nt, m.Nd)
    h = abi.build_args(m, 42)
    code, res = oracle.run(h, m.name, 4)
    assert code == 0
    return h, res


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 40, 1500])
@pytest.mark.parametrize("transfer", [False, True])
def test_gpu_zero_rates_under_a_positive_sum(gpu, oracle_lib, n, transfer):
    m = build(n, transfer and n > 1)
    ho, res = expected(m)
    code, hg, st = run_gpu(m)
    assert code == 0
    assert np.array_equal(hg.U, ho.U)
    assert st.transitions == res.transitions
