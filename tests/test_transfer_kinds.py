"""Schedules whose transfers are mostly proportions, shifts or samples from
weighted columns, which the cluster launch takes in waves of up to a block's
512 only, against the oracle, bit for bit: wave sizes beside that line and
beside the cluster's 8,192, through a plan and through the streamed run, and
mixtures on both sides of the share at which the line moves."""
import numpy as np
import pytest

from helpers import run_gpu, run_oracle
from siminf_gb300 import abi, model as M
from test_transfer_waves import seir, transfers

pytestmark = pytest.mark.gpu


def build(per_day, kind, share=1.0, days=3):
    rng, m = seir(2 * max(per_day, 20), days, per_day)
    c = transfers(rng, m.Nn, per_day, days, 8)
    k = len(c["event"])
    rare = rng.random(k) < share
    # proportions and shifts leave the nodes rich enough for the counts
    n = np.where(rare, 0, c["n"]) if kind == "proportion" else c["n"]
    prop = np.where(n == 0, 0.002, 0.0)
    select = np.where(rare, 3, 2) if kind == "weighted" else np.full(k, 2)
    shift = np.where(rare, 1, 0) if kind == "shift" else np.zeros(k, int)
    m.E = np.array([[1, 1, 1], [0, 1, 2], [0, 1, 1], [0, 1, 3]], dtype=float)
    m.N = np.array([[1], [1], [-1], [0]], dtype=np.int32)
    m.events = M.make_events(c["event"], c["time"], c["node"], c["dest"], n, prop, select, shift,
                             sort=False)
    return m


def check(m):
    from siminf_gb300 import native
    code, res, ho = run_oracle(m, threads=4)
    assert code == 0
    h = abi.build_args(m, 42)
    p = native.Plan(h, m.name)
    p.run()
    p.download()
    p.close()
    assert np.array_equal(h.U, ho.U)
    got, hg, _ = run_gpu(m)                 # the streamed run
    assert got == 0 and np.array_equal(hg.U, ho.U)


@pytest.mark.parametrize("kind", ["proportion", "shift", "weighted"])
@pytest.mark.parametrize("per_day", [40, 512, 513, 8192, 8193])
def test_gpu_waves_of_other_transfers(gpu, oracle_lib, kind, per_day):
    check(build(per_day, kind))


@pytest.mark.parametrize("share", [0.05, 0.125, 0.25])
def test_gpu_mixtures_at_the_line(gpu, oracle_lib, share):
    check(build(900, "proportion", share))
