"""A post time step that leaves entries of v_new unwritten: v and v_new are
two buffers that change places at each day's end, so such an entry holds the
value of two days before.  Models compiled from C code against the oracle,
bit for bit: with and without transfers (day kernels and whole horizons), one
day to the next, across replicates, and in the particle filter."""
import numpy as np
import pytest

from helpers import run_gpu
from oracle import oracle
from siminf_gb300 import abi, model as M, mparse

pytestmark = pytest.mark.gpu

# phi every third day, psi on the day after it, and chi never
SOME_DAYS = """    const int day = (int) t %% 3;
    if (day == 1)
        v_new[0] = v[0] + %s;
    if (day == 2)
        v_new[1] = 0.5 * v[1] + 0.01 * u[1];
    return v_new[0] != v[0] || v_new[1] != v[1] || v_new[2] != v[2];"""


def build(n, days, step="0.02 * u[1]", t0=1, events=None, rate_t=False, replicates=1):
    rng = np.random.default_rng(n)
    u0 = {"S": rng.poisson(60, n), "I": rng.poisson(4, n)}
    infect = "(phi + psi + chi)*upsilon*S" + ("*(1.0 + 0.0*t)" if rate_t else "")
    m = mparse.mparse(["S -> %s -> I" % infect, "I -> gamma*I -> S"], ["S", "I"], u0,
                      np.arange(t0, t0 + days, dtype=float),
                      gdata={"upsilon": 0.02, "gamma": 0.1},
                      v0={"phi": 0.5, "psi": 0.25, "chi": 1.0}, pts_fun=SOME_DAYS % step,
                      events=events, E=np.array([[1, 1], [0, 1]], dtype=float))
    return m.replicate(replicates) if replicates > 1 else m


def check(m):
    oracle.register_c_model(m.name, m.C_code, m.Nc, m.Nt, m.Nd)
    ho = abi.build_args(m, 42)
    code, res = oracle.run(ho, m.name, 4)
    assert code == 0
    got, hg, st = run_gpu(m)
    assert got == 0
    assert np.array_equal(hg.V, ho.V)
    assert np.array_equal(hg.U, ho.U)
    assert st.transitions == res.transitions
    return ho


def one_event(kind, t, n):
    return M.make_events([kind], [t], [1], [2 if kind == 3 else 0], [1], [0.0], [2], [0])


@pytest.mark.parametrize("n", [1, 33, 700])
@pytest.mark.parametrize("days", [1, 2, 3, 20])
def test_gpu_unwritten_v_new_without_transfers(gpu, oracle_lib, n, days):
    check(build(n, days))


def test_gpu_unwritten_v_new_reads_t(gpu, oracle_lib):
    """phi + t on the days that write it (t = 1, 4, 7), from 0."""
    m = build(1, 8, step="t")
    m.v0[:] = 0.0
    ho = check(m)
    assert ho.V.reshape(8, 3)[:, 0].tolist() == [1, 0, 1, 5, 1, 5, 12, 5]


@pytest.mark.parametrize("kind", [0, 3])
@pytest.mark.parametrize("rate_t", [False, True])
def test_gpu_unwritten_v_new_with_an_event(gpu, oracle_lib, kind, rate_t):
    """The same answer whether an exit or a transfer is in the schedule, and
    whether or not the rates read t."""
    check(build(40, 20, events=one_event(kind, 6, 40), rate_t=rate_t))


def test_gpu_unwritten_v_new_replicates(gpu, oracle_lib):
    check(build(30, 20, replicates=3))


def test_gpu_unwritten_v_new_pfilter(gpu, oracle_lib):
    from siminf_gb300.run import pfilter
    m = build(20, 1, t0=0)
    oracle.register_c_model(m.name, m.C_code, m.Nc, m.Nt, m.Nd)
    rng = np.random.default_rng(9)
    t = np.arange(5, 41, 5, dtype=np.int32)
    obs = rng.binomial(8, 0.5, size=(len(t), 20)).astype(np.int32)
    gdata = np.column_stack([rng.uniform(0.005, 0.03, 48), rng.uniform(0.05, 0.2, 48)])
    code, ll, ess, anc = oracle.pfilter(m, 48, t, obs, 1, 0.8, seed=5, gdata=gdata, threads=4)
    r = pfilter(m, 48, t, obs, 1, 0.8, seed=5, gdata=gdata)
    assert code == 0
    assert r.loglik == ll
    assert np.array_equal(r.ess, ess)
    assert np.array_equal(r.ancestors, anc)
