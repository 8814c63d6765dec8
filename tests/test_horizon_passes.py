"""Whole horizons of nodes that no transfer couples (k_horizon) against the
oracle, bit for bit: node counts beside the steps of its launch (a warp's
lanes, the warps that fill the chip), days that end in an event or in an
environmental step, infections that die out, fractional times, sparse
outputs, common random numbers, and errors in the middle of a horizon."""
import numpy as np
import pytest

from helpers import run_gpu, run_oracle
from siminf_gb300 import abi, model as M

pytestmark = pytest.mark.gpu


def build(name, n, days, seed=4, events=True):
    rng = np.random.default_rng(seed)
    S, I = rng.poisson(40, n), rng.poisson(2, n)
    z = np.zeros(n, dtype=int)
    ev, sel = None, {"SIR": 4, "SIS": 1, "SEIR": 2, "SISe": 1, "SISe3": 4}[name]
    if events:
        k = max(4, n // 2)
        t0, t1 = int(np.floor(days[0])) + 1, int(np.floor(days[-1]))
        ev = M.make_events(rng.integers(0, 2, k), rng.integers(t0, t1 + 1, k),
                           rng.integers(1, n + 1, k), np.zeros(k, int), np.ones(k, int),
                           np.zeros(k), np.full(k, sel), np.zeros(k, int))
    env = dict(alpha=0.5, beta_t1=0.19, beta_t2=0.085, beta_t3=0.075, beta_t4=0.185, end_t1=91,
               end_t2=182, end_t3=273, end_t4=365, epsilon=0.01)
    if name == "SIR":
        return M.SIR(np.vstack([S + 30, I, z]), days, 0.3, 0.15, events=ev)
    if name == "SIS":
        return M.SIS(np.vstack([S + 30, I]), days, 0.3, 0.2, events=ev)
    if name == "SEIR":
        return M.SEIR(np.vstack([S + 30, z, I, z]), days, 0.4, 0.25, 0.2, events=ev)
    if name == "SISe":
        return M.SISe(np.vstack([S + 30, I]), days, phi=0.5, upsilon=0.02, gamma=0.1, events=ev,
                      **env)
    return M.SISe3(np.vstack([S + 30, I, S, z, S, I]), days, phi=1.0, upsilon_1=0.02,
                   upsilon_2=0.02, upsilon_3=0.01, gamma_1=0.1, gamma_2=0.1, gamma_3=0.1,
                   events=ev, **env)


def check(m, **kw):
    code, res, ho = run_oracle(m, threads=4, **kw)
    got, hg, st = run_gpu(m, **kw)
    assert code == 0 and got == 0
    for a, b in ((hg.U, ho.U), (hg.V, ho.V), (hg.prU, ho.prU), (hg.prV, ho.prV)):
        assert (a is None and b is None) or np.array_equal(a, b)
    assert st.transitions == res.transitions


@pytest.mark.parametrize("name", ["SIR", "SIS", "SEIR", "SISe", "SISe3"])
@pytest.mark.parametrize("n", [1, 31, 33, 500, 609, 1217])
def test_gpu_horizon_sizes(gpu, oracle_lib, name, n):
    check(build(name, n, np.arange(1, 41, dtype=float)))


@pytest.mark.parametrize("n", [4865, 9729, 19457])
def test_gpu_horizon_lanes(gpu, oracle_lib, n):
    check(build("SIR", n, np.arange(1, 31, dtype=float)))


@pytest.mark.parametrize("name", ["SIR", "SISe"])
def test_gpu_horizon_times(gpu, oracle_lib, name):
    """A start between days, several stored times in a day and days without
    any."""
    check(build(name, 70, np.array([0.25, 1.0, 1.5, 1.75, 7.0, 7.5, 20.0]), events=False))


def test_gpu_horizon_replicates_crn(gpu, oracle_lib):
    m = build("SISe", 60, np.arange(1, 31, dtype=float)).replicate(3)
    check(m)
    ho, hg = abi.build_args(m, 42), abi.build_args(m, 42)
    ho.args.crn = hg.args.crn = 1
    from oracle import oracle
    from siminf_gb300 import native
    assert oracle.run(ho, m.name, 4)[0] == 0
    p = native.Plan(hg, m.name)
    p.run()
    p.download()
    p.close()
    assert np.array_equal(hg.U, ho.U) and np.array_equal(hg.V, ho.V)


def test_gpu_horizon_sparse(gpu, oracle_lib):
    m = build("SISe", 50, np.arange(1, 21, dtype=float))
    rng = np.random.default_rng(2)
    pats = []
    for rows in (m.Nn * m.Nc, m.Nn):
        keep = rng.random((rows, len(m.tspan))) < 0.2
        ir = np.concatenate([np.nonzero(keep[:, c])[0] for c in range(keep.shape[1])])
        jc = np.concatenate([[0], np.cumsum(keep.sum(0))])
        pats.append((ir.astype(np.int32), jc.astype(np.int32)))
    check(m, U_sparse=pats[0], V_sparse=pats[1])


@pytest.mark.parametrize("case", ["rate", "sample"])
def test_gpu_horizon_errors(gpu, oracle_lib, case):
    """The oracle's error for a rate that becomes invalid through an event
    (a negative recovery rate shows once someone is infected) and for an
    exit of more individuals than there are."""
    m = build("SIR", 40, np.arange(1, 21, dtype=float), events=False)
    if case == "rate":
        m.u0[1, :] = 0
        m.ldata[1, 7] = -0.1
        m.events = M.make_events([1], [6], [8], [0], [2], [0.0], [2], [0])
    else:
        m.events = M.make_events([0], [6], [8], [0], [5000], [0.0], [4], [0])
    code, _, _ = run_oracle(m, threads=4)
    got, _, _ = run_gpu(m)
    assert code < 0 and got == code
