"""Nodes whose day a group of lanes steps (ssa_day_group) against the
oracle, bit for bit, where the groups can go wrong: batches of 8, 16 and 32
steps that fill, that end the day inside, and that follow one another for
many batches; rate sums and times that leave their binade; waiting times
that land on the day's end; infections that die out; a G matrix that
refreshes part of the rates."""
import ctypes as C

import numpy as np
import pytest

from helpers import run_oracle
from siminf_gb300 import abi, model as M

pytestmark = pytest.mark.gpu


def with_transfer(m, t, select=2):
    """m with one external transfer at time t, so that its days run through
    the work queue."""
    m.events = M.make_events([3], [t], [1], [2], [1], [0.0], [select], [0])
    return m


def run_plan(m, seed=42, **options):
    from siminf_gb300 import native
    h = abi.build_args(m, seed)
    p = native.Plan(h, m.name, cap_transfers=True, **options)
    p.run()
    p.download()
    transitions = p.stats().transitions
    p.close()
    return h, transitions


def check(m, seed=42, **options):
    """U, V and the transition count of a plan against the oracle's."""
    code, res, ho = run_oracle(m, seed=seed, threads=4)
    assert code == 0
    hg, transitions = run_plan(m, seed, **options)
    assert np.array_equal(hg.U, ho.U)
    assert np.array_equal(hg.V, ho.V)
    assert transitions == res.transitions
    return transitions


def populations(scale, n=37, seed=3):
    rng = np.random.default_rng(seed)
    return rng.poisson(30 * scale, n) + 2, rng.poisson(scale, n)


def build(name, scale, days):
    S, I = populations(scale)
    z = np.zeros_like(S)
    if name == "SEIR":
        return with_transfer(M.SEIR(np.vstack([S, z, I, z]), days, 0.16, 0.25, 0.077), 5)
    if name == "SIR":
        return with_transfer(M.SIR(np.vstack([S, I, z]), days, 0.3, 0.1), 5, 4)
    if name == "SIS":
        return with_transfer(M.SIS(np.vstack([S, I]), days, 0.3, 0.2), 5, 1)
    return with_transfer(M.SISe3(
        np.vstack([S, I, S // 2 + 1, I, S, z]), days, phi=1.0, upsilon_1=0.2, upsilon_2=0.1,
        upsilon_3=0.3, gamma_1=0.1, gamma_2=0.4, gamma_3=0.2, alpha=0.5, beta_t1=0.19,
        beta_t2=0.085, beta_t3=0.075, beta_t4=0.185, end_t1=91, end_t2=182, end_t3=273,
        end_t4=365, epsilon=0.01), 5, 1)


@pytest.mark.parametrize("heavy_rate", [0, 1, 3])
@pytest.mark.parametrize("scale", [1, 9, 60, 700])
@pytest.mark.parametrize("name", ["SEIR", "SIR", "SIS", "SISe3"])
def test_gpu_groups_match_oracle(gpu, oracle_lib, name, scale, heavy_rate):
    """scale 1: a few steps a day and infections that die out; 700:
    hundreds a day, many batches.  heavy_rate sets which nodes get 8, 16
    and 32 lanes (0: the default)."""
    n = check(build(name, scale, np.arange(1, 16, dtype=float)), heavy_rate=heavy_rate)
    assert n > 0


@pytest.mark.parametrize("tt0", [0.0, 0.25, 0.9, 1.5, 3.999, 1023.25, -1.5])
def test_gpu_groups_times_across_binades(gpu, oracle_lib, tt0):
    """Times from 0, below 1 (several binades inside a day), negative, and
    a day that ends on a power of two."""
    m = build("SEIR", 60, np.concatenate([[tt0], np.floor(tt0) + np.arange(2.0, 9.0)]))
    m.events["time"][:] = int(np.floor(tt0)) + 4
    check(m, heavy_rate=1)


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])
def test_gpu_groups_waiting_time_at_the_days_end(gpu, oracle_lib, ulps):
    """A start time from which node 0's first waiting time ends on the
    day's end, and a few units in the last place beside it."""
    S, I = populations(60)
    m0 = M.SIS(np.vstack([S, I]), np.arange(1.0, 6.0), 0.3, 0.2)
    w = oracle_lib.philox((0, 0, 0, 0), (42, 0))[0]
    lam = 0.3 * S[0] * I[0] / (S[0] + I[0]) + 0.2 * I[0]
    tau = float(oracle_lib.neglog_u32(np.array([w], dtype=np.uint32))[0]) / lam
    assert 0.0 < tau < 1.0
    tt0 = 2.0 - tau
    for _ in range(abs(ulps)):
        tt0 = np.nextafter(tt0, 10.0 * np.sign(ulps))
    m = M.SIS(m0.u0, np.array([tt0, 3.0, 4.0, 5.0]), 0.3, 0.2)
    check(with_transfer(m, 4, 1), heavy_rate=1)


@pytest.mark.parametrize("total", [62, 63, 64, 65, 127, 128])
def test_gpu_groups_rate_sum_across_binades(gpu, oracle_lib, total):
    """Rate sums that start beside a power of two and walk across it."""
    n = 20
    I = np.full(n, total * 2)
    S = np.full(n, 10 * total)
    m = M.SIS(np.vstack([S, I]), np.arange(1.0, 9.0), 0.275, 0.25)
    check(with_transfer(m, 3, 1), heavy_rate=1)


def test_gpu_groups_partial_refresh(gpu, oracle_lib):
    """A G matrix that leaves a rate stale, as a caller may pass it: the
    groups keep the rate of the last step that refreshed it."""
    m = build("SEIR", 60, np.arange(1, 12, dtype=float))
    m.G = np.array([[1, 0, 1], [1, 1, 0], [0, 1, 1]], dtype=np.int32)
    check(m, heavy_rate=1)


def test_gpu_groups_replicates(gpu, oracle_lib):
    m = build("SEIR", 60, np.arange(1, 12, dtype=float)).replicate(5)
    check(m, heavy_rate=1)


@pytest.mark.parametrize("bound,code", [(20, -33), (100000, 0)])
def test_gpu_groups_transition_bound(gpu, bound, code):
    """A node that would fire more than the bound inside a batch stops the
    run with the timeout error."""
    from siminf_gb300 import native
    m = build("SEIR", 700, np.arange(1, 8, dtype=float))
    h = abi.build_args(m, 42)
    opt = abi.Options(heavy_rate=1, max_node_day_transitions=bound, cap_transfers=1)
    got = native.lib().siminf_gpu_run_solver_ex(C.cast(h.ref(), C.c_void_p),
                                                native.device_model(m.name).handle,
                                                C.byref(opt))
    assert got == code


def test_gpu_groups_fast_growth(gpu, oracle_lib):
    """Rate sums that grow severalfold within a day: the step that ends
    the day starts later than the batch's first estimate of its time, just
    after a rate sum that left its binade."""
    rng = np.random.default_rng(8)
    n = 30000
    u0 = np.vstack([rng.integers(0, 400, n), rng.integers(0, 4, n), rng.integers(0, 4, n),
                    rng.integers(0, 50, n)])
    m = M.SEIR(u0, np.arange(1.0, 6.0), 2.0, 0.25, 0.077)
    m.events = M.make_events([3], [3], [int(np.argmax(u0[0])) + 1], [2], [1], [0.0], [2], [0])
    check(m, heavy_rate=1)
