"""Whole horizons of nodes that fire many times a day (k_horizon runs a warp
of them day by day, in batches of four draws) against the oracle, bit for
bit: one node a warp and many, rate sums on both sides of the line within one
horizon, busy and quiet nodes in one warp, events and environmental steps at
the busy days' ends, and a bound on the day's transitions that is met inside
one."""
import ctypes as C

import numpy as np
import pytest

from helpers import run_gpu, run_oracle
from siminf_gb300 import abi, model as M

pytestmark = pytest.mark.gpu


def check(m, seed=42):
    code, res, ho = run_oracle(m, seed=seed, threads=4)
    got, hg, st = run_gpu(m, seed=seed)
    assert code == 0 and got == 0
    assert np.array_equal(hg.U, ho.U) and np.array_equal(hg.V, ho.V)
    assert st.transitions == res.transitions
    return ho


def exits(n, t0, t1, select):
    k = 2 * n
    rng = np.random.default_rng(n)
    return M.make_events(np.zeros(k, int), rng.integers(t0, t1, k), rng.integers(1, n + 1, k),
                         np.zeros(k, int), np.full(k, 3), np.zeros(k), np.full(k, select),
                         np.zeros(k, int))


def sir(S, I, days, events=None):
    return M.SIR(np.vstack([S, I, np.zeros_like(S)]), np.arange(1.0, days + 1), 0.4, 0.2,
                 events=events)


@pytest.mark.parametrize("n", [1, 3, 33, 609, 5000])
def test_gpu_busy_days(gpu, oracle_lib, n):
    """An infection that takes off, stays over the line for weeks and dies
    out, in nodes of one size."""
    check(sir(np.full(n, 3000), np.full(n, 20), 50, exits(n, 2, 50, 4)))


@pytest.mark.parametrize("n", [2, 64, 700, 5000])
def test_gpu_busy_and_quiet_nodes_in_a_warp(gpu, oracle_lib, n):
    S = np.where(np.arange(n) % 2 == 0, 4000, 10)
    check(sir(S, np.full(n, 5), 40))


@pytest.mark.parametrize("rate", [63.5, 64.0, 64.5])
def test_gpu_rate_sums_at_the_line(gpu, oracle_lib, rate):
    """Recoveries only, from a rate sum at the line."""
    n, I = 40, 200
    m = M.SIR(np.vstack([np.zeros(n, int), np.full(n, I), np.zeros(n, int)]),
              np.arange(1.0, 12), 0.0, rate / I)
    check(m)


def test_gpu_busy_days_with_an_environment(gpu, oracle_lib):
    n = 70
    check(M.SISe(np.vstack([np.full(n, 900), np.full(n, 300)]), np.arange(0.0, 30), phi=5.0,
                 upsilon=0.05, gamma=0.4, alpha=0.5, beta_t1=0.19, beta_t2=0.085, beta_t3=0.075,
                 beta_t4=0.185, end_t1=91, end_t2=182, end_t3=273, end_t4=365, epsilon=0.01,
                 events=exits(n, 1, 29, 1)))


def test_gpu_busy_days_replicates(gpu, oracle_lib):
    m = sir(np.full(20, 2000), np.full(20, 10), 30, exits(20, 2, 30, 4)).replicate(5)
    check(m)


@pytest.mark.parametrize("bound", [150, 10 ** 6])
def test_gpu_transition_bound_inside_a_busy_day(gpu, oracle_lib, bound):
    """More than `bound` transitions in a node's day end the run with the
    timeout error, a bound that none reaches changes nothing."""
    from siminf_gb300 import native
    m = sir(np.full(8, 3000), np.full(8, 400), 20)
    _, res, ho = run_oracle(m)
    h = abi.build_args(m, 42)
    opt = abi.Options(max_node_day_transitions=bound)
    code = native.lib().siminf_gpu_run_solver_ex(C.cast(h.ref(), C.c_void_p),
                                                 native.device_model(m.name).handle,
                                                 C.byref(opt))
    if bound > 1000:
        assert code == 0 and np.array_equal(h.U, ho.U)
        assert native.last_stats().transitions == res.transitions
    else:
        assert code == -33                  # SIMINF_GPU_ERR_TIMEOUT
