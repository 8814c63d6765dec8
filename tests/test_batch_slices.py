"""The batch's merged event table, written by host threads slice by slice:
models of more events than a slice (131,072) and of none, events past a
model's horizon, and a model whose events are not in order, against each
model's own run."""
import numpy as np
import pytest

from siminf_gb300 import model as M

pytestmark = pytest.mark.gpu


def seir(n, days, per_day, seed, extra_days=0):
    rng = np.random.default_rng(seed)
    u0 = np.vstack([rng.poisson(300, n), np.zeros(n, int), rng.poisson(2, n), np.zeros(n, int)])
    T = days + extra_days
    t = np.repeat(np.arange(1, T + 1), per_day)
    kind = np.tile(np.where(np.arange(per_day) % 7 == 0, 1, 3), T)
    k = len(t)
    node, dest = rng.integers(1, n + 1, k), rng.integers(1, n + 1, k)
    ev = M.make_events(kind, t, node, np.where(kind == 3, dest, 0), np.ones(k, int), [0.0],
                       np.where(kind == 1, 1, 2), [0])
    return M.SEIR(u0, np.arange(1, days + 1, dtype=float), 0.16, 0.25, 0.077, events=ev)


def prevalence(m, seed):
    from siminf_gb300.run import run
    U = run(m, seed=seed, cap_transfers=True).U.reshape(m.Nn, 4, -1)
    num, den = U[:, 2].sum(0), U.sum((0, 1))
    return num / den


def test_gpu_batch_slices_match_single_runs(gpu):
    from siminf_gb300.run import run_batch
    models = [seir(50, 20, 10, 1), seir(3000, 15, 9000, 2), seir(40, 25, 0, 3),
              seir(700, 10, 13200, 4, extra_days=6), seir(60, 12, 40, 5)]
    assert max(len(m.events["time"]) for m in models) > 1 << 17
    seeds = [11, 12, 13, 14, 15]
    prev, _ = run_batch(models, seeds, cap_transfers=True)
    for m, s, p in zip(models, seeds, prev):
        cut = m.events["time"] <= len(m.tspan)
        m.events = {k: np.ascontiguousarray(v[cut]) for k, v in m.events.items()}
        assert np.array_equal(p, prevalence(m, s))


def test_gpu_batch_unordered_model(gpu):
    """A model's events may come in any order of times: the batch sorts
    them, stably, by (time, transfers after the others)."""
    from siminf_gb300.run import run_batch
    a, b = seir(80, 12, 30, 6), seir(80, 12, 30, 6)
    rng = np.random.default_rng(1)
    ev = b.events
    order = rng.permutation(len(ev["time"]))
    b.events = {k: np.ascontiguousarray(v[order]) for k, v in ev.items()}
    e = b.events
    back = np.lexsort((e["event"] == 3, e["time"]))     # stable
    a.events = {k: np.ascontiguousarray(v[back]) for k, v in e.items()}
    other = seir(30, 9, 5, 7)
    p, _ = run_batch([a, other], [3, 4], cap_transfers=True)
    q, _ = run_batch([b, other], [3, 4], cap_transfers=True)
    assert np.array_equal(p[0], q[0]) and np.array_equal(p[1], q[1])
