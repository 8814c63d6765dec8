"""External transfers against the oracle, bit for bit, at the sizes where
their wavefronts change hands -- one block (up to 512 transfers a wave), a
cluster of blocks (up to 8,192), the whole chip -- and at the samples that
leave the register path: long ones, proportions, shifts, weighted columns,
self-transfers."""
import numpy as np
import pytest

from helpers import run_oracle
from siminf_gb300 import abi, model as M

pytestmark = pytest.mark.gpu


def check(m, seed=42):
    from siminf_gb300 import native
    code, res, ho = run_oracle(m, seed=seed, threads=4)
    assert code == 0
    h = abi.build_args(m, seed)
    p = native.Plan(h, m.name, cap_transfers=True)
    for _ in range(2):                      # the second from the run's graph
        h.U[:] = -1
        p.run()
        p.download()
        assert np.array_equal(h.U, ho.U)
    p.close()


def transfers(rng, nodes, per_day, days, n_max):
    """per_day transfers a day from distinct sources, so that a day is one
    wave, then a day's worth of chains over few nodes."""
    cols = {k: [] for k in ("event", "time", "node", "dest", "n")}
    for t in range(1, days + 1):
        src = rng.permutation(nodes // 2)[:per_day] + 1         # lower half sends,
        dst = rng.integers(nodes // 2, nodes, per_day) + 1      # upper half receives
        few = rng.integers(1, 9, (40, 2))                       # then 8 nodes back and forth
        cols["event"].append(np.full(per_day + 40, 3))
        cols["time"].append(np.full(per_day + 40, t))
        cols["node"].append(np.concatenate([src, few[:, 0]]))
        cols["dest"].append(np.concatenate([dst, few[:, 1]]))
        cols["n"].append(rng.integers(1, n_max + 1, per_day + 40))
    return {k: np.concatenate(v) for k, v in cols.items()}


def seir(nodes, days, seed):
    """Nodes rich in every compartment: the transfers' samples draw, and
    are never short of individuals."""
    rng = np.random.default_rng(seed)
    u0 = rng.integers(3000, 5000, (4, nodes))
    m = M.SEIR(u0, np.arange(1, days + 1, dtype=float), 0.001, 0.0005, 0.0005)
    return rng, m


@pytest.mark.parametrize("reps", [1, 3])
@pytest.mark.parametrize("per_day", [1, 511, 512, 513, 4097, 8192, 8193, 9000])
def test_gpu_wave_sizes(gpu, oracle_lib, per_day, reps):
    rng, m = seir(2 * max(per_day, 20), 3, per_day)
    c = transfers(rng, m.Nn, per_day, 3, 8)
    m.events = M.make_events(c["event"], c["time"], c["node"], c["dest"], c["n"], [0.0], [2], [0],
                             sort=False)
    check(m.replicate(reps) if reps > 1 else m)


@pytest.mark.parametrize("n_max", [1, 4, 13, 60])
def test_gpu_long_samples(gpu, oracle_lib, n_max):
    """Samples of more draws than a thread holds ready, at every offset of
    the node's stream in its Philox block."""
    rng, m = seir(2000, 6, n_max)
    c = transfers(rng, m.Nn, 900, 6, n_max)
    m.events = M.make_events(c["event"], c["time"], c["node"], c["dest"], c["n"], [0.0], [2], [0],
                             sort=False)
    check(m)


def test_gpu_mixed_transfers(gpu, oracle_lib):
    """Counts and proportions, shifted and not, from one and several
    compartments, equal and unequal weights, to another node and to
    itself, and nodes with one kind of individual or none."""
    rng, m = seir(600, 5, 9)
    m.u0[:, ::7] = 0
    m.u0[1:, ::5] = 0
    m.u0[:3, ::11] = 0
    m.E = np.array([[1, 1, 1, 0], [0, 1, 2, 1], [0, 1, 1, 1], [0, 1, 3, 0]], dtype=float)
    m.N = np.array([[1], [1], [-1], [0]], dtype=np.int32)
    k = 1500
    n = rng.integers(0, 4, k)
    ev = M.make_events(np.full(k, 3), rng.integers(1, 6, k), rng.integers(1, 601, k),
                       rng.integers(1, 601, k), n, np.where(n == 0, rng.random(k) * 0.01, 0.0),
                       rng.integers(1, 5, k), rng.integers(0, 2, k) * (rng.random(k) < 0.3))
    own = rng.random(k) < 0.05
    ev["dest"][own] = ev["node"][own]
    m.events = ev
    from siminf_gb300 import native
    from oracle import oracle
    ho, hg = abi.build_args(m, 42), abi.build_args(m, 42)
    assert oracle.run(ho, m.name, 4, cap_transfers=True)[0] == 0
    p = native.Plan(hg, m.name, cap_transfers=True)
    p.run()
    p.download()
    p.close()
    assert np.array_equal(hg.U, ho.U)
