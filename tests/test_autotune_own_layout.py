"""The autotuner measures the layout the plan was created with, whatever its
threshold, and keeps its choice for plans created alike: thresholds between
the fixed candidates, the default of large models, a model compiled from C
code, and every candidate's trajectories, thresholds below one among them."""
import numpy as np
import pytest

from helpers import parity_cases
from siminf_gb300 import abi, model as M

pytestmark = pytest.mark.gpu


def seir_case():
    return dict(parity_cases())["seir_events_300x120"]


def candidates(r):
    return [(r.heavy_rate[k], r.two_pass[k], r.ssa_variant[k], r.wave_block[k])
            for k in range(r.n_candidates)]


@pytest.mark.parametrize("options,own", [
    ({}, (0.5, 0, 0, 128)),
    ({"heavy_rate": 3}, (3.0, 0, 0, 128)),
    ({"heavy_rate": 100, "two_pass": 1, "wave_block": 512}, (100.0, 1, 0, 512)),
    ({"heavy_rate": -1, "ssa_variant": 1}, (0.0, 0, 1, 128)),
])
def test_gpu_autotune_measures_the_plan_s_own_layout(gpu, options, own):
    from siminf_gb300 import native
    m = seir_case()
    p = native.Plan(abi.build_args(m, 42), m.name, **options)
    r = p.tune(probe_days=-6)
    p.close()
    assert own in candidates(r)
    assert 0 <= r.chosen < r.n_candidates


def test_gpu_autotune_large_model(gpu):
    from siminf_gb300 import native
    n = 500000
    u0 = np.zeros((4, n))
    u0[0], u0[2, ::40] = 50, 3
    m = M.SEIR(u0, np.arange(1.0, 4.0), 0.16, 0.25, 0.077,
               events=M.make_events([3], [2], [1], [2], [1], [0.0], [2], [0]))
    p = native.Plan(abi.build_args(m, 42), m.name)
    r = p.tune(probe_days=-3)
    p.close()
    assert (4.0, 1, 0, 128) in candidates(r)


def test_gpu_autotune_choice_belongs_to_the_layout(gpu):
    """A plan created with a threshold of its own does not hand its choice to
    a default plan, nor takes the default's."""
    from siminf_gb300 import native
    m = seir_case()
    plans = [native.Plan(abi.build_args(m, 42), m.name, **o)
             for o in ({"heavy_rate": 1}, {}, {}, {"heavy_rate": 1})]
    r = [p.tune(probe_days=7) for p in plans]
    assert [bool(x.cached) for x in r] == [False, False, True, True]
    assert r[2].chosen == r[1].chosen and r[3].chosen == r[0].chosen
    assert 0.5 in r[1].heavy_rate[:r[1].n_candidates]
    again = plans[1].tune(probe_days=7)     # its layout is the tuned one by now
    assert again.cached and again.chosen == r[1].chosen
    for p in plans:
        p.close()


def test_gpu_autotune_candidates_below_one(gpu, monkeypatch):
    """Every candidate gives the untuned plan's trajectories, thresholds that
    the integer option cannot name set through the environment."""
    from siminf_gb300 import native
    m = seir_case()
    h = abi.build_args(m, 42)
    p = native.Plan(h, m.name)
    p.run()
    p.download()
    r = p.tune(probe_days=-6)
    p.close()
    for k in range(r.n_candidates):
        monkeypatch.setenv("SIMINF_HEAVY_RATE", repr(r.heavy_rate[k]))
        hk = abi.build_args(m, 42)
        pk = native.Plan(hk, m.name, two_pass=1 if r.two_pass[k] else -1,
                         ssa_variant=r.ssa_variant[k], wave_block=r.wave_block[k])
        pk.run()
        pk.download()
        pk.close()
        assert np.array_equal(h.U, hk.U), k


def test_gpu_autotune_compiled_model(gpu):
    from siminf_gb300 import native
    from test_devmodel import seirs_custom
    m = seirs_custom(nodes=120, days=30)
    p = native.Plan(abi.build_args(m, 42), m.name)
    r = p.tune(probe_days=-6)
    p.close()
    assert (8.0, 0, 0, 128) in candidates(r)
