"""The all-events method with a lane for each transition (k_aem_day) against
the oracle, bit for bit: models of two, three and six transitions (groups of
2, 4 and 8 lanes), node counts beside a warp's groups, with and without the
heavy part, and a node bound to the transition limit."""
import ctypes as C

import numpy as np
import pytest

from siminf_gb300 import abi, model as M
from test_horizon_passes import build

pytestmark = pytest.mark.gpu


def both(m, **options):
    from oracle import oracle
    from siminf_gb300 import native
    ho, hg = abi.build_args(m, 42, solver=1), abi.build_args(m, 42, solver=1)
    co, res = oracle.run(ho, m.name, 4)
    opt = abi.Options(**options)
    cg = native.lib().siminf_gpu_run_solver_ex(C.cast(hg.ref(), C.c_void_p),
                                               native.device_model(m.name).handle, C.byref(opt))
    return co, ho, res, cg, hg, native.last_stats()


@pytest.mark.parametrize("heavy_rate", [0, 2])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 9, 15, 17, 33, 700])
@pytest.mark.parametrize("name", ["SIR", "SEIR", "SISe3"])
def test_gpu_aem_groups(gpu, oracle_lib, name, n, heavy_rate):
    co, ho, res, cg, hg, st = both(build(name, n, np.arange(1, 16, dtype=float)),
                                   heavy_rate=heavy_rate)
    assert co == 0 and cg == 0
    assert np.array_equal(hg.U, ho.U) and np.array_equal(hg.V, ho.V)
    assert st.transitions == res.transitions


def test_gpu_aem_busy_nodes(gpu, oracle_lib):
    """Hundreds of events a day beside nodes with none."""
    rng = np.random.default_rng(3)
    n = 40
    u0 = np.vstack([rng.poisson(2000, n), np.zeros(n, int),
                    rng.poisson(300, n) * (np.arange(n) % 3 == 0), np.zeros(n, int)])
    co, ho, res, cg, hg, st = both(M.SEIR(u0, np.arange(1.0, 9.0), 0.3, 0.25, 0.1))
    assert co == 0 and cg == 0 and np.array_equal(hg.U, ho.U)
    assert st.transitions == res.transitions


def test_gpu_aem_transition_bound(gpu):
    from siminf_gb300 import native
    u0 = np.array([[2000, 5], [0, 0], [300, 0], [0, 0]])
    m = M.SEIR(u0, np.arange(1.0, 6.0), 0.3, 0.25, 0.1)
    h = abi.build_args(m, 42, solver=1)
    opt = abi.Options(max_node_day_transitions=30)
    assert native.lib().siminf_gpu_run_solver_ex(
        C.cast(h.ref(), C.c_void_p), native.device_model(m.name).handle, C.byref(opt)) == -33
