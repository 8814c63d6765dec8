"""The work that users of this package have it do, as cases to be timed.

Every case goes through a public entry point: run() on host arrays, a
device-resident Plan (one model, replicates, the all-events solver),
pfilter(), Pmcmc, run_batch(), and the consumers of a trajectory.  The
sizes are those of the benchmark configurations, of the tests and of the
serving mix, some of them cut in days so that a pass takes at most about a
second.  All inputs come from the seed alone.

A case is {"name", "kind", sizes...}; `draw` gives further cases of the
ranges that the listed ones stand for.
"""
import ctypes as C

import numpy as np
import torch

from siminf_gb300 import abi, model, native, trajectory
from siminf_gb300.run import Pmcmc, pfilter, run as run_model, run_batch


def listed():
    return [
        # The benchmark's smallest configuration: one run() of a
        # thousand-node SIR model, where latency and launches count.
        {"name": "sir_1k_150d", "kind": "sir", "nodes": 1000, "days": 150},
        # The largest plain SIR request of the serving mix.
        {"name": "sir_20k_365d", "kind": "sir", "nodes": 20_000, "days": 365},
        # A livestock model of three age classes with an environmental
        # compartment: six compartments, six transitions, births, ageing,
        # exits and animal movements between 1,600 herds for two years.
        {"name": "sise3_1600_730d", "kind": "sise3", "nodes": 1600, "days": 730},
        # The smallest SEIR-with-events request of the serving mix.
        {"name": "seir_10k_365d", "kind": "seir", "nodes": 10_000, "days": 365,
         "replicates": 1, "solver": "ssm", "resident": False},
        # A larger one, half a year, its events and trajectory in host memory.
        {"name": "seir_100k_180d", "kind": "seir", "nodes": 100_000, "days": 180,
         "replicates": 1, "solver": "ssm", "resident": False},
        # The headline workload over its first eight months, from a quiet
        # start past the epidemic's peak, with inputs and trajectory on the
        # device.
        {"name": "seir_1m_240d_resident", "kind": "seir", "nodes": 1_000_000, "days": 240,
         "replicates": 1, "solver": "ssm", "resident": True},
        # Sixteen replicates of one model in one plan (the mssm solver).
        {"name": "seir_100k_x16_150d", "kind": "seir", "nodes": 100_000, "days": 150,
         "replicates": 16, "solver": "ssm", "resident": True},
        # The all-events solver on the same workload.
        {"name": "aem_100k_120d", "kind": "seir", "nodes": 100_000, "days": 120,
         "replicates": 1, "solver": "aem", "resident": True},
        # The particle-filter configuration: 4,096 particles of 500 nodes,
        # 52 weekly observations, end to end.
        {"name": "pfilter_4096", "kind": "pfilter", "particles": 4096, "nodes": 500,
         "weeks": 52},
        # A short chain of small filters, as pmcmc() and the serving mix's
        # smallest particle filters run them.
        {"name": "pmcmc_256x4", "kind": "pmcmc", "particles": 256, "nodes": 500, "weeks": 52,
         "iterations": 4},
        # A batch of uneven ABC proposals, run as one with their prevalence
        # and distances.
        {"name": "abc_48", "kind": "abc", "proposals": 48},
        # What is read from a finished trajectory: prevalence at the levels
        # of the population and of the nodes, and one compartment in long
        # format.
        {"name": "consumers_1m_60d", "kind": "consumers", "nodes": 1_000_000, "columns": 60},
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["sir", "sise3", "seir", "replicates", "aem", "resident", "pfilter",
                       "pmcmc", "abc", "consumers"])
    if kind == "sir":
        return {"kind": "sir", "nodes": _log_int(rng, 100, 20_000), "days": rng.randint(30, 365)}
    if kind == "sise3":
        return {"kind": "sise3", "nodes": _log_int(rng, 100, 4000), "days": rng.randint(90, 730)}
    if kind == "seir":
        return {"kind": "seir", "nodes": _log_int(rng, 5000, 100_000),
                "days": rng.randint(30, 180), "replicates": 1, "solver": "ssm",
                "resident": False}
    if kind == "replicates":
        return {"kind": "seir", "nodes": _log_int(rng, 1000, 100_000),
                "days": rng.randint(20, 150), "replicates": rng.randint(2, 16), "solver": "ssm",
                "resident": True}
    if kind == "aem":
        return {"kind": "seir", "nodes": _log_int(rng, 1000, 100_000),
                "days": rng.randint(30, 120), "replicates": 1, "solver": "aem",
                "resident": True}
    if kind == "resident":
        return {"kind": "seir", "nodes": _log_int(rng, 50_000, 1_000_000),
                "days": rng.randint(30, 240), "replicates": 1, "solver": "ssm",
                "resident": True}
    if kind == "pfilter":
        return {"kind": "pfilter", "particles": _log_int(rng, 256, 4096),
                "nodes": rng.randint(40, 500), "weeks": rng.randint(6, 52)}
    if kind == "pmcmc":
        return {"kind": "pmcmc", "particles": _log_int(rng, 64, 1024),
                "nodes": rng.randint(40, 500), "weeks": rng.randint(6, 52),
                "iterations": rng.randint(1, 4)}
    if kind == "abc":
        return {"kind": "abc", "proposals": rng.randint(4, 48)}
    return {"kind": "consumers", "nodes": _log_int(rng, 10_000, 1_000_000),
            "columns": rng.randint(10, 60)}


# ------------------------------------------------------------------
# Inputs.
# ------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randint(g, hi, n):
    return torch.randint(0, hi, (n,), generator=g, device="cuda", dtype=torch.int64)


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _poisson(g, lam, n):
    return torch.poisson(torch.full((n,), float(lam), device="cuda"), generator=g).to(torch.int64)


def _some(g, total, p):
    """The indices of a Bernoulli(p) draw for each of `total` places, in order."""
    n = int(_poisson(g, total * p, 1).item()) if total * p < 1e7 else int(total * p)
    return torch.unique(_randint(g, total, n))


def _host(x, dtype=np.int32):
    return np.ascontiguousarray(x.cpu().numpy().astype(dtype, copy=False))


def _events(parts, days):
    """Event columns in the order of SimInf_events -- time, event kind,
    select, input -- from groups (day, kind, node, dest, n, select, shift),
    zero-based nodes."""
    key = torch.cat([p[0] * 64 + p[1] * 16 + p[5] for p in parts])
    order = torch.argsort(key, stable=True)

    def col(f):
        return _host(torch.cat([f(p) for p in parts])[order].to(torch.int32))

    def const(p, v):
        return torch.full_like(p[2], v)

    ev = {"event": col(lambda p: const(p, p[1])), "time": col(lambda p: p[0] + 1),
          "node": col(lambda p: p[2] + 1),
          "dest": col(lambda p: const(p, 0) if p[3] is None else p[3] + 1),
          "n": col(lambda p: const(p, p[4]) if isinstance(p[4], int) else p[4]),
          "select": col(lambda p: const(p, p[5])), "shift": col(lambda p: const(p, p[6]))}
    ev["proportion"] = np.zeros(len(ev["time"]))
    return ev


def _at(index, nodes):
    return torch.div(index, nodes, rounding_mode="floor"), index % nodes


def _seir(nodes, days, seed, beta=0.16, epsilon=0.25, gamma=0.077):
    """SEIR with scheduled events, as the benchmark's workload has it: S ~
    Poisson(300), one node in a hundred with Poisson(3) infected; enter and
    exit events with probability 0.002 a node-day; nodes / 2 external
    transfers a day of 1 + Poisson(3) individuals over a fixed graph of 2 *
    nodes edges with uniform sources and a truncated power law (exponent
    2.1, cutoff sqrt(edges)) of destinations."""
    g = _gen(seed)
    S = _poisson(g, 300, nodes)
    I = _poisson(g, 3, nodes) * (_rand(g, nodes) < 0.01)
    u0 = _host(torch.stack([S, torch.zeros_like(S), I, torch.zeros_like(S)]))
    transfers = max(1, nodes // 2)
    edges = 4 * transfers
    a, cut = 1.1, float(np.sqrt(edges))
    w = (1.0 - _rand(g, nodes) * (1.0 - cut ** -a)) ** (-1.0 / a)
    cum = torch.cumsum(w, 0)
    src = _randint(g, nodes, edges)
    dst = torch.searchsorted(cum, _rand(g, edges) * cum[-1]).clamp_(max=nodes - 1)
    dst = torch.where(dst == src, (dst + 1) % nodes, dst)
    ex_t, ex_n = _at(_some(g, nodes * days, 0.002), nodes)
    en_t, en_n = _at(_some(g, nodes * days, 0.002), nodes)
    pick = _randint(g, edges, transfers * days)
    day = torch.arange(days, device="cuda").repeat_interleave(transfers)
    ev = _events([(ex_t, 0, ex_n, None, 1, 2, 0), (en_t, 1, en_n, None, 1, 1, 0),
                  (day, 3, src[pick], dst[pick], 1 + _poisson(g, 3, transfers * days), 2, 0)],
                 days)
    return model.SEIR(u0, np.arange(1, days + 1, dtype=float), beta=beta, epsilon=epsilon,
                      gamma=gamma, events=ev)


def _sise3(nodes, days, seed):
    """SISe3 herds: a birth a fortnight, an exit from each age class and an
    ageing step from each a month, a movement of adults every three weeks."""
    g = _gen(seed)
    zero = torch.zeros(nodes, dtype=torch.int64, device="cuda")
    inf = (_rand(g, nodes) < 0.1).to(torch.int64)
    u0 = _host(torch.stack([_poisson(g, 10, nodes), zero, _poisson(g, 20, nodes), zero,
                            _poisson(g, 70, nodes), inf * _poisson(g, 5, nodes)]))

    def group(p, kind, n, select, shift=0):
        t, k = _at(_some(g, nodes * days, p), nodes)
        return (t, kind, k, None, n, select, shift)

    t, k = _at(_some(g, nodes * days, 1 / 21), nodes)
    to = (k + 1 + _randint(g, max(1, nodes - 1), len(k))) % nodes
    ev = _events([group(1 / 60, 0, 1, 4), group(1 / 60, 0, 1, 5), group(1 / 30, 0, 1, 6),
                  group(1 / 14, 1, 1, 1), group(1 / 30, 2, 1, 4, 1), group(1 / 30, 2, 1, 5, 2),
                  (t, 3, k, to, 1 + _poisson(g, 1, len(k)), 6, 0)], days)
    return model.SISe3(u0, np.arange(1, days + 1, dtype=float), phi=1.0,
                       upsilon_1=0.0357, upsilon_2=0.0357, upsilon_3=0.00935,
                       gamma_1=0.1, gamma_2=0.1, gamma_3=0.1, alpha=1.0,
                       beta_t1=0.19, beta_t2=0.085, beta_t3=0.075, beta_t4=0.185,
                       end_t1=91, end_t2=182, end_t3=273, end_t4=365, epsilon=0.0, events=ev)


def _pfilter(case, seed):
    """A SISe model with its environmental state, and weekly observations
    Binomial(I, 0.8) of a discretised ground truth."""
    rng = np.random.default_rng(seed)
    n, weeks = case["nodes"], case["weeks"]
    S = rng.poisson(100, n)
    I = rng.poisson(2, n) * (rng.random(n) < 0.05)
    u0 = np.vstack([S, I]).astype(np.int32)
    phi = np.zeros(n)
    obs = np.zeros((weeks, n), dtype=np.int32)
    for d in range(1, 7 * weeks + 1):
        up = rng.binomial(S, 1.0 - np.exp(-0.012 * phi))
        down = rng.binomial(I, 1.0 - np.exp(-0.1))
        S, I = S - up + down, I + up - down
        phi = phi * 0.97 + 0.05 * I / np.maximum(S + I, 1)
        if d % 7 == 0:
            obs[d // 7 - 1] = rng.binomial(I, 0.8)
    times = np.arange(7, 7 * weeks + 1, 7, dtype=np.int32)
    m = model.SISe_pf(u0, np.array([0.0]), upsilon=0.012, gamma=0.1)
    return rng, m, times, obs


def _consumers_U(case, seed):
    """A stored trajectory of four compartments, values as the SEIR workload
    leaves them mid-epidemic."""
    g = _gen(seed)
    n = case["nodes"] * case["columns"]
    U = torch.empty((n, 4), dtype=torch.int32, device="cuda")
    for c, lam in enumerate((250.0, 5.0, 15.0, 30.0)):
        U[:, c] = torch.poisson(torch.full((n,), lam, device="cuda"), generator=g).to(torch.int32)
    return U


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sir":
        # the configuration's 99 susceptible and 5 infected a node, jittered
        rng = np.random.default_rng(seed)
        n = case["nodes"]
        u0 = {"S": rng.poisson(99, n), "I": 1 + rng.poisson(4, n), "R": np.zeros(n)}
        return {"kind": kind, "seed": seed,
                "model": model.SIR_mparse(u0, np.arange(1, case["days"] + 1, dtype=float),
                                          beta=0.16, gamma=0.077)}
    if kind == "sise3":
        return {"kind": kind, "seed": seed, "model": _sise3(case["nodes"], case["days"], seed)}
    if kind == "seir":
        m = _seir(case["nodes"], case["days"], seed)
        if not case["resident"]:
            return {"kind": kind, "seed": seed, "model": m}
        if case["replicates"] > 1:
            m = m.replicate(case["replicates"])
        holder = abi.build_args(m, seed, solver=1 if case["solver"] == "aem" else 0)
        plan = native.Plan(holder, m.name, cap_transfers=True)
        return {"kind": "plan", "plan": plan}
    if kind in ("pfilter", "pmcmc"):
        rng, m, times, obs = _pfilter(case, seed)
        P = case["particles"]
        state = {"kind": kind, "seed": seed, "model": m, "particles": P, "times": times,
                 "obs": obs}
        if kind == "pfilter":
            state["gdata"] = np.column_stack([rng.uniform(0.005, 0.03, P),
                                              rng.uniform(0.05, 0.2, P)])
        else:
            state["iterations"] = case["iterations"]
        return state
    if kind == "abc":
        rng = np.random.default_rng(seed)
        # the mix of node counts and of horizons in fixed shares, so that a
        # case's work hardly depends on the seed
        sizes = [100, 1000, 100, 1000, 10_000, 100, 1000, 100, 10_000, 50_000]
        models = [_seir(sizes[j % 10], 60 + (j * 97) % 306, int(seed) * 1000 + j,
                        beta=rng.uniform(0.05, 0.5), epsilon=rng.uniform(0.1, 0.5),
                        gamma=rng.uniform(0.02, 0.2)) for j in range(case["proposals"])]
        t = np.arange(365)
        target = 0.12 * np.exp(-0.5 * ((t - 150) / 45.0) ** 2)
        return {"kind": kind, "models": models,
                "seeds": [int(s) for s in rng.integers(1, 2 ** 62, len(models))],
                "targets": [target[:len(m.tspan)] for m in models]}
    return {"kind": kind, "U": _consumers_U(case, seed), "nodes": case["nodes"],
            "columns": case["columns"]}


class _DeviceU:
    """A plan's U on the device, as torch takes foreign memory; holds the plan."""

    def __init__(self, plan):
        d = C.c_void_p()
        native.check(native.lib().siminf_gpu_plan_outputs(plan.handle, C.byref(d), None, None))
        a = plan.holder.args
        self.plan = plan
        self.__cuda_array_interface__ = {
            "shape": (a.Nrep * a.tlen, a.Nn * a.Nc), "typestr": "<i4", "version": 3,
            "data": (d.value, False), "strides": None}


def run(state):
    kind = state["kind"]
    if kind == "sir":
        return run_model(state["model"], seed=state["seed"]).U
    if kind in ("seir", "sise3"):
        res = run_model(state["model"], seed=state["seed"], cap_transfers=True)
        return {"U": res.U, "V": res.V} if kind == "sise3" else res.U
    if kind == "plan":
        state["plan"].run()
        return torch.as_tensor(_DeviceU(state["plan"]), device="cuda")
    if kind == "pfilter":
        r = pfilter(state["model"], state["particles"], state["times"], state["obs"], 1, 0.8,
                    seed=state["seed"], gdata=state["gdata"])
        return {"loglik": r.loglik, "ess": r.ess, "ancestors": r.ancestors}
    if kind == "pmcmc":
        chain = Pmcmc(state["model"], state["particles"], state["times"], state["obs"], 1, 0.8,
                      pars=[0, 1], theta=[0.012, 0.1], prior_lo=[0.001, 0.01],
                      prior_hi=[0.05, 0.5], covmat=np.diag([1e-6, 1e-5]), seed=state["seed"])
        rows = chain.run(state["iterations"])
        chain.close()
        return rows
    if kind == "abc":
        prev, dist = run_batch(state["models"], state["seeds"], state["targets"],
                               cap_transfers=True)
        return {"prevalence": np.concatenate(prev), "distance": dist}
    d_U, n, cols = state["U"].data_ptr(), state["nodes"], state["columns"]
    p1, _ = trajectory.prevalence_device(d_U, n, 4, cols, 0b0100, 0b1111, level=1)
    p2, _ = trajectory.prevalence_device(d_U, n, 4, cols, 0b0100, 0b1111, level=2)
    I, _ = trajectory.trajectory_device(d_U, n, 4, cols, [3])
    return {"prevalence": p1, "node_prevalence": p2, "I": I}


# ------------------------------------------------------------------
# What a pass cannot do without: event columns (36 B each) and initial
# states read once, the trajectory written once; a few flops a stored value
# stand for the transitions, whose number depends on the epidemic.
# ------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "sir":
        b = 4.0 * 3 * case["nodes"] * (case["days"] + 1)
    elif kind == "sise3":
        nd = case["nodes"] * case["days"]
        b = 32.0 * (nd + case["nodes"]) + 36.0 * nd * 0.25
    elif kind == "seir":
        nd = float(case["nodes"] * case["days"])
        R = case["replicates"]
        b = 16.0 * R * (nd + case["nodes"]) + 36.0 * nd * 0.504
    elif kind in ("pfilter", "pmcmc"):
        P, n, w = case["particles"], case["nodes"], case["weeks"]
        b = (16.0 * n + 4.0) * P * w * case.get("iterations", 1)
    elif kind == "abc":
        nd = case["proposals"] * 7240.0 * 212
        b = nd * 0.504 * 36.0
    else:
        n = float(case["nodes"] * case["columns"])
        b = 16.0 * n + 4.0 * n + 16.0 * case["columns"]
    return {"bytes": b, "flops": b / 4.0}


def exact(case, seed):
    """Prevalence and the long format are plain arithmetic on U; the
    simulations' outputs have no value without the simulation."""
    if case["kind"] != "consumers":
        return None
    U = _consumers_U(case, seed).reshape(case["columns"], case["nodes"], 4)
    total = U.sum(2, dtype=torch.int64)
    I = U[:, :, 2].to(torch.int64)
    p1 = I.sum(1).double() / total.sum(1).double()
    p2 = (I > 0).sum(1).double() / (total > 0).sum(1).double()
    return {"prevalence": p1.cpu().numpy(), "node_prevalence": p2.cpu().numpy(),
            "I": U[:, :, 2].reshape(1, -1).cpu().numpy()}
