"""The workloads this framework's speed is measured on.

Every case goes through the public Python API: a problem is created once (the
plan and its tables on the device, which a program keeps), and one pass is one
call a program makes on it: an anneal and the reading of its results, a batch
of anneals, a stream of requests through the server, or the energies of given
states. Sizes follow the framework's own benchmark, tests and examples.

A pass's branches are those of one Markov chain per branch, fixed by the
problem's sweep order and the counter-based draws: any change of one decision
gives another branch, so branches and integer energies are compared exactly.
"""
import numpy as np

from qublar_b200 import (OPT_DEFER_UPLOAD, OPT_RESID_CLUSTER, Budget, IsingProblem, QuboProblem, ResidualProblem,
                         Schedule, Server, autotune_batch, branch_fractions, run_batch, solve_batch, synth)


def listed():
    return [
        # The smallest call: the complete 16-spin graph of the engine's self-check, annealed
        # for its ground state. Launches and the host's part of a call count.
        {"name": "maxcut_k16", "kind": "maxcut", "graph": "complete", "n": 16, "wmax": 15, "replicas": 32, "sweeps": 100},
        # The plain method's headline size: ER(800, 0.06), 16 replicas, 1000 sweeps.
        {"name": "maxcut_er800", "kind": "maxcut", "graph": "er", "n": 800, "degree": 48, "replicas": 16, "sweeps": 1000},
        # The same graph for time-to-solution statistics: thousands of replicas at once.
        {"name": "maxcut_er800_wide", "kind": "maxcut", "graph": "er", "n": 800, "degree": 48, "replicas": 4096,
         "sweeps": 300},
        # Integer weights that need 32 bits, odd sizes (the tests' signed sparse graphs).
        {"name": "maxcut_signed", "kind": "maxcut", "graph": "sparse", "n": 3001, "degree": 8, "wmax": 1000,
         "replicas": 50, "sweeps": 400},
        # A sparse graph too large for a CTA's shared memory (the serving mix's large Max-Cut).
        {"name": "maxcut_60k", "kind": "maxcut", "graph": "regular", "n": 60000, "degree": 5, "replicas": 32,
         "sweeps": 100},
        # A detector study: a small pyramid, branch fractions of an odd number of branches.
        {"name": "tomography_small", "kind": "tomography", "bits": 5000, "branches": 24, "anneal": 200, "hold": 50},
        # The tomography headline: 306,328 bits, 75,594 rays, 16 branches, the posterior schedule.
        {"name": "tomography_pyramid", "kind": "tomography", "bits": 306328, "branches": 16, "anneal": 200, "hold": 50},
        # A weighted QUBO of the size of the sequencing study's instances.
        {"name": "qubo_small", "kind": "qubo", "graph": "random", "n": 120, "degree": 12, "replicas": 64, "sweeps": 1000},
        # The precision headline's problem: N = 200,000, a 58^3 lattice with long-range edges
        # of average degree 20, 64 replicas; a fifth of its 5000 sweeps, the same temperatures.
        {"name": "qubo_lattice", "kind": "qubo", "graph": "lattice", "n": 200000, "side": 58, "degree": 20,
         "replicas": 64, "sweeps": 1000},
        # The batching headline's mix (tori and d-regular graphs, N log-uniform, 32 replicas),
        # fewer instances and sweeps, the launch shape autotuned once.
        {"name": "batch_mixed", "kind": "batch", "instances": 128, "n_min": 200, "n_max": 20000, "replicas": 32,
         "sweeps": 200, "tuned": True},
        # A short stream of the serving mix through one server, everything submitted at once.
        {"name": "serve_mixed", "kind": "serve", "requests": 8, "n_min": 1000, "n_max": 60000, "sweeps": 200},
        # The energies of given states from scratch, in fp64 (the check of returned branches).
        {"name": "score_pyramid", "kind": "score", "form": "residual", "n": 40000, "states": 33},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["maxcut", "maxcut", "tomography", "tomography", "qubo", "qubo", "batch", "serve", "score"])
    if kind == "maxcut":
        graph = rng.choice(["complete", "er", "sparse", "regular", "torus"])
        n = {"complete": _log(rng, 8, 200), "er": _log(rng, 200, 2000), "sparse": _log(rng, 100, 20000),
             "regular": _log(rng, 200, 60000), "torus": _log(rng, 9, 200) ** 2}[graph]
        degree = min(n - 1, {"complete": n - 1, "er": rng.randint(8, 60), "sparse": rng.randint(3, 16),
                             "regular": rng.randint(3, 50), "torus": 4}[graph])
        sweeps = _log(rng, 50, 1000)
        # about the largest listed case's attempts and neighbour updates at most
        most = max(1, int(1.5e9 / (n * sweeps)))
        return {"kind": kind, "graph": graph, "n": n, "degree": degree,
                "wmax": rng.choice([1, 7, 100, 1000]) if graph in ("complete", "sparse") else 1,
                "replicas": min(most, _log(rng, 1, 8192)), "sweeps": sweeps}
    if kind == "tomography":
        bits = _log(rng, 300, 200000)
        sweeps = min(400, int(4e9 / (bits * 64)) + 20)
        hold = rng.randint(0, sweeps // 4)
        return {"kind": kind, "bits": bits, "branches": _log(rng, 1, 64 if bits < 100000 else 16),
                "anneal": sweeps - hold, "hold": hold}
    if kind == "qubo":
        graph = rng.choice(["random", "lattice"])
        side = rng.randint(5, 50)
        n = _log(rng, 20, 3000) if graph == "random" else side ** 3 + rng.randint(0, 500)
        sweeps = min(_log(rng, 100, 1500), int(1.2e8 / n) + 20)
        return {"kind": kind, "graph": graph, "n": n, "side": side,
                "degree": rng.randint(3, min(16, n // 2)) if graph == "random" else rng.randint(8, 24),
                "replicas": _log(rng, 1, 150 if n < 20000 else 64), "sweeps": sweeps}
    if kind == "batch":
        n_min = _log(rng, 50, 1000)
        return {"kind": kind, "instances": _log(rng, 4, 128), "n_min": n_min, "n_max": _log(rng, n_min, 20000),
                "replicas": _log(rng, 4, 48), "sweeps": _log(rng, 30, 200), "tuned": rng.random() < 0.5}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(2, 8), "n_min": 1000, "n_max": _log(rng, 2000, 60000),
                "sweeps": rng.randint(50, 200)}
    return {"kind": "score", "form": rng.choice(["residual", "qubo", "ising"]), "n": _log(rng, 500, 100000),
            "states": _log(rng, 1, 64)}


# ---- inputs ------------------------------------------------------------------------------------

def _pairs(n, m, rng):
    """m distinct pairs u < v of n vertices."""
    m = min(m, n * (n - 1) // 2)
    keys = np.zeros(0, np.int64)
    while keys.size < m:
        a = rng.integers(0, n, size=(int(1.2 * (m - keys.size)) + 16, 2))
        a = np.sort(a[a[:, 0] != a[:, 1]], axis=1)
        keys = np.unique(np.concatenate([keys, a[:, 0] * n + a[:, 1]]))
    keys = np.sort(rng.permutation(keys)[:m])
    return (keys // n).astype(np.int32), (keys % n).astype(np.int32)


def _graph(case, seed):
    """(n, eu, ev, ew) of an integer Max-Cut case."""
    kind, n = case["graph"], int(case["n"])
    rng = np.random.default_rng(seed)
    if kind == "complete":
        return synth.random_complete(n, int(case["wmax"]), seed + 1)
    if kind == "er":
        return synth.erdos_renyi(n, case["degree"] / n, seed + 1)
    if kind == "torus":
        return synth.torus_pm1(int(round(n ** 0.5)), seed + 1)
    if kind == "regular":
        return synth.random_regular(n, int(case["degree"]), seed + 1)
    eu, ev = _pairs(n, n * int(case["degree"]) // 2, rng)
    wmax = int(case["wmax"])
    return n, eu, ev, (rng.integers(1, wmax + 1, eu.size) * rng.choice([-1, 1], eu.size)).astype(np.int32)


def _lattice(n, side, degree, rng):
    """A periodic side^3 lattice plus random long-range edges to the average degree over n sites."""
    idx = np.arange(side ** 3).reshape(side, side, side)
    lat = np.concatenate([np.stack([idx.ravel(), np.roll(idx, -1, axis=a).ravel()], 1) for a in range(3)])
    lat = np.sort(lat, axis=1)
    keys = np.unique(lat[:, 0].astype(np.int64) * n + lat[:, 1])
    need = n * degree // 2 - keys.size
    if need > 0:
        a = np.sort(rng.integers(0, n, size=(need + need // 20 + 64, 2)), axis=1)
        far = np.setdiff1d(a[a[:, 0] != a[:, 1]] @ np.array([n, 1]), keys)
        keys = np.concatenate([keys, rng.permutation(far)[:need]])
    return (keys // n).astype(np.int32), (keys % n).astype(np.int32)


def _qubo(case, seed):
    """{n, eu, ev, ew, h, offset}: couplings and linear terms N(0, 1) in fp32."""
    rng = np.random.default_rng(seed)
    n = int(case["n"])
    if case["graph"] == "lattice":
        eu, ev = _lattice(n, int(case["side"]), int(case["degree"]), rng)
    else:
        eu, ev = _pairs(n, n * int(case["degree"]) // 2, rng)
    return {"n": n, "eu": eu, "ev": ev, "ew": rng.standard_normal(eu.size).astype(np.float32),
            "h": rng.standard_normal(n).astype(np.float32), "offset": 0.0}


def _pyramid(bits, seed):
    """The tomography problem's arrays: the headline's pyramid, or one scaled to about `bits` bits."""
    seed = 20260929 + seed
    if bits == 306328:
        return synth.tomography(synth.tomo_params(seed=seed), device=0)
    scale = (max(bits, 300) / 312000.0) ** (1.0 / 3.0)
    return synth.tomography(synth.small_tomo_params(scale, max(8, int(round(120 * scale))), seed=seed), device=0)


def _score_data(case, seed):
    rng = np.random.default_rng(seed + 99)
    n, form = int(case["n"]), case["form"]
    if form == "residual":
        data = _pyramid(n, seed)
        n = data["row_ptr"].size - 1
    elif form == "qubo":
        data = _qubo({"n": n, "graph": "random", "degree": 8}, seed)
    else:
        data = _graph({"n": n, "graph": "sparse", "degree": 8, "wmax": 1000}, seed)
    return data, (rng.random((int(case["states"]), n)) < 0.3).astype(np.uint8)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "maxcut":
        P = IsingProblem(*_graph(case, seed), device=0)
        if case["graph"] == "er":
            sched = Budget(3.0, 0.05, case["sweeps"], 0)
        else:
            sched = P.scaled_schedule(case["sweeps"] - case["sweeps"] // 20, case["sweeps"] // 20)
        return {"kind": kind, "problem": P, "schedule": sched, "branches": int(case["replicas"])}
    if kind == "tomography":
        P = ResidualProblem.from_arrays(_pyramid(int(case["bits"]), seed), device=0)
        return {"kind": kind, "problem": P, "schedule": Schedule(50.0, 1.0, case["anneal"], case["hold"], 50),
                "branches": int(case["branches"])}
    if kind == "qubo":
        P = QuboProblem.from_dict(_qubo(case, seed), device=0)
        hold = case["sweeps"] // 10
        return {"kind": kind, "problem": P, "schedule": Schedule(3.0, 0.05, case["sweeps"] - hold, hold, 64),
                "branches": int(case["replicas"])}
    if kind == "batch":
        # the benchmark's sizes, another graph of each per seed
        items = []
        specs = synth.mixed_batch_specs(int(case["instances"]), 2026, case["n_min"], case["n_max"])
        for k, (form, n, degree, sub) in enumerate(specs):
            P = IsingProblem(*synth.build_spec((form, n, degree, sub + seed)), device=0)
            items.append((P, P.scaled_schedule(case["sweeps"], 0), int(case["replicas"]), 1000 * k))
        return {"kind": kind, "items": items, "config": autotune_batch(items) if case["tuned"] else None}
    if kind == "serve":
        # the benchmark's sizes and schedules, another problem of each per seed
        requests = []
        specs = synth.serve_specs(int(case["requests"]), 77, case["n_min"], case["n_max"])
        for k, sp in enumerate(specs):
            sp["seed"] += seed
            sweeps = max(20, sp["sweeps"] * int(case["sweeps"]) // 2750)
            if sp["kind"] == "tomography":
                flags = OPT_DEFER_UPLOAD | (0 if sp["n"] >= 10000 else OPT_RESID_CLUSTER)
                P = ResidualProblem.from_arrays(_pyramid(sp["n"], seed + k), device=0, flags=flags)
                sched = Schedule(50.0, 1.0, sweeps - sweeps // 5, sweeps // 5, 50)
            else:
                P = IsingProblem(*synth.build_request(sp), device=0, flags=OPT_DEFER_UPLOAD)
                sched = P.scaled_schedule(sweeps, 0)
            requests.append((P, sched, int(sp["branches"]), k))
        return {"kind": kind, "server": Server(device=0), "requests": requests}
    data, X = _score_data(case, seed)
    if case["form"] == "residual":
        P = ResidualProblem.from_arrays(data, device=0)
    elif case["form"] == "qubo":
        P = QuboProblem.from_dict(data, device=0)
    else:
        P = IsingProblem(*data, device=0)
    return {"kind": kind, "problem": P, "X": X}


# ---- one pass ----------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "maxcut":
        out = run_batch(state["problem"], state["schedule"], 1, state["branches"])
        return {"x": out.X, "energy": out.energy}
    if kind == "tomography":
        frac, x = branch_fractions(state["problem"], state["schedule"], state["branches"], keep=True)
        return {"fraction": frac, "x": x}
    if kind == "qubo":
        r = state["problem"].solve(state["schedule"], state["branches"])
        try:
            return {"x": r.branches(), "energy": r.energies()}
        finally:
            r.close()
    if kind == "batch":
        b = solve_batch(state["items"], state["config"])
        try:
            count = range(len(state["items"]))
            return {"x": np.concatenate([b.branches(k).ravel() for k in count]),
                    "energy": np.concatenate([b.energies_tracked(k) for k in count]),
                    "fraction": np.concatenate([b.marginals(k) for k in count])}
        finally:
            b.close()
    if kind == "serve":
        S = state["server"]
        ids = [S.submit(P, sched, R, off) for P, sched, R, off in state["requests"]]
        out = []
        for i in ids:
            S.wait(i)
            out.append({"x": S.branches(i), "energy": S.energies(i), "fraction": S.marginals(i)})
            S.release(i)
        return out
    return state["problem"].energies(state["X"])


# ---- what a pass cannot do without -------------------------------------------------------------

# Operations of one attempt beside its sums: half a ten-round Philox block of eight
# operations a round, and the Metropolis test.
_ATTEMPT = 50


def _graph_work(n, degree, replicas, sweeps):
    nnz = n * degree
    return {"bytes": nnz * 8 + n * 8 + replicas * (n + 8),
            "flops": float(replicas) * sweeps * n * _ATTEMPT + replicas * nnz}


def _tomography_work(bits, branches, sweeps):
    # straight chords through a cube of `bits` cells cross about 2 cube roots of cells per
    # ray, and there is about one ray for every four cells of the headline pyramid
    scale = (bits / 312000.0) ** (1.0 / 3.0)
    nnz = 10.9e6 * scale ** 3
    return {"bytes": nnz * 8 + bits * 40 + branches * bits + bits * 4,
            "flops": float(branches) * sweeps * (bits * _ATTEMPT + 2 * nnz)}


def _mean_size(case):
    """The mean of a log-uniform size."""
    lo, hi = case["n_min"], case["n_max"]
    return float((hi - lo) / np.log(hi / lo)) if hi > lo else float(lo)


def work(case):
    kind = case["kind"]
    if kind == "maxcut":
        return _graph_work(case["n"], case["degree"] if "degree" in case else case["n"] - 1, case["replicas"],
                           case["sweeps"])
    if kind == "tomography":
        return _tomography_work(case["bits"], case["branches"], case["anneal"] + case["hold"])
    if kind == "qubo":
        return _graph_work(case["n"], case["degree"], case["replicas"], case["sweeps"])
    if kind == "batch":
        mean = _mean_size(case)
        w = _graph_work(mean, 15, case["replicas"], case["sweeps"])
        return {k: v * case["instances"] for k, v in w.items()}
    if kind == "serve":
        mean = _mean_size(case)
        a = _graph_work(mean, 7.5, 20, case["sweeps"])
        b = _tomography_work(mean, 20, case["sweeps"])
        return {k: float(case["requests"]) * (a[k] + b[k]) / 2 for k in a}
    n, K = case["n"], case["states"]
    nnz = n * 36 if case["form"] == "residual" else n * 4
    return {"bytes": float(nnz * 12 + n * K + 8 * K), "flops": float(2 * nnz * K)}


def tolerance(case):
    if case["kind"] in ("maxcut", "batch") or (case["kind"] == "score" and case["form"] == "ising"):
        return "exact"   # bits, integer energies, exact counts over the replicas
    # fp64 energies, summed in another order: 2e-15 seen between summation orders. Bits may
    # not differ at all.
    return {"rel": 1e-13, "max": 1e-12}


def exact(case, seed):
    """The energies of given states in fp64. The solves have none: their
    branches follow from the framework's own sweep order and draws."""
    if case["kind"] != "score":
        return None
    data, X = _score_data(case, seed)
    if case["form"] == "ising":
        _, eu, ev, ew = data
        return np.array([-int(np.sum(ew.astype(np.int64) * (x[eu] != x[ev]))) for x in X], np.int64)
    if case["form"] == "qubo":
        J, h = data["ew"].astype(np.float64), data["h"].astype(np.float64)
        return np.array([data["offset"] + np.sum(h * x) + np.sum(J * (x[data["eu"]] & x[data["ev"]])) for x in X])
    n = X.shape[1]
    bit = np.repeat(np.arange(n), np.diff(data["row_ptr"]))
    of = np.repeat(np.arange(n), np.diff(data["nbr_ptr"]))
    once = data["nbr"] > of
    u, v = of[once], data["nbr"][once]
    e = []
    for x in X:
        r = np.bincount(data["ray"], data["a"].astype(np.float64) * x[bit], minlength=data["d"].size) - data["d"]
        e.append(0.5 * np.sum(data["w"] * r * r) + data["kappa"] * np.sum(x, dtype=np.float64) +
                 data["lambda"] * np.count_nonzero(x[u] != x[v]))
    return np.array(e)
