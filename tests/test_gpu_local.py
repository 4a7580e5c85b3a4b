"""The residual sweep with a CTA per branch against the lockstep and the cluster
sweep and the oracle, bit for bit: empty and single rays, bits without rays, bits of one to
more than sixteen segments, more branches than SMs, negative weights, long
neighbour lists, the refresh, traces."""
import numpy as np
import pytest

from oracle import oracle as O
from qublar_b200 import OPT_RESID_CLUSTER, ResidualProblem, Schedule, sweep_launches, synth

pytestmark = pytest.mark.gpu


def _random(n, rays, degrees, seed, nbrs=3):
    """Bits with the given numbers of rays (cycled), a ring of neighbours, some negative weights."""
    rng = np.random.default_rng(seed)
    row, ray, a = [0], [], []
    for i in range(n):
        k = min(rays, degrees[i % len(degrees)])
        ray += list(rng.choice(rays, k, replace=False))
        a += list(rng.uniform(0.05, 0.4, k))
        row.append(len(ray))
    nb = [[] for _ in range(n)]
    for i in range(n):
        for s in range(1, nbrs + 1):
            j = (i + s) % n
            if j != i and j not in nb[i]:
                nb[i].append(j)
                nb[j].append(i)
    ptr = np.cumsum([0] + [len(v) for v in nb])
    w = rng.uniform(0.5, 3.0, rays) * rng.choice([1.0, 1.0, 1.0, -1.0], rays)
    return {"d": rng.uniform(0.0, 1.0, rays), "w": w, "row_ptr": np.array(row, np.int32),
            "ray": np.array(ray, np.int32), "a": np.array(a, np.float32), "nbr_ptr": ptr.astype(np.int32),
            "nbr": np.array([j for v in nb for j in v], np.int32), "lambda": 0.3, "kappa": 0.4, "field": None}


CASES = {
    "exhaustive16": (synth.exhaustive16, 20, 60),
    "pyramid": (lambda: synth.tomography(synth.small_tomo_params(0.16, 16)), 9, 70),
    "edges": (lambda: _random(230, 600, [0, 1, 2, 15, 16, 17, 31, 32, 33, 48, 200, 255, 256, 257, 300, 530], 4), 5, 25),
    "one_ray": (lambda: _random(12, 1, [1, 0], 2, 1), 3, 30),
    "long_neighbours": (lambda: _random(90, 40, [3, 20], 6, 14), 4, 40),
    "many_branches": (lambda: _random(60, 30, [4, 9], 7), 331, 30),
}


@pytest.mark.parametrize("order", ["lockstep", "cluster"])
@pytest.mark.parametrize("name", list(CASES))
def test_equals_the_planned_sweep_and_the_oracle(name, order, monkeypatch):
    make, R, sweeps = CASES[name]
    arr = make()
    P = ResidualProblem.from_arrays(arr, flags=OPT_RESID_CLUSTER if order == "cluster" else 0)
    s = Schedule(20.0, 0.6, sweeps, 6, 11)
    names = ["resid_local_cluster", "resid_cluster"] if order == "cluster" else ["resid_local"] + [f"resid_lockstep_{k}" for k in (1, 2, 3, 4)]
    before = [sweep_launches(k) for k in names]
    monkeypatch.setenv("QB_RESID_KERNEL", "local")
    r = P.solve(s, R, 3, trace=True)
    u = P.solve(s, R, 3)   # without the trace: class barriers across sweeps too
    assert (u.branches() == r.branches()).all()
    monkeypatch.setenv("QB_RESID_KERNEL", order)
    o = P.solve(s, R, 3, trace=True)
    ran = [sweep_launches(k) - b for k, b in zip(names, before)]
    assert ran[0] == 2 and sum(ran[1:]) == (1 if order == "cluster" else (R + 63) // 64)
    monkeypatch.delenv("QB_RESID_KERNEL")
    X = r.branches()
    assert (X == o.branches()).all() and (r.marginals() == o.marginals()).all()
    assert np.array_equal(r.energies(), o.energies())
    a, b = r.info(), o.info()
    assert a.accepted == b.accepted and a.max_drift == b.max_drift
    scale = np.maximum(1.0, np.abs(o.energy_trace()).max())
    assert np.abs(r.energy_trace() - o.energy_trace()).max() <= 1e-12 * sweeps * scale   # fp64 sums in another order
    visits, _ = P.colouring()
    temps = O.temperatures(s.t_hot, s.t_cold, s.anneal_sweeps, s.hold_sweeps)
    for k in (0, R - 1):
        x, _ = O.resid_anneal_coloured(arr, visits, temps, s.refresh_sweeps, k + 4, mode=P.info().variant)
        assert (X[k] == x).all(), k


@pytest.mark.parametrize("make,R,kernel", [
    (lambda: _random(40, 1200, [1000], 3, 0), 16, "resid_cluster"),          # a warp would walk 1,000 rays
    (lambda: _random(400, 900, [2], 3, 24), 149, "resid_cluster"),           # 48 neighbours, two waves of branches
    (lambda: _random(400, 900, [2], 3, 24), 16, "resid_local_cluster"),
    (lambda: _random(60, 300, [20], 3), 16, "resid_local_cluster"),
])
def test_cluster_plans_take_the_local_sweep_where_it_pays(make, R, kernel, monkeypatch):
    P = ResidualProblem.from_arrays(make(), flags=OPT_RESID_CLUSTER)
    s = Schedule(20.0, 0.6, 20, 2, 7)
    before = sweep_launches(kernel)
    r = P.solve(s, R, 3)
    assert sweep_launches(kernel) == before + 1
    monkeypatch.setenv("QB_RESID_KERNEL", "cluster" if "local" in kernel else "local")
    assert (P.solve(s, R, 3).branches() == r.branches()).all()


def test_a_forced_cluster_size_is_the_cluster_sweep(monkeypatch):
    monkeypatch.setenv("QB_RESID_CLUSTER", "4")
    P = ResidualProblem.from_arrays(_random(60, 300, [20], 3), flags=OPT_RESID_CLUSTER)
    s = Schedule(20.0, 0.6, 20, 2, 7)
    before = sweep_launches("resid_cluster")
    x = P.solve(s, 5, 3).branches()
    assert sweep_launches("resid_cluster") == before + 1
    monkeypatch.delenv("QB_RESID_CLUSTER")
    assert (P.solve(s, 5, 3).branches() == x).all()
