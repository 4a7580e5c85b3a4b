"""The few-replica integer sweep (draws reduced to the largest accepted dE,
off the sweep's chain) against the CTA-per-replica sweep and the oracle, bit
for bit: tiny and wide classes, a warp per flip and a lane per flip, helper
CTAs, an adjacency too large for shared memory, couplings from 1 to 10^6 (both
precisions of the limit's logarithm), and the per-sweep trace."""
import numpy as np
import pytest

from oracle import oracle as O
from qublar_b200 import IsingProblem, Schedule, sweep_launches, synth

pytestmark = pytest.mark.gpu


def _sparse(n, m, wmax, seed):
    rng = np.random.default_rng(seed)
    keys = np.unique(rng.integers(0, n, 2 * m) * n + rng.integers(0, n, 2 * m))
    u, v = keys // n, keys % n
    keep = u < v
    u, v = u[keep][:m], v[keep][:m]
    w = rng.integers(1, wmax + 1, u.size) * rng.choice([-1, 1], u.size)
    return n, u.astype(np.int32), v.astype(np.int32), w.astype(np.int32)


CASES = {
    "k16": (lambda: synth.random_complete(16, 15, 3), 32, 60, "ising_dense"),
    "two": (lambda: (2, np.array([0], np.int32), np.array([1], np.int32), np.array([5], np.int32)), 3, 20, "ising_dense"),
    "er": (lambda: synth.erdos_renyi(300, 0.16, 2), 5, 80, "ising_replica_w8"),
    "er_no_helpers": (lambda: synth.erdos_renyi(300, 0.16, 2), 148, 20, "ising_replica_w8"),
    "dense_1000": (lambda: synth.random_complete(121, 1000, 7), 4, 60, "ising_dense"),
    "dense_1e6": (lambda: synth.random_complete(65, 1000000, 7), 4, 60, "ising_dense"),
    "dense_33": (lambda: synth.random_complete(33, 7, 1), 200, 30, "ising_dense"),
    "dense_128": (lambda: synth.random_complete(128, 1, 2), 3, 30, "ising_dense"),
    "dense_224": (lambda: synth.random_complete(224, 500, 2), 3, 17, "ising_dense"),
    "torus": (lambda: synth.torus_pm1(30, 3), 7, 50, "ising_replica_w8"),
    "dense_many": (lambda: synth.random_complete(50, 1, 3), 700, 20, "ising_dense"),
    "sparse_helpers": (lambda: _sparse(3001, 12000, 900, 5), 3, 40, "ising_replica_w32"),
    "sparse_two_ctas": (lambda: _sparse(2001, 9000, 100, 6), 60, 20, "ising_replica_w8"),
    "sparse_no_helpers": (lambda: _sparse(6001, 9000, 900, 6), 100, 12, "ising_replica_w32"),
    "long_rows_w8": (lambda: synth.random_regular(2000, 100, 8), 2, 12, "ising_replica_w8_far"),
    "long_rows_w32": (lambda: _sparse(801, 19000, 900, 8), 2, 12, "ising_replica_w32_far"),
}


@pytest.mark.parametrize("name", list(CASES))
def test_equals_the_cta_per_replica_sweep_and_the_oracle(name, monkeypatch):
    make, R, sweeps, kernel = CASES[name]
    g = make()
    P = IsingProblem(*g)
    s = P.scaled_schedule(sweeps, 3)
    before = sweep_launches(kernel), sweep_launches("ising_fields")
    r = P.solve(s, R, 9, trace=True)
    monkeypatch.setenv("QB_ISING_THREADS", "512")
    o = P.solve(s, R, 9, trace=True)
    assert (sweep_launches(kernel), sweep_launches("ising_fields")) == (before[0] + 1, before[1] + 1)
    monkeypatch.delenv("QB_ISING_THREADS")
    assert (r.branches() == o.branches()).all() and (r.fields() == o.fields()).all()
    assert (r.energies_tracked() == o.energies_tracked()).all() and (r.energies() == o.energies()).all()
    assert (r.energy_trace() == o.energy_trace()).all()
    G = O.Graph(*g)
    order, _ = P.colouring()
    temps = O.temperatures(s.t_hot, s.t_cold, s.anneal_sweeps, s.hold_sweeps)
    for k in (0, R - 1):
        key, half = O.ising_key_half(k, 9)
        x, f, e = G.anneal_coloured(order, temps, key, half=half)
        assert (r.branches()[k] == x).all() and r.energies_tracked()[k] == e


@pytest.mark.parametrize("t", [1e-3, 0.7, 4095.0, 4097.0, 3e7, 2.0 ** 39, 2.0 ** 40, 1.0001 * 2.0 ** 40, 1e16])
def test_temperatures_of_every_size(t, monkeypatch):
    """Both precisions of the limit's logarithm; above 2^40 the CTA-per-replica sweep."""
    g = synth.random_complete(40, 20000, 1)
    P = IsingProblem(*g)
    s = Schedule(t, t / 3, 25, 2, 0)
    kernel = "ising_dense" if t <= 2.0 ** 40 else "ising_fields"
    before = sweep_launches(kernel)
    r = P.solve(s, 6)
    assert sweep_launches(kernel) == before + 1
    monkeypatch.setenv("QB_ISING_THREADS", "64")
    o = P.solve(s, 6)
    assert (r.branches() == o.branches()).all() and (r.energies_tracked() == o.energies_tracked()).all()


@pytest.mark.parametrize("R,kernel", [(148, "ising_dense"), (200, "ising_fields"), (1500, "ising_fields")])
def test_dense_graphs_leave_the_dense_kernel_where_its_waves_are_longer(R, kernel):
    """200 bits in 34 classes: one CTA of the dense kernel fills an SM, so beyond
    one replica per SM the CTA-per-replica sweep's class chain is shorter."""
    n, eu, ev, ew = synth.erdos_renyi(200, 0.5, 3)
    P = IsingProblem(n, eu, ev, np.where(np.arange(ew.size) % 2, 90, -ew).astype(np.int32))
    s = P.scaled_schedule(20, 2)
    before = sweep_launches(kernel)
    r = P.solve(s, R, 3)
    assert sweep_launches(kernel) == before + 1
    G = O.Graph(n, eu, ev, np.where(np.arange(ew.size) % 2, 90, -ew).astype(np.int32))
    order, _ = P.colouring()
    temps = O.temperatures(s.t_hot, s.t_cold, s.anneal_sweeps, s.hold_sweeps)
    for k in (0, R - 1):
        key, half = O.ising_key_half(k, 3)
        x, _, e = G.anneal_coloured(order, temps, key, half=half)
        assert (r.branches()[k] == x).all() and r.energies_tracked()[k] == e


def test_replicas_with_helper_ctas_run_in_one_wave():
    """Sixteen clusters of eight CTAs do not fit the device at once: a second
    wave of clusters would double the time of eight replicas."""
    P = IsingProblem(*_sparse(4001, 8000, 1, 4))
    s = P.scaled_schedule(300, 0)
    ms, before = {}, sweep_launches("ising_replica_w8")
    for R in (8, 16):
        t = []
        for _ in range(5):
            r = P.solve(s, R, 0)
            t.append(r.info().anneal_ms)
            r.close()
        ms[R] = min(t)
    assert sweep_launches("ising_replica_w8") == before + 10
    assert ms[16] < 1.5 * ms[8], ms


@pytest.mark.parametrize("make,R,kernel", [
    (lambda: synth.erdos_renyi(500, 0.6, 3), 5, "ising_fields"),            # rows of 300, adjacency off chip
    (lambda: synth.random_regular(2000, 100, 3), 5, "ising_replica_w8_far"),
    (lambda: _sparse(2001, 9000, 100, 6), 100, "ising_fields"),             # wide classes, no SM for helpers
    (lambda: _sparse(2001, 9000, 100, 6), 60, "ising_replica_w8"),
    (lambda: _sparse(6001, 9000, 900, 6), 100, "ising_replica_w32"),
])
def test_the_few_replica_sweep_is_taken_where_it_pays(make, R, kernel, monkeypatch):
    P = IsingProblem(*make())
    s = P.scaled_schedule(12, 1)
    before = sweep_launches(kernel)
    r = P.solve(s, R, 4)
    assert sweep_launches(kernel) == before + 1
    monkeypatch.setenv("QB_ISING_THREADS", "256")
    o = P.solve(s, R, 4)
    assert (r.branches() == o.branches()).all() and (r.fields() == o.fields()).all()
    assert (r.energies_tracked() == o.energies_tracked()).all()
