"""The word sweep (graphs of one coupling size: replicas as the bits of a word)
against the field-carrying sweeps and the oracle, bit for bit.

Sizes sit where the kernel's index arithmetic can go wrong: degrees around the
16 neighbours of a register, bits without neighbours, class tails, replica
counts that do not fill a unit, couplings other than 1, and the two widths of
the adjacency (32,768 bits).
"""
import numpy as np
import pytest

from oracle import oracle as O
from qublar_b200 import Budget, IsingProblem, solve_batch, sweep_launches, synth

pytestmark = pytest.mark.gpu


def _star_graph(n, degrees, w, seed):
    """Bit k of the first len(degrees) has degrees[k] neighbours of its own
    among the rest; the remaining bits have at most one."""
    rng = np.random.default_rng(seed)
    eu, ev, at = [], [], len(degrees)
    for k, d in enumerate(degrees):
        eu += [k] * d
        ev += list(range(at, at + d))
        at += d
    assert at <= n
    return n, np.array(eu, np.int32), np.array(ev, np.int32), (w * rng.choice([-1, 1], len(eu))).astype(np.int32)


GRAPHS = {
    "degrees": lambda: _star_graph(400, [0, 1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 64], 1, 3),
    "w7": lambda: (lambda g: (g[0], g[1], g[2], 7 * g[3]))(synth.random_regular(203, 9, 5)),
    "torus": lambda: synth.torus_pm1(19, 8),
    "dense": lambda: synth.erdos_renyi(90, 0.6, 4),
    "two": lambda: (2, np.array([0], np.int32), np.array([1], np.int32), np.array([-3], np.int32)),
}


@pytest.mark.parametrize("R", [4, 7, 16, 33, 70])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_words_equal_the_oracle(name, R):
    g = GRAPHS[name]()
    P = IsingProblem(*g)
    s = P.scaled_schedule(30, 4)
    before = sweep_launches("ising_word_16")
    B = solve_batch([(P, s, R, 6)])
    assert sweep_launches("ising_word_16") == before + 1
    X, E, F = B.branches(0), B.energies_tracked(0), B.fields(0)
    G = O.Graph(*g)
    order, _ = P.colouring()
    temps = O.temperatures(s.t_hot, s.t_cold, s.anneal_sweeps, s.hold_sweeps)
    for r in sorted({0, 1, R // 2, R - 1}):
        key, half = O.ising_key_half(r, 6)
        x, f, e = G.anneal_coloured(order, temps, key, half=half)
        assert (X[r] == x).all() and E[r] == e, r
    for r in range(R):
        assert E[r] == -G.cut(X[r]) and (F[r] == G.fields(X[r])).all()
    B.close()


@pytest.mark.parametrize("R", [32, 29, 16, 8, 4])
@pytest.mark.parametrize("name", ["degrees", "w7", "torus"])
def test_every_unit_width_equals_the_oracle(name, R):
    """Enough instances that none is split: units of 32, 16, 8 and 4 replicas."""
    g = GRAPHS[name]()
    P = IsingProblem(*g)
    s = P.scaled_schedule(12, 2)
    B = solve_batch([(P, s, R, 64 * k) for k in range(700)])
    assert B.info().work_items == 700
    G = O.Graph(*g)
    order, _ = P.colouring()
    temps = O.temperatures(s.t_hot, s.t_cold, s.anneal_sweeps, s.hold_sweeps)
    for k in (0, 311, 699):
        X, E, F = B.branches(k), B.energies_tracked(k), B.fields(k)
        for r in range(R):
            key, half = O.ising_key_half(r, 64 * k)
            x, f, e = G.anneal_coloured(order, temps, key, half=half)
            assert (X[r] == x).all() and E[r] == e and (F[r] == f).all(), (k, r)
    B.close()


@pytest.mark.parametrize("n", [32767, 32768, 32769])
def test_both_adjacency_widths_equal_the_field_sweep(n, monkeypatch):
    g = synth.random_regular(n, 5, 11)
    P = IsingProblem(*g)
    s = P.scaled_schedule(8, 1)
    kernel = "ising_word_16" if n <= 32768 else "ising_word_32"
    before = sweep_launches(kernel), sweep_launches("ising_fields")
    B = solve_batch([(P, s, 10, 0)])
    monkeypatch.setenv("QB_ISING_THREADS", "512")
    r = P.solve(s, 10)
    assert (sweep_launches(kernel), sweep_launches("ising_fields")) == (before[0] + 1, before[1] + 1)
    assert (B.branches(0) == r.branches()).all()
    assert (B.energies_tracked(0) == r.energies_tracked()).all() and (B.fields(0) == r.fields()).all()


@pytest.mark.parametrize("R", [149, 301, 1200])
def test_many_replicas_equal_the_cta_per_replica_sweep(R, monkeypatch):
    g = synth.random_regular(331, 21, 2)
    P = IsingProblem(*g)
    b = Budget(6.0, 0.2, 40, 3)
    before = sweep_launches("ising_word_16"), sweep_launches("ising_fields")
    r = P.solve(b, R, 4)
    monkeypatch.setenv("QB_ISING_THREADS", "128")
    o = P.solve(b, R, 4)
    assert (sweep_launches("ising_word_16"), sweep_launches("ising_fields")) == (before[0] + 1, before[1] + 1)
    assert (r.branches() == o.branches()).all() and (r.fields() == o.fields()).all()
    assert (r.energies_tracked() == o.energies_tracked()).all() and (r.energies() == o.energies()).all()


@pytest.mark.parametrize("n,d,R", [(32700, 3, 33), (40001, 3, 70), (33000, 5, 1), (90000, 4, 32)])
def test_whole_device_words_equal_the_field_sweep(n, d, R, monkeypatch):
    """Large graphs of few classes: words in global memory on a cooperative grid."""
    g = synth.random_regular(n, d, 3) if n != 90000 else synth.torus_pm1(300, 5)
    P = IsingProblem(*g)
    s = P.scaled_schedule(9, 1)
    kernel = "ising_grid_16" if P.n <= 32768 else "ising_grid_32"
    before = sweep_launches(kernel), sweep_launches("ising_fields")
    r = P.solve(s, R, 12)
    monkeypatch.setenv("QB_ISING_THREADS", "512")
    o = P.solve(s, R, 12)
    assert (sweep_launches(kernel), sweep_launches("ising_fields")) == (before[0] + 1, before[1] + 1)
    assert (r.branches() == o.branches()).all() and (r.fields() == o.fields()).all()
    assert (r.energies_tracked() == o.energies_tracked()).all() and (r.energies() == o.energies()).all()
    assert (r.marginals() == o.marginals()).all()


@pytest.mark.parametrize("graph,R,kernel", [("long rows", 200, "ising_fields"), ("long rows", 4096, "ising_word_16"),
                                            ("short rows", 200, "ising_word_16")])
def test_words_are_taken_where_their_class_step_pays(graph, R, kernel):
    """Long rows make the word sweep's class step long: few replicas of such a
    graph stay on the CTA-per-replica sweep."""
    g = synth.erdos_renyi(400, 0.5, 4) if graph == "long rows" else synth.random_regular(700, 20, 4)
    P = IsingProblem(*g)
    s = P.scaled_schedule(40, 2)
    before = sweep_launches(kernel)
    r = P.solve(s, R, 2)
    assert sweep_launches(kernel) == before + 1
    G = O.Graph(*g)
    order, _ = P.colouring()
    temps = O.temperatures(s.t_hot, s.t_cold, s.anneal_sweeps, s.hold_sweeps)
    for k in (0, 1, R - 1):
        key, half = O.ising_key_half(k, 2)
        x, f, e = G.anneal_coloured(order, temps, key, half=half)
        assert (r.branches()[k] == x).all() and r.energies_tracked()[k] == e and (r.fields()[k] == f).all()


@pytest.mark.parametrize("L,R,kernel", [(64, 16, "ising_replica_w8"), (64, 148, "ising_fields"), (100, 16, "ising_grid_16"),
                                        (128, 100, "ising_grid_16")])
def test_the_whole_device_is_taken_where_its_class_step_pays(L, R, kernel, monkeypatch):
    """Two classes of L x L / 2 bits: a grid barrier costs more than a CTA's visit
    of 2,048 of them and less than one of 5,000."""
    P = IsingProblem(*synth.torus_pm1(L, 5))
    s = P.scaled_schedule(20, 2)
    before = sweep_launches(kernel)
    r = P.solve(s, R, 2)
    assert sweep_launches(kernel) == before + 1
    monkeypatch.setenv("QB_ISING_THREADS", "512")
    o = P.solve(s, R, 2)
    assert (r.branches() == o.branches()).all() and (r.fields() == o.fields()).all()
    assert (r.energies_tracked() == o.energies_tracked()).all()
