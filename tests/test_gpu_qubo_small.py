"""The weighted-QUBO sweep of one CTA (fields in shared memory) against the
cooperative sweep and the oracle, bit for bit: fewer bits than warps, one class,
classes of one bit, rows of more than 32 neighbours, uneven replica counts over
several CTAs, the refresh, the trace."""
import numpy as np
import pytest

from oracle import oracle as O
from qublar_b200 import QuboProblem, Schedule, sweep_launches, synth

pytestmark = pytest.mark.gpu


def _complete(n, seed):
    rng = np.random.default_rng(seed)
    u, v = np.triu_indices(n, 1)
    return {"n": n, "eu": u.astype(np.int32), "ev": v.astype(np.int32),
            "ew": rng.standard_normal(u.size).astype(np.float32), "h": rng.standard_normal(n).astype(np.float32),
            "offset": 0.5}


CASES = {
    "one_bit": (lambda: {"n": 1, "eu": [], "ev": [], "ew": [], "h": [0.3], "offset": 0.0}, 5),
    "no_edges": (lambda: {"n": 40, "eu": [], "ev": [], "ew": [], "h": np.linspace(-1, 1, 40), "offset": 0.0}, 64),
    "five_bits": (lambda: _complete(5, 1), 3),
    "k15": (lambda: _complete(15, 2), 33),
    "k16": (lambda: _complete(16, 3), 65),
    "k70": (lambda: _complete(70, 4), 64),
    "star": (lambda: {"n": 50, "eu": [0] * 49, "ev": list(range(1, 50)), "ew": np.linspace(-2, 2, 49), "h": None,
                      "offset": 0.0}, 40),
    "sparse": (lambda: synth.random_qubo(120, 700, 5), 130),
    "widest": (lambda: synth.random_qubo(840, 1900, 6), 64),
}


@pytest.mark.parametrize("name", list(CASES))
def test_equals_the_cooperative_sweep_and_the_oracle(name, monkeypatch):
    make, R = CASES[name]
    q = make()
    q = {**q, "eu": np.asarray(q["eu"], np.int32), "ev": np.asarray(q["ev"], np.int32),
         "ew": np.asarray(q["ew"], np.float32), "h": None if q["h"] is None else np.asarray(q["h"], np.float32)}
    P = QuboProblem.from_dict(q)
    s = Schedule(2.5, 0.1, 60, 7, 9)
    before = sweep_launches("qubo_small"), sweep_launches("qubo_lockstep")
    monkeypatch.setenv("QB_QUBO_KERNEL", "small")
    r = P.solve(s, R, 2)
    t = P.solve(s, R, 2, trace=True)
    monkeypatch.setenv("QB_QUBO_KERNEL", "lockstep")
    o = P.solve(s, R, 2, trace=True)
    assert (sweep_launches("qubo_small"), sweep_launches("qubo_lockstep")) == (before[0] + 2, before[1] + (R + 63) // 64)
    X = r.branches()
    assert (X == o.branches()).all() and (X == t.branches()).all()
    assert np.array_equal(r.energies(), o.energies())
    a, b = r.info(), o.info()
    assert a.accepted == b.accepted and a.max_drift == b.max_drift
    E = o.energy_trace()
    assert np.abs(t.energy_trace() - E).max() <= 1e-12 * 70 * max(1.0, np.abs(E).max())   # fp64 sums in another order
    order, cptr = P.colouring()
    temps = O.temperatures(s.t_hot, s.t_cold, s.anneal_sweeps, s.hold_sweeps)
    if q["h"] is None:
        q["h"] = np.zeros(q["n"], np.float32)
    for k in sorted({0, min(R, 64) - 1, R - 1}):
        key, half = O.qubo_key_half(k, 2)
        x, _, _ = O.qubo_anneal_coloured(q, order, cptr, temps, s.refresh_sweeps, key, half)
        assert (X[k] == x).all(), k
