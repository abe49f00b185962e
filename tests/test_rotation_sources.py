"""The generated passes of a circuit of fixed gates do not depend on the values of its matrices, so a circuit
rebuilt with new angles finds its kernels compiled: angles at and around pi, and passes of several hundred rotations,
whose gathered factors are multiplied in at fixed places (CPU)."""
import numpy as np
import pytest

import mossquantum_b200 as mq
from mossquantum_b200.gates import U3
from tests.test_schedule import lowering_errors, schedule_info


def sources(circ, n, monkeypatch, path):
    path.mkdir()
    monkeypatch.setenv("MB_JIT_DUMP", str(path))
    schedule_info(circ, n, t=10, R=3)
    monkeypatch.delenv("MB_JIT_DUMP")
    return [p.read_text() for p in sorted(path.glob("pass_*.cu"))]


def brickwork(n, layers, theta, rng):
    c = mq.QCircuit()
    for layer in range(layers):
        for q in range(1, n + 1):
            c.push(mq.QuantumGate(q, U3(theta(rng), *rng.uniform(0.1, 6.2, 2))))
        for q in range(1 + layer % 2, n, 2):
            c.push(mq.CZGate(q, q + 1))
    return c


def uniform(rng):
    return rng.uniform(0, 2 * np.pi)


def near_pi(rng):
    return np.pi + 10.0 ** rng.uniform(-15, -1) * rng.choice([-1, 1])


def some_near_pi(rng):
    return near_pi(rng) if rng.random() < 0.05 else uniform(rng)


FORMS = [uniform, some_near_pi, near_pi, lambda rng: np.pi, lambda rng: rng.choice([0.3, np.pi, np.pi - 1e-3, 3.0])]


@pytest.mark.parametrize("n,layers", [(14, 4), (11, 60), (10, 200)])
def test_same_sources(monkeypatch, tmp_path, n, layers):
    got = [sources(brickwork(n, layers, f, np.random.default_rng(k)), n, monkeypatch, tmp_path / str(k))
           for k, f in enumerate([uniform, uniform, some_near_pi, some_near_pi])]
    assert got[0] and any(len(s) > 1000 for s in got[0])
    for other in got[1:]:
        assert other == got[0]


@pytest.mark.parametrize("form", range(5))
def test_values(form):
    n = 9
    c = brickwork(n, 40, FORMS[form], np.random.default_rng(form))
    for t, R in ((8, 3), (9, 4)):
        ea, eb = lowering_errors(c, n, t=t, R=R)
        assert ea <= 1e-12 and eb <= 1e-12, (ea, eb)
