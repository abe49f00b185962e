"""A circuit that is new on every call pays for no memory of checked compilations (CPU)."""
import importlib

import numpy as np
import pytest

import mossquantum_b200 as mq
from mossquantum_b200.states import StateVector

backend = importlib.import_module("mossquantum_b200.backend")
circuit = importlib.import_module("mossquantum_b200.circuit")


class Lib:
    def mb_apply(self, *args):
        return 0


@pytest.fixture
def counted(monkeypatch):
    """apply_ without a device: counts value keys and lowerings."""
    counts = {"key": 0, "lowering": 0, "compiled": 0}
    key, lowering = circuit.QCircuit.value_key, circuit._matrix_lowering

    class Compiled:
        handle = None

        def __init__(self, *args):
            counts["compiled"] += 1

        def theta_from(self, values):
            return np.asarray(values)

        def close(self):
            pass

    def count_key(self):
        counts["key"] += 1
        return key(self)

    def count_lowering(items):
        counts["lowering"] += 1
        return lowering(items)

    monkeypatch.setattr(circuit, "CompiledCircuit", Compiled)
    monkeypatch.setattr(circuit.QCircuit, "value_key", count_key)
    monkeypatch.setattr(circuit, "_matrix_lowering", count_lowering)
    monkeypatch.setattr(backend, "_matrix_lowering", count_lowering)
    monkeypatch.setattr(backend.N, "lib", lambda: Lib())
    state = StateVector.__new__(StateVector)
    state.n, state.batch, state.handle = 3, 1, None
    return counts, state


def matrices():
    return mq.QCircuit([mq.QuantumGate(1, np.eye(2)), mq.CZGate(1, 2), mq.HGate(3)])


def test_matrix_circuits(counted):
    counts, state = counted
    c = matrices()
    backend.apply_(c, state)
    assert counts == {"key": 0, "lowering": 1, "compiled": 1}      # used once: nothing else
    for _ in range(3):
        backend.apply_(c, state)
    assert counts["compiled"] == 1 and counts["lowering"] == 2       # remembered from the second call on
    c[0].data[1, 1] = -1.0
    backend.apply_(c, state)
    assert counts["compiled"] == 2 and counts["lowering"] == 3       # and in-place changes are seen
    c[0].data[1, 1] = 1.0
    backend.apply_(c, state)
    assert counts["compiled"] == 2


def test_circuits_with_angles(counted):
    """Their key replaces the general signature, so the first call takes it and the second is known."""
    counts, state = counted
    c = mq.QCircuit([mq.RxGate(1, 0.3, isparas=True), mq.CNOTGate(1, 2)])
    backend.apply_(c, state)
    assert counts["key"] == 1 and counts["compiled"] == 1
    lowerings = counts["lowering"]
    backend.apply_(c, state)
    assert counts["key"] == 2 and counts["compiled"] == 1 and counts["lowering"] == lowerings


def test_checks_still_run(counted):
    counts, state = counted
    c = matrices()
    backend.apply_(c, state)
    c[1].pos = (1, 4)
    with pytest.raises(ValueError):
        backend.apply_(c, state)
    with pytest.raises(ValueError):
        backend.apply_(c, state)
