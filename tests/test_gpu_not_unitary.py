"""Gradients of circuits with matrices that are not unitary: small pure states, pure batches and weighted
density matrices keep the order of the gates in the reverse sweep and agree with the gate-by-gate sweep (the fused
passes of single pure states from 9 qubits and of density matrices with equal weights move gates on different
qubits past one another, as they always did). 1e-11 and 1e-10, as between the
forms of any gradient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def circuit(mq, n, rng):
    c = mq.QCircuit()
    for layer in range(3):
        for q in range(1, n + 1):
            c.push([mq.RxGate, mq.RyGate, mq.RzGate][(q + layer) % 3](q, float(rng.uniform(0, 6)), isparas=True))
            if (q + layer) % 2:
                c.push(mq.QuantumGate(q, 0.8 * np.eye(2) + 0.3 * rng.normal(size=(2, 2))))
        for q in range(1, n):
            c.push(mq.CNOTGate(q, q + 1))
    return c


@pytest.mark.parametrize("n,B,dm,weighted", [(2, 7, False, False), (6, 1, False, False), (8, 3, False, True), (10, 2, False, True),
                                             (13, 2, False, False), (5, 4, True, True)])
@pytest.mark.parametrize("every", [0, 5])
def test_agrees_with_the_plain_sweep(mq, monkeypatch, n, B, dm, weighted, every):
    rng = np.random.default_rng(n + B)
    c = circuit(mq, n, rng)
    H = mq.QubitsOperator([mq.QubitsTerm([1], ["Z"], 0.7), mq.QubitsTerm([1, 2], ["X", "Y"], 0.4), mq.QubitsTerm([n], ["X"], -0.5)])
    v = rng.normal(size=(1 << n, B)) + 1j * rng.normal(size=(1 << n, B))
    v /= np.linalg.norm(v, axis=0)
    s = mq.StateVector(v[:, 0]) if B == 1 else mq.BatchStateVector(v)
    if dm:
        s = mq.DensityMatrix(s) if B == 1 else mq.BatchDensityMatrix(s)
    how = dict(reduction="weighted_sum", weights=np.linspace(-1.0, 1.5, B)) if weighted else {}
    obj = mq.ExpectationObjective(c, H, s) if B == 1 else mq.BatchExpectationObjective(c, H, s, **how)
    theta = np.array(c.active_parameters())
    method = mq.AdjointGradient(checkpoint_every=every)
    val, g = mq.value_and_gradient(method, obj, theta)
    monkeypatch.setenv("MB_ADJOINT_PLAIN", "1")
    vr, gr = mq.value_and_gradient(method, obj, theta)
    scale = max(1.0, abs(vr), np.max(np.abs(gr)))
    assert abs(val - vr) <= 1e-11 * scale and np.max(np.abs(g - gr)) <= 1e-10 * scale
