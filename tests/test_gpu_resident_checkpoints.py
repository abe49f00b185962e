"""Checkpointed gradients of small circuits whose matrices are not unitary: a checkpoint at every
instruction makes the sweep exact for any matrix (the state is read back, not undone). Against central
differences with h = 1e-6: truncation 1e-12 and rounding 1e-9 of values of order one, so 1e-7."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def circuit(mq, n, rng, two):
    c = mq.QCircuit()
    for q in range(1, n + 1):
        c.push(mq.RyGate(q, float(rng.uniform(0, 6)), isparas=True))
    c.push(mq.QuantumGate(1, [[1.0, 0.3], [0.0, 0.8]]))
    c.push(mq.CNOTGate(1, 2))
    c.push(mq.RxGate(1, float(rng.uniform(0, 6)), isparas=True))
    if two == "dense":
        c.push(mq.QuantumGate((1, 2), np.eye(4) + 0.2 * rng.normal(size=(4, 4))))
    elif two == "diagonal":
        c.push(mq.QuantumGate((1, 2), np.diag([1.0, 0.9, 1.1j, 0.7])))
    c.push(mq.RzGate(2, float(rng.uniform(0, 6)), isparas=True))
    c.push(mq.QuantumGate(2, [[0.9, 0.1j], [0.2, 1.1]]))
    c.push(mq.RyGate(n, float(rng.uniform(0, 6)), isparas=True))
    return c


@pytest.mark.parametrize("n,two", [(2, "none"), (3, "dense"), (6, "diagonal"), (10, "dense"), (12, "none"), (13, "dense")])
def test_matrices_that_are_not_unitary(mq, n, two):
    rng = np.random.default_rng(n)
    c = circuit(mq, n, rng, two)
    H = mq.QubitsOperator([mq.QubitsTerm([1], ["Z"], 0.7), mq.QubitsTerm([1, 2], ["X", "Y"], 0.4), mq.QubitsTerm([n], ["X"], -0.5)])
    obj = mq.ExpectationObjective(c, H, mq.StateVector(n))
    theta = np.array(c.active_parameters())
    val, g = mq.value_and_gradient(mq.AdjointGradient(checkpoint_every=1), obj, theta)
    assert abs(val - obj.evaluate(theta)) <= 1e-11
    for i in range(len(theta)):
        d = np.zeros(len(theta))
        d[i] = 1e-6
        assert abs(g[i] - (obj.evaluate(theta + d) - obj.evaluate(theta - d)) / 2e-6) <= 1e-7
