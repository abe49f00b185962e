"""Objectives of small pure states (one launch: linear frame, gate runs, reverse) against the oracle,
over every gate form the launch takes and the sizes where its thread layout changes. 1e-11 on
values, 1e-10 on gradients."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def unit(n, B, seed):
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(1 << n, B)) + 1j * rng.normal(size=(1 << n, B))
    return v / np.linalg.norm(v, axis=0)


def unitary(d, rng):
    q, r = np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def mixed_circuit(mq, n, count, rng, fallback=False):
    """Gates of every kind on random qubits, half of the angles active."""
    c = mq.QCircuit()
    one = [mq.XGate, mq.YGate, mq.ZGate, mq.HGate, mq.SGate, mq.TGate, mq.sqrtXGate]
    two = [mq.CNOTGate, mq.CZGate, mq.SWAPGate, mq.iSWAPGate]
    for _ in range(count):
        q = [int(x) for x in rng.permutation(np.arange(1, n + 1))]
        a, act = float(rng.uniform(0, 2 * np.pi)), bool(rng.random() < 0.6)
        k = int(rng.integers(9 if n < 2 else 13 if n < 3 else 16))
        if k < 4:
            c.push([mq.RxGate, mq.RyGate, mq.RzGate, mq.PHASEGate][k](q[0], a, isparas=act))
        elif k < 6:
            c.push(one[rng.integers(len(one))](q[0]))
        elif k == 6:
            c.push(mq.QuantumGate(q[0], unitary(2, rng)))
        elif k < 9:
            c.push([mq.RxGate, mq.RyGate, mq.RzGate][k % 3](q[0], a, isparas=act).adjoint())
        elif k == 9:
            c.push([mq.CRxGate, mq.CRyGate, mq.CRzGate, mq.CPHASEGate][rng.integers(4)](q[0], q[1], a, isparas=act))
        elif k == 10:
            c.push(mq.QuantumGate((q[0], q[1]), unitary(4, rng)))
        elif k < 13:
            c.push(two[rng.integers(len(two))](q[0], q[1]))
        elif k == 13:
            c.push(mq.TOFFOLIGate(q[0], q[1], q[2]))
        elif k == 14:
            c.push(mq.CCPHASEGate(q[0], q[1], q[2], a, isparas=act))
        else:
            c.push(mq.QuantumGate((q[0], q[1], q[2]), np.diag(np.exp(1j * rng.uniform(0, 6, 8)))))
    if fallback:
        c.push(mq.FREDKINGate(1, 2, 3))
    c.push(mq.RyGate(1, 0.3, isparas=True))
    return c


def observable(mq, n, rng):
    terms = [mq.QubitsTerm([], [], 0.25)]
    for k in range(1, min(n, 4) + 1):
        for _ in range(3):
            pos = [int(x) for x in rng.choice(np.arange(1, n + 1), size=k, replace=False)]
            terms.append(mq.QubitsTerm(pos, [["X", "Y", "Z"][rng.integers(3)] for _ in range(k)], float(rng.normal())))
    return mq.QubitsOperator(terms)


@pytest.mark.parametrize("n,B,count,fallback", [
    (1, 1, 12, False), (2, 3, 20, False), (3, 1, 30, True), (5, 2, 40, False), (6, 17, 40, False), (7, 1, 50, False),
    (8, 3, 60, False), (10, 1, 60, False), (11, 2, 60, False), (12, 1, 60, False), (12, 3, 40, True),
    (13, 1, 40, False)])
def test_mixed_gates(mq, O, n, B, count, fallback):
    rng = np.random.default_rng(100 * n + B)
    c, H, v = mixed_circuit(mq, n, count, rng, fallback), observable(mq, n, rng), unit(n, B, n)
    theta = np.array(c.active_parameters())
    if B == 1:
        obj, w = mq.ExpectationObjective(c, H, mq.StateVector(v[:, 0])), [1.0]
    else:
        w = np.linspace(-0.5, 1.5, B)
        obj = mq.BatchExpectationObjective(c, H, mq.BatchStateVector(v), reduction="weighted_sum", weights=w)
    val, g = mq.value_and_gradient(mq.AdjointGradient(), obj, theta)
    vr, gr = 0.0, 0.0
    for b in range(B):
        vb, gb = O.adjoint(c.specs(), v[:, b], n, H.specs())
        vr, gr = vr + w[b] * vb, gr + w[b] * gb
    assert abs(val - vr) <= 1e-11 and np.max(np.abs(g - gr)) <= 1e-10
    assert abs(obj.evaluate(theta) - vr) <= 1e-11


def test_shared_values_and_many_rows(mq, O):
    """More gradients than a chunk of rows holds, shared parameters, repeated calls, one changed angle."""
    from mossquantum_b200 import workloads as W
    n = 9
    c = W.hea_circuit(n, 3, W.hea_angles(n, 3, W.rng_for(2)))
    H, theta = W.xxz(n), np.array(c.active_parameters())
    obj = mq.ExpectationObjective(c, H, mq.StateVector(n), parameter_map=mq.ParameterMap([1 + k % 40 for k in range(81)]))
    free = theta[:40]
    for step in range(2):
        c.reset_parameters([free[k % 40] for k in range(81)])
        vr, gr = O.adjoint(c.specs(), O.zero_state(n), n, H.specs())
        val, g = mq.value_and_gradient(mq.AdjointGradient(), obj, free)
        assert abs(val - vr) <= 1e-11 and abs(obj.evaluate(free) - vr) <= 1e-11
        assert np.max(np.abs(g - [gr[k::40].sum() for k in range(40)])) <= 1e-10
        free = free + 0.1
