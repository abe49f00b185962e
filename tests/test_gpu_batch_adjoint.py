"""Gradients of weighted batch losses against the oracle's per-sample gradients, and density-matrix
expectations from Pauli strings against the dense keys. Tolerances as everywhere: 1e-11 on values,
1e-10 on gradients."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def unit(n, B, seed):
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(1 << n, B)) + 1j * rng.normal(size=(1 << n, B))
    return v / np.linalg.norm(v, axis=0)


def weighted(O, c, states, n, H, w, dm):
    vr, gr = 0.0, 0.0
    for b, wb in enumerate(w):
        x = np.outer(states[:, b], states[:, b].conj()).ravel(order="F") if dm else states[:, b]
        vb, gb = O.adjoint(c.specs(), x, n, H.specs(), dm=True) if dm else O.adjoint(c.specs(), x, n, H.specs())
        vr, gr = vr + wb * vb, gr + wb * gb
    return vr, gr


@pytest.mark.parametrize("n,B,pure", [(1, 2, True), (2, 9, False), (4, 5, True), (4, 17, False), (5, 3, True)])
@pytest.mark.parametrize("weights", [False, True])
def test_noisy_batches_combine(mq, O, n, B, pure, weights):
    from mossquantum_b200 import workloads as W
    c = W.hea_circuit(n, 2, W.hea_angles(n, 2, W.rng_for(8)), noise=(0.01, 0.02))
    H = W.xxz(n) if n > 1 else mq.QubitsOperator([mq.QubitsTerm([1], ["X"], 0.7)])
    v = unit(n, B, n * B)
    init = mq.BatchStateVector(v)
    if not pure:
        init = mq.BatchDensityMatrix(init)
    how = dict(reduction="weighted_sum", weights=np.linspace(-0.5, 1.5, B)) if weights else {}
    obj = mq.BatchExpectationObjective(c, H, init, **how)
    val, g = mq.value_and_gradient(mq.AdjointGradient(), obj, c.active_parameters())
    vr, gr = weighted(O, c, v, n, H, obj.sample_weights(), True)
    assert abs(val - vr) <= 1e-11 and np.max(np.abs(g - gr)) <= 1e-10


@pytest.mark.parametrize("n,B", [(1, 1), (2, 3), (5, 1), (7, 4), (9, 2)])
def test_density_strings_match_keys(mq, monkeypatch, n, B):
    rng = np.random.default_rng(n + 10 * B)
    v = unit(n, 2 * B, n)
    rho = np.stack([0.75 * np.outer(v[:, 2 * b], v[:, 2 * b].conj())
                    + 0.25 * np.outer(v[:, 2 * b + 1], v[:, 2 * b + 1].conj()) for b in range(B)], axis=2)
    s = mq.BatchDensityMatrix(rho)
    names = ["X", "Y", "Z", "+", "-", "I", "u", "d"]
    terms = [mq.QubitsTerm([], [], 0.3 - 0.1j)]
    for k in range(1, min(n, 5) + 1):
        pos = [int(x) for x in rng.choice(np.arange(1, n + 1), size=k, replace=False)]
        terms.append(mq.QubitsTerm(pos, [names[rng.integers(8)] for _ in range(k)], complex(rng.normal(), rng.normal())))
    dense = [rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)) for _ in range(min(n, 5))]
    many = [mq.QubitsTerm(list(range(1, len(dense) + 1)), dense, 1.0)]      # 4^k strings on one key
    for H in (mq.QubitsOperator(terms), mq.QubitsOperator(many)):
        got = mq.expectation(H, s)
        monkeypatch.setenv("MB_EXPECT_KEYS", "1")
        keys = mq.expectation(H, s)
        monkeypatch.delenv("MB_EXPECT_KEYS")
        scale = max(1.0, np.max(np.abs(keys)))
        assert np.max(np.abs(got - keys)) <= 1e-11 * scale
        for b in range(B):
            assert abs(got[b] - np.trace(H.matrix(n) @ rho[:, :, b])) <= 1e-11 * scale


@pytest.mark.parametrize("n,B,ck", [(13, 3, 0), (13, 2, 31), (14, 1, 0)])
def test_pure_reverse_with_runs(mq, O, n, B, ck):
    """Runs of gates undone as one 2x2 with cross sums, beside controlled and two-qubit gates that stay
    apart, fixed gates inside runs, adjoint gates, and one parameter per gate."""
    rng = np.random.default_rng(n + B)
    a = lambda: float(rng.uniform(0, 2 * np.pi))
    c = mq.QCircuit()
    for layer in range(2):
        for q in range(1, n + 1):
            c.push(mq.RxGate(q, a(), isparas=True))
            c.push([mq.HGate(q), mq.RyGate(q, a(), isparas=True).adjoint(), mq.TGate(q), mq.PHASEGate(q, a(), isparas=True)][q % 4])
            c.push(mq.RzGate(q, a(), isparas=q % 3 != 0))
            if q % 5 == 0:
                c.push(mq.RxGate(q, a(), isparas=True))
        for q in range(1, n):
            c.push(mq.CNOTGate(q, q + 1) if q % 3 else mq.CRyGate(q + 1, q, a(), isparas=True))
        c.push(mq.iSWAPGate(2, 9))
    H, v = mq.QubitsOperator([mq.QubitsTerm([1, n], ["X", "Y"], 0.5), mq.QubitsTerm([4], ["Z"], -1.0)]), unit(n, B, n)
    w = np.linspace(0.5, -0.75, B) if B > 1 else [1.0]
    if B > 1:
        obj = mq.BatchExpectationObjective(c, H, mq.BatchStateVector(v), reduction="weighted_sum", weights=w)
    else:
        obj = mq.ExpectationObjective(c, H, mq.StateVector(v[:, 0]))
    val, g = mq.value_and_gradient(mq.AdjointGradient(checkpoint_every=ck), obj, c.active_parameters())
    vr, gr = weighted(O, c, v, n, H, w, False)
    assert abs(val - vr) <= 1e-11 and np.max(np.abs(g - gr)) <= 1e-10
