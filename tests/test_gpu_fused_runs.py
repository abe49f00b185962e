"""Products of fused runs formed after binding: run lengths around the unroll of four, with 2x2 (pure)
and 4x4 (density matrix, channels inside the run) products, one row or one per sample. 1e-12 max-abs on states,
1e-11 on expectations, the bounds of the gate and batch tests: a run of k gates adds k roundings of 1e-16."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def circuit(mq, n, lengths, theta, dm, rng):
    c = mq.QCircuit()
    for k, length in enumerate(lengths):
        q = 1 + k % n
        for i in range(length):
            kind = i % 5
            if kind == 0:
                c.push(mq.RxGate(q, theta[k], isparas=True))
            elif kind == 1:
                u = np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))[0]
                c.push(mq.QuantumGate(q, u))
            elif kind == 2:
                c.push(mq.RzGate(q, 0.3 * theta[k], isparas=True))
            elif kind == 3:
                c.push(mq.AmplitudeDamping(q, gamma=0.05) if dm else mq.SGate(q))
            else:
                c.push(mq.ZGate(q))
        c.push(mq.CNOTGate(q, 1 + (k + 1) % n))
    return c


@pytest.mark.parametrize("lengths", [[2], [3, 5, 4], [2, 9, 1, 17, 8, 3, 4, 5, 16]])
@pytest.mark.parametrize("dm", [False, True])
def test_one_row(mq, O, lengths, dm):
    n = 5 if dm else 9
    rng = np.random.default_rng(sum(lengths))
    c = circuit(mq, n, lengths, rng.uniform(-3, 3, size=len(lengths)), dm, rng)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    s = mq.StateVector(v / np.linalg.norm(v))
    x = s.to_numpy()
    got = mq.apply_(c, mq.DensityMatrix(s) if dm else s).to_numpy()
    x = np.outer(x, x.conj()).ravel(order="F") if dm else x
    assert np.max(np.abs(got.ravel(order="F") - O.apply(c.specs(), x, n, dm))) <= 1e-12


@pytest.mark.parametrize("lengths", [[2], [3, 5, 4], [2, 9, 1, 17, 8, 3, 4, 5, 16]])
@pytest.mark.parametrize("dm,persistent", [(True, False), (False, False), (False, True)])
@pytest.mark.parametrize("B", [1, 3])
def test_rows(mq, O, lengths, dm, persistent, B):
    from mossquantum_b200 import workloads as W
    from mossquantum_b200.batch import BatchPlan
    n = 5 if dm else 9
    rng = np.random.default_rng(sum(lengths) + 10 * B)
    c = circuit(mq, n, lengths, np.zeros(len(lengths)), dm, rng)
    how = dict(kind="density") if dm else dict(persistent=persistent)
    plan = BatchPlan({n: (c, B)}, W.xxz, **how)
    th = rng.uniform(-3, 3, size=(B, c.nparameters()))
    res = plan.run({n: th})
    for b in range(B):
        x = O.apply(c.copy().reset_parameters(th[b]).specs(), O.zero_state(n, dm), n, dm)
        assert abs(res[n][b] - O.expect(x, n, W.xxz(n).specs(), dm=dm)) <= 1e-11
    plan.close()
