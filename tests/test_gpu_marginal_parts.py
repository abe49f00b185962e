"""Marginals whose sums are split: parts of fewer and of more terms than a lane loads at once, added by a
block or a warp per bin, at the sizes where the form changes, and twice in a row with the same bits. A bin adds at
most 2^20 squares of total weight <= 1: 2^20 * 2.3e-16 / 2^6 (parts of sums) stays below 4e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,B,qubits", [
    (9, 1, [1]), (11, 1, [3]), (11, 3, [2, 10]), (12, 64, [3, 7]), (12, 64, list(range(2, 9))), (16, 1, [1]), (16, 1, [16, 2, 5]),
    (19, 1, [19]), (20, 1, [1]), (20, 1, [4, 20]), (20, 1, [1, 2, 3]), (20, 1, [1, 2, 3, 4]), (20, 1, [6, 1, 2, 3, 4]),
    (20, 1, [1, 2, 3, 4, 5, 20]), (20, 2, [2, 9, 17])])
def test_split_sums(mq, n, B, qubits):
    rng = np.random.default_rng(n + B)
    v = rng.normal(size=(1 << n, B)) + 1j * rng.normal(size=(1 << n, B))
    v /= np.linalg.norm(v, axis=0)
    s = mq.StateVector(v[:, 0]) if B == 1 else mq.BatchStateVector(v)
    got = np.asarray(mq.probabilities(s, qubits)).reshape(-1, B, order="F")
    rest = [q for q in range(1, n + 1) if q not in qubits]
    order = [n - q for q in reversed(rest)] + [n - q for q in reversed(qubits)]
    for b in range(B):
        ref = (np.abs(v[:, b].reshape([2] * n).transpose(order).reshape(-1, 1 << len(qubits))) ** 2).sum(axis=0)
        assert np.max(np.abs(got[:, b] - ref)) <= 4e-12
    again = np.asarray(mq.probabilities(s, qubits)).reshape(-1, B, order="F")
    assert np.array_equal(got, again)


@pytest.mark.parametrize("n,qubits", [(10, [1]), (12, [1, 2, 3]), (12, [12, 1])])
def test_density_diagonals(mq, n, qubits):
    rng = np.random.default_rng(n)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v /= np.linalg.norm(v)
    s = mq.StateVector(v)
    got = np.asarray(mq.probabilities(mq.DensityMatrix(s), qubits))
    assert np.max(np.abs(got - np.asarray(mq.probabilities(s, qubits)))) <= 4e-12
