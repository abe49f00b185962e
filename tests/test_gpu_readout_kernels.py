"""Marginals and pure-state partial traces at the edges of their kernels' tiles and splits,
against numpy sums over the same amplitudes. Tolerance: a bin or entry adds at most 2^14 products
of total weight <= 1, so its rounding error stays below 2^14 * 2.3e-16 = 4e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 4e-12


def rand(n, B, seed):
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(1 << n, B)) + 1j * rng.normal(size=(1 << n, B))
    return v / np.linalg.norm(v, axis=0)


def axes_last(v, n, qubits):
    """(2^rest, 2^len(qubits)) view of a state with qubits[0] as the lowest column bit."""
    rest = [q for q in range(1, n + 1) if q not in qubits]
    order = [n - q for q in reversed(rest)] + [n - q for q in reversed(qubits)]
    return v.reshape([2] * n).transpose(order).reshape(-1, 1 << len(qubits))


@pytest.mark.parametrize("n,qubits", [
    (1, [1]), (3, [2]), (4, [4, 1]), (5, []), (5, [5, 1, 3]), (6, [6]), (9, [9, 5, 6, 1]), (12, [1]), (12, [12]),
    (13, [3]), (14, [14, 2, 7]), (11, list(range(1, 12))), (11, list(range(11, 0, -1))), (17, [17, 1, 9])])
def test_marginals(mq, n, qubits):
    for B in (1, 3):
        v = rand(n, B, 7 * n + B)
        s = mq.StateVector(v[:, 0]) if B == 1 else mq.BatchStateVector(v)
        got = np.asarray(mq.probabilities(s, qubits)).reshape(-1, B, order="F")
        for b in range(B):
            ref = (np.abs(axes_last(v[:, b], n, qubits)) ** 2).sum(axis=0)
            assert np.max(np.abs(got[:, b] - ref)) <= TOL
        if n <= 6:
            rho = np.stack([np.outer(v[:, b], v[:, b].conj()) for b in range(B)], axis=2)
            d = mq.DensityMatrix(rho[:, :, 0]) if B == 1 else mq.BatchDensityMatrix(rho)
            assert np.max(np.abs(np.asarray(mq.probabilities(d, qubits)).reshape(-1, B, order="F") - got)) <= TOL


@pytest.mark.parametrize("n,keep", [
    (2, [1]), (2, [2]), (5, [3]), (5, [1, 5]), (8, [1, 2, 3]), (8, [2, 4, 6, 8]), (9, [1, 2, 3, 4, 5, 6, 7, 8]),
    (10, [3, 4, 5, 6, 7, 8, 10]), (10, [1, 3, 5, 7, 9, 10]), (13, [13]), (13, [6, 7]), (14, [1, 4, 7, 10, 13, 14]),
    (14, [2, 3, 5, 8, 9, 11, 13]), (16, [1, 16])])
def test_partial_trace_pure(mq, n, keep):
    traced = [q for q in range(1, n + 1) if q not in keep]
    for B in (1, 2):
        v = rand(n, B, 11 * n + B)
        if B == 1:
            got = [mq.partial_tr(mq.StateVector(v[:, 0]), traced)]
        else:
            got = mq.partial_tr(mq.BatchStateVector(v), traced)
        for b in range(B):
            m = axes_last(v[:, b], n, keep)
            assert np.max(np.abs(got[b].to_numpy() - m.T @ m.conj())) <= TOL


@pytest.mark.parametrize("n,keep", [(2, [1]), (6, [1, 6]), (7, [2]), (9, [9]), (9, [3, 4, 5])])
def test_partial_trace_density(mq, n, keep):
    v = rand(n, 2, 13 * n)
    rho = 0.75 * np.outer(v[:, 0], v[:, 0].conj()) + 0.25 * np.outer(v[:, 1], v[:, 1].conj())
    traced = [q for q in range(1, n + 1) if q not in keep]
    got = mq.partial_tr(mq.DensityMatrix(rho), traced).to_numpy()
    ref = sum(w * (m.T @ m.conj()) for w, m in ((0.75, axes_last(v[:, 0], n, keep)), (0.25, axes_last(v[:, 1], n, keep))))
    assert np.max(np.abs(got - ref)) <= TOL
