"""Staged sources are kept by what they are generated from: observables that differ in one thing each (real or
complex coefficients, a letter, a position, the order, the size) do not take each other's. 1e-11 as for every
expectation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_neighbouring_observables(mq, O):
    def H(n, letters, positions, coeffs):
        return mq.QubitsOperator([mq.QubitsTerm(p, l, c) for p, l, c in zip(positions, letters, coeffs)])

    pos, real = [[1, 2], [3, 7], [2, 9, 13], [14]], [0.5, -0.7, 0.3, 1.1]
    base = [["X", "X"], ["Y", "X"], ["Z", "X", "Y"], ["Z"]]
    forms = [(14, base, pos, real), (14, base, pos, [0.5, -0.7j, 0.3, 1.1]), (14, base, pos, [0.5j, -0.7j, 0.3 + 1j, 1.1]),
             (14, [["X", "Y"]] + base[1:], pos, real), (14, base, [[1, 3]] + pos[1:], real), (14, base[::-1], pos[::-1], real),
             (15, base, pos, real), (14, base, pos, [0.1, 0.2, 0.3, 0.4])]
    for n, letters, positions, coeffs in forms + forms:
        rng = np.random.default_rng(n)
        v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        v /= np.linalg.norm(v)
        op = H(n, letters, positions, coeffs)
        assert abs(mq.expectation(op, mq.StateVector(v)) - O.expect(v, n, op.specs())) <= 1e-11
