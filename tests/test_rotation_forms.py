"""Tangent-form rotations at the edges of their range: cosines around the bound, exactly zero, and
chains whose gathered factors pass the point where a pass multiplies them in early. Tolerances as in
the lowering and gate tests (1e-12 max-abs; a chain of k rotations adds k roundings of 1e-16)."""
import numpy as np
import pytest

import mossquantum_b200 as mq
from tests.test_schedule import lowering_errors


def rotation(c, rng):
    """U3 with cosine c and random phases."""
    a, b, g = np.exp(1j * rng.uniform(0, 2 * np.pi, 3))
    s = np.sqrt(1 - c * c)
    return g * np.array([[c, -s * b], [s * a, c * a * b]])


def chain(n, cosines, rng):
    """Each cosine on a qubit of a moving pair, cut by CZ so that runs do not multiply."""
    circ = mq.QCircuit()
    for k, c in enumerate(cosines):
        q = 1 + k % n
        circ.push(mq.QuantumGate(q, rotation(c, rng)))
        circ.push(mq.CZGate(q, 1 + (k + 1) % n))
    return circ


COSINES = [[1.0, 0.5], [1 / 1024, np.nextafter(1 / 1024, 0)], [0.0, 0.3], [2.0 ** -9] * 100, [1e-12, 0.9, 2e-3]]


@pytest.mark.parametrize("cosines", COSINES)
@pytest.mark.parametrize("dm", [False, True])
def test_lowering(cosines, dm):
    n = 5 if dm else 9
    c = chain(n, cosines * 3, np.random.default_rng(5))
    for t, R in ((8, 3), (9, 4)):
        ea, eb = lowering_errors(c, n, dm=dm, t=t, R=R)
        assert ea <= 1e-12 and eb <= 1e-12, (ea, eb)


@pytest.mark.gpu
@pytest.mark.parametrize("jit", [False, True])
@pytest.mark.parametrize("cosines", COSINES)
def test_passes(mq, O, monkeypatch, cosines, jit):
    monkeypatch.setenv("MB_JIT_MIN_BITS", "8" if jit else "30")
    rng = np.random.default_rng(6)
    for n in (9, 12):
        c = chain(n, cosines * 3, rng)
        psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        psi /= np.linalg.norm(psi)
        got = mq.apply_(c, mq.StateVector(psi)).to_numpy()
        assert np.max(np.abs(got - O.apply(c.specs(), psi, n))) <= 1e-12
