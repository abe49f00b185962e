"""Staged Pauli expectation passes against the oracle: flip masks inside the register bits, across
stages and tiles, wider than the registers (partners from the tile), odd numbers of Y, complex
coefficients, batches. Tolerance 1e-11 as for every expectation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def states(n, B, seed):
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(1 << n, B)) + 1j * rng.normal(size=(1 << n, B))
    return v / np.linalg.norm(v, axis=0)


def spread(mq, n, rng, real):
    names, terms = ["X", "Y", "Z"], [mq.QubitsTerm([], [], 0.4)]
    for k in (1, 1, 2, 2, 2, 3, 4):
        pos = [int(x) for x in rng.choice(np.arange(1, n + 1), size=k, replace=False)]
        c = float(rng.normal()) if real else complex(rng.normal(), rng.normal())
        terms.append(mq.QubitsTerm(pos, [names[rng.integers(3)] for _ in range(k)], c))
    return mq.QubitsOperator(terms)


def wide(mq, n, rng):
    """A five-qubit flip, and one beside Z on other qubits."""
    pos = [int(x) for x in rng.choice(np.arange(1, n + 1), size=5, replace=False)]
    return mq.QubitsOperator([mq.QubitsTerm(pos, ["X", "Y", "X", "Y", "Y"], 0.7), mq.QubitsTerm(pos, ["Y"] * 5, 0.2 - 0.1j),
                              mq.QubitsTerm(pos[:2], ["Z", "Z"], -1.0)])


@pytest.mark.parametrize("n,B", [(10, 1), (14, 3), (18, 1), (19, 2), (20, 1)])
def test_staged_passes(mq, O, monkeypatch, n, B):
    from mossquantum_b200 import _native as N
    from mossquantum_b200 import workloads as W
    monkeypatch.setenv("MB_PAULI_JIT_MIN_BITS", "10")
    rng = np.random.default_rng(n)
    v = states(n, B, n)
    s = mq.StateVector(v[:, 0]) if B == 1 else mq.BatchStateVector(v)
    for H in (W.xxz(n), W.tfim(n), spread(mq, n, rng, True), spread(mq, n, rng, False), wide(mq, n, rng),
              mq.QubitsOperator([mq.QubitsTerm([1, n], ["Z", "Z"], 1.5)])):
        N.profile(True)
        got = np.atleast_1d(mq.expectation(H, s))
        mq.synchronize()
        assert "mbk_pauli" in N.profile_report()
        N.profile(False)
        for b in range(B):
            assert abs(got[b] - O.expect(v[:, b], n, H.specs())) <= 1e-11
