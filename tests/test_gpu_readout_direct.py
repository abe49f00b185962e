"""Readout of the whole register in its own order is a copy of squares in one kernel. Each bin is one
product, so two roundings and the division by the total: 4e-16 relative and 2^n roundings of the total."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,B,dm", [(1, 1, False), (4, 3, False), (9, 2, False), (13, 1, False), (3, 2, True), (6, 1, True)])
def test_whole_register(mq, n, B, dm):
    from mossquantum_b200 import _native as N
    rng = np.random.default_rng(n)
    v = rng.normal(size=(1 << n, B)) + 1j * rng.normal(size=(1 << n, B))
    v /= np.linalg.norm(v, axis=0)
    s = mq.StateVector(v[:, 0]) if B == 1 else mq.BatchStateVector(v)
    if dm:
        s = mq.DensityMatrix(s) if B == 1 else mq.BatchDensityMatrix(s)
    N.profile(True)
    got = np.asarray(mq.probabilities(s)).reshape(-1, B, order="F")
    seen = N.profile_report()
    N.profile(False)
    assert "k_probabilities" in seen and "k_marginal" not in seen
    assert np.max(np.abs(got - np.abs(v) ** 2)) <= 4e-12
    if n > 1:      # any other order goes through the marginal kernel
        N.profile(True)
        swapped = np.asarray(mq.probabilities(s, [2, 1] + list(range(3, n + 1)))).reshape(-1, B, order="F")
        assert "k_marginal" in N.profile_report()
        N.profile(False)
        i = np.arange(1 << n)
        j = (i & ~3) | ((i & 1) << 1) | ((i >> 1) & 1)
        assert np.max(np.abs(swapped[j] - got)) <= 4e-12


def test_negative_and_complex_diagonals_are_refused(mq):
    bad = np.diag([1.2, -0.2]).astype(complex)
    with pytest.raises(Exception):
        mq.probabilities(mq.DensityMatrix(bad))
    with pytest.raises(Exception):
        mq.probabilities(mq.DensityMatrix(np.diag([0.5 + 0.1j, 0.5])))
