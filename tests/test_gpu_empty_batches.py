"""Empty batches: every call is a no-op that launches nothing, and what is refused otherwise is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dm", [(3, False), (9, False), (12, False), (14, False), (2, True), (5, True)])
def test_nothing_is_launched(mq, n, dm):
    from mossquantum_b200 import workloads as W
    c, H = W.hea_circuit(n, 2), W.tfim(n)
    theta = np.random.default_rng(n).uniform(0, 6, size=c.nparameters())
    s = mq.BatchDensityMatrix(n, 0) if dm else mq.BatchStateVector(n, 0)
    H.handle()
    before = mq.launch_count()
    for how in ({}, {"plain": True}):
        assert mq.apply_(c, s, theta=theta, **how) is s
        assert mq.apply_(c, s, theta=np.zeros((0, c.nparameters())), **how) is s
    assert len(mq.expectation(H, s)) == 0
    out = mq.apply_observable(H, s)
    assert out.batch == 0
    assert mq.launch_count() == before
    with pytest.raises(Exception):
        mq.apply_(c, s, theta=np.full(c.nparameters(), np.nan))


def test_neighbours_are_untouched(mq, O):
    """A state beside many empty applies keeps its amplitudes."""
    from mossquantum_b200 import workloads as W
    n = 10
    c = W.hea_circuit(n, 2, W.hea_angles(n, 2, W.rng_for(1)))
    states = [mq.apply_(c, mq.StateVector(n)) for _ in range(4)]
    ref = O.apply(c.specs(), O.zero_state(n), n)
    for k in range(6):
        mq.apply_(W.hea_circuit(n, 2 + k, W.hea_angles(n, 2 + k, W.rng_for(k))), mq.BatchStateVector(n, 0))
    for s in states:
        assert np.max(np.abs(s.to_numpy() - ref)) <= 1e-12
