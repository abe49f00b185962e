"""MB_EXPECT_KEYS=1 keeps every expectation on the dense keys, those of objectives included. 1e-11 as for
every expectation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 11, 14])
def test_objectives_on_dense_keys(mq, O, monkeypatch, n):
    from mossquantum_b200 import _native as N
    from mossquantum_b200 import workloads as W
    c, H = W.hea_circuit(n, 1), W.xxz(n)
    theta = np.random.default_rng(n).uniform(0, 6, size=c.nparameters())
    obj = mq.ExpectationObjective(c, H, mq.StateVector(n))
    monkeypatch.setenv("MB_EXPECT_KEYS", "1")
    N.profile(True)
    got = obj.evaluate(theta)
    seen = N.profile_report()
    N.profile(False)
    assert not {"k_resident", "mbk_pauli", "k_pauli_pass"} & set(seen)
    ref = O.expect(O.apply(c.copy().reset_parameters(theta).specs(), O.zero_state(n), n), n, H.specs())
    assert abs(got - ref) <= 1e-11
