"""A schedule that does not fit the memory budget gives back what it had allocated."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_failed_schedules_leave_nothing_behind(mq):
    from mossquantum_b200 import _native as N
    from mossquantum_b200 import workloads as W
    from mossquantum_b200.objectives import UnsupportedGradient
    n = 13
    H, state = W.tfim(n), mq.StateVector(n)
    theta = np.random.default_rng(1).uniform(0, 6, size=3 * n * 2)

    def call():
        obj = mq.ExpectationObjective(W.hea_circuit(n, 2), H, state)
        return mq.value_and_gradient(mq.AdjointGradient(), obj, theta)

    value, grad = call()
    gc.collect()
    used, budget = N.memory_info()
    failed = 0
    try:
        for extra in range(1 << 17, 1 << 20, 3 << 12):
            N.check(N.lib().mb_init(0, used + extra))
            try:
                v, g = call()
                assert abs(v - value) <= 1e-11 and np.max(np.abs(g - grad)) <= 1e-10
            except (mq.BudgetExceeded, UnsupportedGradient):
                failed += 1
            gc.collect()
            assert N.memory_info()[0] == used, extra
    finally:
        N.check(N.lib().mb_init(0, budget))
    assert failed
