"""Uploads of parameter values: the caller's memory is free again when a call returns, whatever memory it
is, and a call that cannot be recorded into a graph leaves later uploads as they were. 1e-12 max-abs on
amplitudes, the bound of the gate tests."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_page_locked_values_may_be_overwritten(mq, O):
    """More values than one staging buffer holds, in page-locked memory, changed right after the call."""
    import torch
    from mossquantum_b200 import workloads as W
    n, layers, B = 2, 43, 4200
    c = W.hea_circuit(n, layers)
    P = c.nparameters()
    assert B * P > 1 << 20
    values = np.random.default_rng(3).uniform(0, 2 * np.pi, size=(B, P))
    locked = torch.empty((B, P), dtype=torch.float64, pin_memory=True).numpy()
    for _ in range(3):
        locked[:] = values
        s = mq.apply_(c, mq.BatchStateVector(n, B), theta=locked)
        locked[:] = 0.0
        got = s.to_numpy()
        edge = (1 << 20) // P
        for b in (0, edge - 1, edge, edge + 1, B - 1):
            ref = O.apply(c.copy().reset_parameters(values[b]).specs(), O.zero_state(n), n)
            assert np.max(np.abs(got[:, b] - ref)) <= 1e-12


def test_gradient_is_refused_while_recording(mq, O):
    from mossquantum_b200 import _native as N
    from mossquantum_b200 import workloads as W
    n = 4
    c, H = W.hea_circuit(n, 1), W.tfim(n)
    rng = np.random.default_rng(4)
    theta = rng.uniform(0, 2 * np.pi, size=c.nparameters())
    obj = mq.ExpectationObjective(c, H, mq.StateVector(n))
    mq.value_and_gradient(mq.AdjointGradient(), obj, theta)
    L, graph = N.lib(), ctypes.c_void_p()
    N.check(L.mb_graph_begin())
    try:
        with pytest.raises(mq.UnsupportedOperation):
            mq.value_and_gradient(mq.AdjointGradient(), obj, theta)
    finally:
        rc = L.mb_graph_end(ctypes.byref(graph))
    assert rc == 0
    L.mb_graph_free(graph)
    for _ in range(10):
        theta = rng.uniform(0, 2 * np.pi, size=c.nparameters())
        got = mq.apply_(c, mq.StateVector(n), theta=theta).to_numpy()
        ref = O.apply(c.copy().reset_parameters(theta).specs(), O.zero_state(n), n)
        assert np.max(np.abs(got - ref)) <= 1e-12
