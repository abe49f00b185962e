"""Memory kept between small objectives is bounded: 8 MiB on the device, whatever the batch was. 1e-11 on
values, 1e-10 on gradients."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_batches_give_their_memory_back(mq, O):
    from mossquantum_b200 import _native as N
    from mossquantum_b200 import workloads as W
    n, layers, B = 2, 60, 6000
    gc.collect()
    before = N.memory_info()[0]
    c, H = W.hea_circuit(n, layers), W.tfim(n)
    theta = np.random.default_rng(1).uniform(0, 6, size=c.nparameters())
    w = np.zeros(B)
    w[[0, 17, B - 1]] = [0.5, -1.0, 2.0]
    v = np.random.default_rng(2).normal(size=(4, B)) + 0j
    v /= np.linalg.norm(v, axis=0)
    obj = mq.BatchExpectationObjective(c, H, mq.BatchStateVector(v), reduction="weighted_sum", weights=w)
    val, g = mq.value_and_gradient(mq.AdjointGradient(), obj, theta)
    specs = c.copy().reset_parameters(theta).specs()
    vr, gr = 0.0, 0.0
    for b in np.nonzero(w)[0]:
        vb, gb = O.adjoint(specs, v[:, b], n, H.specs())
        vr, gr = vr + w[b] * vb, gr + w[b] * gb
    assert abs(val - vr) <= 1e-11 and np.max(np.abs(g - gr)) <= 1e-10
    del obj, c, H
    gc.collect()
    assert N.memory_info()[0] - before <= (8 << 20) + 4096
