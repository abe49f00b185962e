"""An observable's strings go to the device with the first call that reads them there. 1e-11 as for every
expectation."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_made_by_the_first_reader(mq, O):
    from mossquantum_b200 import _native as N
    from mossquantum_b200 import workloads as W
    gc.collect()
    n = 6
    rng = np.random.default_rng(2)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v /= np.linalg.norm(v)
    s = mq.StateVector(v)
    rho = mq.DensityMatrix(s)
    H = W.xxz(n)
    ref = O.expect(v, n, H.specs())
    used = N.memory_info()[0]
    H.handle()
    dense = N.memory_info()[0] - used
    assert dense == 1280                              # five keys of 4x4 matrices and nothing else
    assert abs(mq.expectation(H, s) - ref) <= 1e-11
    assert N.memory_info()[0] - used == dense
    assert abs(mq.expectation(H, rho) - ref) <= 1e-11
    first = N.memory_info()[0] - used
    assert first > dense
    assert abs(mq.expectation(H, rho) - ref) <= 1e-11
    obj = mq.ExpectationObjective(mq.QCircuit([mq.RzGate(1, 0.2, isparas=True)]), H, s)
    assert abs(obj.evaluate([0.0]) - ref.real) <= 1e-11
    del H, obj
    gc.collect()
    assert N.memory_info()[0] <= used + (8 << 20)


def test_recorded_before_any_reader(mq, O):
    """A recording cannot put strings on the device, and stays on the dense keys."""
    import ctypes

    from mossquantum_b200 import _native as N
    from mossquantum_b200 import workloads as W
    n = 4
    rho = mq.DensityMatrix(mq.apply_(W.hea_circuit(n, 1, W.hea_angles(n, 1, W.rng_for(1))), mq.StateVector(n)))
    H = W.xxz(n)
    H.handle()
    L, dev, graph = N.lib(), ctypes.c_void_p(), ctypes.c_void_p()
    N.check(L.mb_buffer_alloc(16, ctypes.byref(dev)))
    N.check(L.mb_graph_begin())
    rc = L.mb_expect_to_device(H.handle().handle, rho.handle, dev)
    N.check(L.mb_graph_end(ctypes.byref(graph)))
    N.check(rc)
    N.check(L.mb_graph_launch(graph))
    out = np.zeros(2)
    N.check(L.mb_buffer_download(dev, N.dptr(out), 16))
    L.mb_graph_free(graph)
    L.mb_buffer_free(dev)
    assert abs(complex(out[0], out[1]) - np.trace(H.matrix(n) @ rho.to_numpy())) <= 1e-11
