"""Register width of forward schedules from 2^20 amplitudes: 16 amplitudes per thread, and 8 where a pass
would exceed the source limit; short segments keep 8. 1e-12 max-abs, the bound of the gate tests; the
two widths run the same gates with other groupings, so they agree to the same bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def state(mq, dm, c, n):
    return mq.apply_(c, mq.DensityMatrix(n) if dm else mq.StateVector(n)).to_numpy().ravel(order="F")


# limits in KB: between the largest sources of the two widths (58 and 93, 27 and 34), or above both
@pytest.mark.parametrize("n,dm,limit", [(19, False, "75"), (20, False, "128"), (20, False, "75"), (21, False, "75"),
                                        (10, True, "128"), (10, True, "30")])
def test_widths(mq, O, monkeypatch, n, dm, limit):
    from mossquantum_b200 import _native as N
    from mossquantum_b200 import workloads as W
    monkeypatch.setenv("MB_JIT_MAX_SOURCE_KB", limit)
    if dm:
        c = W.hea_circuit(n, 1, W.hea_angles(n, 1, W.rng_for(3)), noise=(0.01, 0.02))
    else:
        c = W.u3_brickwork(n, 6, W.u3_params(n, 6, W.rng_for(3)))
    ref = O.apply(c.specs(), O.zero_state(n, dm), n, dm)
    for _ in range(2):
        N.profile(True)
        got = state(mq, dm, c, n)
        seen = N.profile_report()
        N.profile(False)
        assert np.max(np.abs(got - ref)) <= 1e-12
        assert "k_tile_pass" not in seen
