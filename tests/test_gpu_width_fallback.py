"""The register width a schedule falls back to is its own: a circuit whose passes are too long for either
width does not change the width of the next circuit of the same size. 1e-12 max-abs as in the gate tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(mq, O, monkeypatch, n, layers, limit):
    """Kernels seen and the tuned width after a circuit with sources of at most `limit` KB."""
    from mossquantum_b200 import _native as N
    from mossquantum_b200 import autotune
    from mossquantum_b200 import workloads as W
    monkeypatch.setenv("MB_JIT_MAX_SOURCE_KB", limit)
    c = W.u3_brickwork(n, layers, W.u3_params(n, layers, W.rng_for(5)))
    N.profile(True)
    got = mq.apply_(c, mq.StateVector(n)).to_numpy()
    seen = N.profile_report()
    N.profile(False)
    assert np.max(np.abs(got - O.apply(c.specs(), O.zero_state(n), n))) <= 1e-12
    return seen, autotune.get(n)


# largest sources in KB: 93 at 16 amplitudes per thread, 58 at 8 (six layers)
@pytest.mark.parametrize("n", [18, 20])
def test_fallback_stays_with_the_schedule(mq, O, monkeypatch, n):
    from mossquantum_b200 import autotune
    before = autotune.get(n)
    try:
        seen, width = run(mq, O, monkeypatch, n, 6, "30")
        assert "k_tile_pass" in seen            # partly interpreted at width 4
        assert width == before
        seen, width = run(mq, O, monkeypatch, n, 6, "75")
        assert "k_tile_pass" not in seen        # width 3 has every specialised kernel
        assert width == before
    finally:
        autotune.set(n, *before)


def test_autotuner_does_not_time_a_fallback_as_the_width_asked_for(mq, monkeypatch):
    """Widths 3 of both tiles exceed the limit, so neither may win."""
    from mossquantum_b200 import autotune
    from mossquantum_b200 import workloads as W
    n = 20
    before, fusion = autotune.get(n), autotune.get_fusion(n)
    monkeypatch.setenv("MB_JIT_MAX_SOURCE_KB", "30")
    try:
        c = W.u3_brickwork(n, 6, W.u3_params(n, 6, W.rng_for(6)))
        t, r, ms = autotune.autotune(c, mq.StateVector(n))
        assert r == 4
    finally:
        autotune.set(n, *before)
        autotune.set_fusion(n, fusion)
