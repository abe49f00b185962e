"""Staged expectation passes compile within the limits of the other generated kernels, and for wide
programs only once the observable is used again. 1e-11 as for every expectation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def observable(mq, n, step, names="XY", tail=0.3):
    """Flip masks and sign patterns of this step alone, so that no kernel of them is compiled already."""
    terms = [mq.QubitsTerm([1 + (step * k) % n, 1 + (step * k + 3) % n], [names[k % 2], "Z" if k % 3 else "Y"], 0.1 + 0.01 * k)
             for k in range(n)]
    return mq.QubitsOperator(terms + [mq.QubitsTerm([2, n], ["Z", "Z"], tail)])


def state(mq, n):
    rng = np.random.default_rng(n)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v /= np.linalg.norm(v)
    return v, mq.StateVector(v)


def seen(mq, H, s):
    from mossquantum_b200 import _native as N
    N.profile(True)
    got = mq.expectation(H, s)
    rep = N.profile_report()
    N.profile(False)
    return got, rep


@pytest.mark.parametrize("name,value,step", [("MB_JIT_MAX_SOURCE_KB", "1", 5), ("MB_JIT_BUDGET_S", "1e-9", 7)])
def test_past_a_limit(mq, O, monkeypatch, name, value, step):
    """Interpreted however often."""
    n = 24
    v, s = state(mq, n)
    H = observable(mq, n, step)
    ref = O.expect(v, n, H.specs())
    monkeypatch.setenv(name, value)
    for _ in range(3):
        got, rep = seen(mq, H, s)
        assert "k_pauli_pass" in rep and "mbk_pauli" not in rep and abs(got - ref) <= 1e-11


def test_wide_programs_compile_at_the_second_use(mq, O):
    n = 24
    v, s = state(mq, n)
    H = observable(mq, n, 11)
    ref = O.expect(v, n, H.specs())
    for call in range(3):
        got, rep = seen(mq, H, s)
        assert ("k_pauli_pass" in rep) == (call == 0) and ("mbk_pauli" in rep) == (call > 0)
        assert abs(got - ref) <= 1e-11
    # the same strings with other coefficients find the kernels
    again = observable(mq, n, 11, tail=-0.7)
    got, rep = seen(mq, again, s)
    assert "mbk_pauli" in rep and "k_pauli_pass" not in rep
    assert abs(got - O.expect(v, n, again.specs())) <= 1e-11


def test_prepared_plans_compile_before_they_are_recorded(mq, O):
    import ctypes

    from mossquantum_b200 import _native as N
    n = 24
    v, s = state(mq, n)
    H = observable(mq, n, 13)
    L, dev = N.lib(), ctypes.c_void_p()
    N.check(L.mb_buffer_alloc(16, ctypes.byref(dev)))
    N.profile(True)
    N.check(L.mb_expect_to_device(H.handle().handle, s.handle, dev))
    rep = N.profile_report()
    N.profile(False)
    assert "mbk_pauli" in rep and "k_pauli_pass" not in rep
    out = np.zeros(2)
    N.check(L.mb_buffer_download(dev, N.dptr(out), 16))
    L.mb_buffer_free(dev)
    assert abs(complex(out[0], out[1]) - O.expect(v, n, H.specs())) <= 1e-11


def test_narrow_programs_compile_at_once(mq, O):
    n = 16
    v, s = state(mq, n)
    H = observable(mq, n, 5)
    got, rep = seen(mq, H, s)
    assert "mbk_pauli" in rep and "k_pauli_pass" not in rep
    assert abs(got - O.expect(v, n, H.specs())) <= 1e-11
