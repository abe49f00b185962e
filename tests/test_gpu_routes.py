"""Each form of an objective, with proof that it is the one that ran: the one-launch form, the fused
reverse passes and the plain sweep at the sizes where several of them apply, checkpoints, shared parameters, the
staged expectation passes, and the branches of the one-launch form that depend on the number of parameters or on shared
memory. 1e-11 on values, 1e-10 on gradients; two forms of one call agree to 1e-11 and 1e-10 as well."""
import numpy as np
import pytest

from tests.test_gpu_pauli_stages import spread, wide
from tests.test_gpu_resident import mixed_circuit, observable, unit

pytestmark = pytest.mark.gpu


def profiled(call):
    from mossquantum_b200 import _native as N
    N.profile(True)
    out = call()
    seen = N.profile_report()
    N.profile(False)
    return out, set(seen)


def weighted(O, specs, v, n, H, w):
    vr, gr = 0.0, 0.0
    for b, wb in enumerate(w):
        vb, gb = O.adjoint(specs, v[:, b], n, H.specs())
        vr, gr = vr + wb * vb, gr + wb * gb
    return vr, gr


def objective(mq, c, H, v, w):
    if len(w) == 1:
        return mq.ExpectationObjective(c, H, mq.StateVector(v[:, 0]))
    return mq.BatchExpectationObjective(c, H, mq.BatchStateVector(v), reduction="weighted_sum", weights=w)


@pytest.mark.parametrize("n,B", [(8, 1), (8, 3), (9, 1), (9, 2), (10, 1), (11, 3), (12, 1)])
def test_forms_of_small_gradients(mq, O, monkeypatch, n, B):
    from mossquantum_b200 import workloads as W
    c = W.hea_circuit(n, 3)
    theta = np.random.default_rng(n).uniform(0, 6, size=c.nparameters())
    H, v, w = W.xxz(n), unit(n, B, n), np.linspace(1.0, -0.5, B)
    vr, gr = weighted(O, c.copy().reset_parameters(theta).specs(), v, n, H, w)
    obj = objective(mq, c, H, v, w)
    for form, env in (("k_resident", {}), ("k_adjoint_pass_jit", {"MB_RESIDENT": "0"}),
                      (None, {"MB_RESIDENT": "0", "MB_ADJOINT_PLAIN": "1"})):
        for k, x in env.items():
            monkeypatch.setenv(k, x)
        for every in (0, 7):
            (val, g), seen = profiled(lambda: mq.value_and_gradient(mq.AdjointGradient(checkpoint_every=every), obj, theta))
            want = form if n >= 9 or form != "k_adjoint_pass_jit" else None     # the fused passes start at 9 qubits
            assert seen & {"k_resident", "k_adjoint_pass_jit"} == ({want} if want else set())
            assert abs(val - vr) <= 1e-11 and np.max(np.abs(g - gr)) <= 1e-10
        value, seen = profiled(lambda: obj.evaluate(theta))
        assert ("k_resident" in seen) == (form == "k_resident") and abs(value - vr) <= 1e-11
        for k in env:
            monkeypatch.delenv(k)


@pytest.mark.parametrize("n", [9, 11, 12])
def test_shared_parameters_in_the_fused_passes(mq, O, monkeypatch, n):
    from mossquantum_b200 import workloads as W
    c = W.hea_circuit(n, 3)
    P = c.nparameters()
    pm = mq.ParameterMap(c, [(i % (P // 3)) + 1 for i in range(P)])
    obj = mq.ExpectationObjective(c, W.tfim(n), mq.StateVector(n), parameter_map=pm)
    x = np.random.default_rng(1).uniform(0, 2 * np.pi, size=pm.nparameters())
    vr, gr = O.adjoint(c.copy().reset_parameters(pm.expand(x)).specs(), O.zero_state(n), n, W.tfim(n).specs())
    monkeypatch.setenv("MB_RESIDENT", "0")
    (v, g), seen = profiled(lambda: mq.value_and_gradient(mq.AdjointGradient(), obj, x))
    assert "k_adjoint_pass_jit" in seen and "k_resident" not in seen
    assert abs(v - vr) <= 1e-11 and np.max(np.abs(g - mq.accumulate_parameter_gradients(pm, gr))) <= 1e-10


@pytest.mark.parametrize("n,B,count,fallback", [(1, 1, 12, False), (3, 1, 30, True), (5, 2, 40, False), (9, 1, 60, False),
                                                (12, 2, 40, True), (12, 1, 60, False), (13, 1, 40, False)])
def test_mixed_gates_take_the_form_they_should(mq, n, B, count, fallback):
    rng = np.random.default_rng(100 * n + B)
    c, H, v = mixed_circuit(mq, n, count, rng, fallback), observable(mq, n, rng), unit(n, B, n)
    obj, theta = objective(mq, c, H, v, np.linspace(-0.5, 1.5, B)), np.array(c.active_parameters())
    for call in (lambda: mq.value_and_gradient(mq.AdjointGradient(), obj, theta), lambda: obj.evaluate(theta)):
        assert ("k_resident" in profiled(call)[1]) == (not fallback and n <= 12)


@pytest.mark.parametrize("n,layers,extra", [(4, 32, 0), (4, 32, 1), (5, 40, 0), (10, 20, 3)])
@pytest.mark.parametrize("B", [1, 3])
def test_parameters_in_the_launch_or_in_a_copy(mq, O, n, layers, extra, B):
    """384 parameters travel with the launch; 385 and 600 in a copy before it, beside the weights."""
    from mossquantum_b200 import workloads as W
    c = W.hea_circuit(n, layers)
    for k in range(extra):
        c.push(mq.RyGate(1 + k, 0.0, isparas=True))
    assert c.nparameters() in (384, 385, 600, 603)
    H, v, w = W.tfim(n), unit(n, B, n), np.linspace(1.0, -0.5, B)
    obj = objective(mq, c, H, v, w)
    rng = np.random.default_rng(n + extra)
    for _ in range(2):
        theta = rng.uniform(0, 6, size=c.nparameters())
        vr, gr = weighted(O, c.copy().reset_parameters(theta).specs(), v, n, H, w)
        (val, g), seen = profiled(lambda: mq.value_and_gradient(mq.AdjointGradient(), obj, theta))
        assert "k_resident" in seen
        assert abs(val - vr) <= 1e-11 and np.max(np.abs(g - gr)) <= 1e-10
        value, seen = profiled(lambda: obj.evaluate(theta))
        assert "k_resident" in seen and abs(value - vr) <= 1e-11


@pytest.mark.parametrize("n,layers,gradient", [(12, 30, False), (10, 60, False), (12, 8, True)])
def test_shared_memory_decides(mq, O, n, layers, gradient):
    """Plans that do not fit an SM with both states run in the fused passes, or gate by gate where even those
    have too long a source."""
    from mossquantum_b200 import workloads as W
    c = W.hea_circuit(n, layers)
    theta = np.random.default_rng(n).uniform(0, 6, size=c.nparameters())
    H, v = W.xxz(n), unit(n, 1, n)
    obj = objective(mq, c, H, v, [1.0])
    vr, gr = weighted(O, c.copy().reset_parameters(theta).specs(), v, n, H, [1.0])
    (val, g), seen = profiled(lambda: mq.value_and_gradient(mq.AdjointGradient(), obj, theta))
    assert ("k_resident" in seen) == gradient and (gradient or seen & {"k_adjoint_pass_jit", "k_dense"})
    assert abs(val - vr) <= 1e-11 and np.max(np.abs(g - gr)) <= 1e-10
    assert abs(obj.evaluate(theta) - vr) <= 1e-11


@pytest.mark.parametrize("n", [14, 18, 20])
def test_staged_passes_run(mq, O, n):
    from mossquantum_b200 import workloads as W
    rng = np.random.default_rng(n)
    v = unit(n, 1, n)
    s = mq.StateVector(v[:, 0])
    for H in (W.xxz(n), W.tfim(n), spread(mq, n, rng, True), spread(mq, n, rng, False), wide(mq, n, rng)):
        got, seen = profiled(lambda: mq.expectation(H, s))
        assert "mbk_psum" in seen
        assert abs(got - O.expect(v[:, 0], n, H.specs())) <= 1e-11
