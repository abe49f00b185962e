"""Objectives and the device adjoint gradient method.

Mirrors src/api/objectives.jl:15-244 (ExpectationObjective, BatchExpectationObjective,
evaluate, evaluate_batch), src/api/gradient_methods.jl:14-138 (value_and_gradient,
value_and_pullback, supports_gradient, differentiable_value) and the AdjointGradient
implementation of src/differentiation/objectives.jl:79-296, which here runs as one
``mb_adjoint`` call on the GPU.
"""
from __future__ import annotations

import numpy as np

from . import _native as N
from .backend import _validate_positions, backend, supports
from .circuit import ParameterMap, QCircuit, accumulate_parameter_gradients
from .operators import as_operator
from .states import _DeviceState


class UnsupportedGradient(Exception):
    """Mirror of MOSSQuantum.UnsupportedGradient (gradient_methods.jl:20-25)."""


class AdjointGradient:
    """Adjoint reverse sweep on the device (the B200 counterpart of CPU AdjointGradient)."""

    def __init__(self, checkpoint_every: int = 0):
        self.checkpoint_every = int(checkpoint_every)

    def __repr__(self):
        return f"AdjointGradient(checkpoint_every={self.checkpoint_every})"


B200AdjointGradient = AdjointGradient


class ExpectationObjective:
    """Re <H> after ``template`` bound to the input values, on a copy of ``initial_state``."""

    def __init__(self, template: QCircuit, observable, initial_state: _DeviceState, parameter_map=None):
        if not isinstance(template, QCircuit):
            template = QCircuit([template])
        self.template = template
        self.observable = as_operator(observable)
        self.initial_state = initial_state.copy()
        self.parameter_map = parameter_map if parameter_map is not None else ParameterMap(template)
        if len(self.parameter_map) != template.nparameters():
            raise ValueError("parameter map does not match the template")

    def nparameters(self):
        return self.parameter_map.nparameters()

    def _slots(self, values):
        values = np.asarray(values, dtype=np.float64)
        if values.shape != (self.nparameters(),):
            raise ValueError(f"expected {self.nparameters()} parameter values")
        if not np.all(np.isfinite(values)):
            raise ValueError("parameter values must be finite")
        return self.parameter_map.expand(values)

    def _sample_values(self, values):
        slots = self._slots(values)
        template, state, op = self.template, self.initial_state, self.observable
        key = template.value_key()
        known = template.known(state.n, key)
        if known is None:
            if not supports(backend(state), template, state, "apply"):
                raise N.UnsupportedOperation("B200Backend cannot apply this template")
            _validate_positions(template, state.n)
            compiled = template.compiled(state.n, values=key)
            template.remember(state.n, compiled, key)
        else:
            compiled = known[0]
        if not supports(backend(state), op, state, "expectation"):
            raise N.UnsupportedOperation("B200Backend cannot take the expectation of this observable")
        if op.nqubits() > state.n:
            raise ValueError("observable acts outside the register")
        theta = compiled.theta_from(slots)
        out = np.zeros(2 * state.batch)
        N.check(N.lib().mb_objective_values(compiled.handle, op.handle().handle, state.handle, N.ptr(theta), theta.size,
                                            N.ptr(out)), "evaluate")
        return out[0::2].copy()

    def evaluate(self, values) -> float:
        return float(self._sample_values(values)[0])


class BatchExpectationObjective(ExpectationObjective):
    """Batch objective reduced by ``:mean`` (default), ``:sum`` or ``:weighted_sum``."""

    def __init__(self, template, observable, initial_state, reduction="mean", weights=None, parameter_map=None):
        if not initial_state.is_batch:
            raise ValueError("BatchExpectationObjective needs a batch state")
        if initial_state.batch < 1:
            raise ValueError("scalar batch objectives require at least one sample")
        super().__init__(template, observable, initial_state, parameter_map)
        reduction = reduction.lstrip(":")
        if reduction not in ("mean", "sum", "weighted_sum"):
            raise ValueError("reduction must be mean, sum or weighted_sum")
        if reduction == "weighted_sum":
            if weights is None or len(weights) != initial_state.batch or not np.all(np.isfinite(weights)):
                raise ValueError("weighted_sum needs one finite weight per sample")
        elif weights is not None:
            raise ValueError("weights are only accepted with weighted_sum")
        self.reduction = reduction
        self.weights = None if weights is None else np.asarray(weights, dtype=np.float64)

    def sample_weights(self):
        B = self.initial_state.batch
        if self.reduction == "mean":
            return np.full(B, 1.0 / B)
        if self.reduction == "sum":
            return np.ones(B)
        return self.weights.copy()

    def evaluate_batch(self, values):
        return self._sample_values(values)

    def evaluate(self, values) -> float:
        return float(np.dot(self.sample_weights(), self.evaluate_batch(values)))


def evaluate(objective, values):
    return objective.evaluate(values)


def evaluate_batch(objective, values):
    return objective.evaluate_batch(values)


def supports_gradient(method, objective) -> bool:
    from .sampled import SAMPLED_METHODS, supports_sampled
    if isinstance(method, SAMPLED_METHODS):
        return supports_sampled(method, objective)
    return _gradient_circuit(method, objective) is not None


def _gradient_circuit(method, objective):
    """The compiled template if the adjoint method takes this objective, else None."""
    if not isinstance(method, AdjointGradient) or not isinstance(objective, ExpectationObjective):
        return None
    template, n = objective.template, objective.initial_state.n
    try:
        key = template.value_key()
        known = template.known(n, key)
        if known is not None:
            compiled = known[0]
        else:
            compiled = template.compiled(n, values=key)
            if supports(backend(objective.initial_state), template, objective.initial_state, "apply"):
                _validate_positions(template, n)
                template.remember(n, compiled, key)
    except Exception:
        return None
    return compiled if compiled.gradient_ok and objective.observable.is_hermitian() else None


def value_and_gradient(method, objective, values, rng=None):
    """(value, gradient) with one gradient entry per independent parameter. Adjoint gradients
    run as one device reverse sweep; ParameterShift / FiniteDifference / SPSAGradient evaluate
    their shifted parameter vectors as one batch on the device."""
    from .sampled import SAMPLED_METHODS, estimate_gradient
    if isinstance(method, SAMPLED_METHODS):
        est = estimate_gradient(method, objective, values, rng=rng)
        return est.value, est.gradient
    compiled = _gradient_circuit(method, objective)
    if compiled is None:
        raise UnsupportedGradient(f"{method!r} does not support this objective")
    slots = objective._slots(values)
    state = objective.initial_state
    theta = compiled.theta_from(slots)
    grad = np.zeros(max(1, compiled.nslots))
    value = np.zeros(1)
    weights = None
    if isinstance(objective, BatchExpectationObjective):
        weights = np.ascontiguousarray(objective.sample_weights())
    rc = N.lib().mb_adjoint(compiled.handle, objective.observable.handle().handle, state.handle, N.ptr(theta),
                            theta.size, None if weights is None else N.ptr(weights), method.checkpoint_every,
                            N.ptr(value), N.ptr(grad))
    N.check(rc, "value_and_gradient")
    return float(value[0]), accumulate_parameter_gradients(objective.parameter_map, compiled.gradient_from(grad))


def value_and_pullback(method, objective, values):
    """(value, back) with back(seed) = seed * gradient; the sweep runs once, on first use."""
    if not supports_gradient(method, objective):
        raise UnsupportedGradient(f"{method!r} does not support this objective")
    saved = np.array(values, dtype=np.float64, copy=True)
    value, grad = value_and_gradient(method, objective, saved)

    def back(seed):
        seed = float(seed)
        if seed == 0:
            return np.zeros_like(grad)
        return seed * grad

    return value, back


def differentiable_value(method, objective, values):
    return objective.evaluate(values)
