"""The work that programs have this framework do, as cases that can be timed and checked.

A case is a dict of plain values. ``listed`` names the fixed ones, ``draw`` gives more of the same
ranges, ``prepare`` makes what a program holds before the call (states, circuits, plans), ``run``
is one pass through the public entry points, and ``exact`` is the same result computed with plain
torch in 64 bits.
"""
import math

import numpy as np
import torch

import mossquantum_b200 as mq
from mossquantum_b200 import workloads as W
from mossquantum_b200.batch import BatchPlan


# ---------------------------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # One objective value of a small variational circuit: the optimiser's innermost call
        # (the 8-qubit scalar objective of the published repeated-evaluation benchmark).
        {"name": "evaluate_n8", "kind": "evaluate", "n": 8, "layers": 2, "model": "tfim"},
        # The same objective with its adjoint gradient.
        {"name": "gradient_n8", "kind": "gradient", "n": 8, "layers": 2, "model": "tfim", "checkpoint": False},
        # A mini-batch of 16 encoded inputs on 6 qubits, shared parameters, mean loss (the
        # published batch-evaluation configuration).
        {"name": "batch_gradient_n6_b16", "kind": "batch_gradient", "n": 6, "layers": 2, "batch": 16, "model": "tfim",
         "weighted": False},
        # A larger mini-batch: 48 weighted samples of 12 qubits.
        {"name": "batch_gradient_n12_b48", "kind": "batch_gradient", "n": 12, "layers": 4, "batch": 48, "model": "xxz",
         "weighted": True},
        # The reference's CPU-scheduling circuit: 20 qubits, 20 layers of RX/RY/RZ and a CNOT
        # ladder, angles bound on every call.
        {"name": "rotations_n20", "kind": "rotations", "n": 20, "layers": 20},
        # The scale circuit of the benchmark: 28 qubits, 20 layers of U3 and CZ brickwork.
        {"name": "brickwork_n28", "kind": "brickwork", "n": 28, "layers": 20},
        # The benchmark's large gradient: 24 qubits, 1152 angles, checkpoints every 4 layers.
        {"name": "gradient_n24", "kind": "gradient", "n": 24, "layers": 16, "model": "tfim", "checkpoint": True},
        # One noisy density matrix, circuit and energy: an odd size from the serving mix.
        {"name": "noisy_n9", "kind": "noisy", "n": 9, "layers": 4, "batch": 1, "model": "xxz"},
        # The benchmark's noisy mini-batch gradient: 64 density matrices of 10 qubits.
        {"name": "noisy_gradient_n10_b64", "kind": "noisy_gradient", "n": 10, "layers": 4, "batch": 64, "model": "tfim",
         "gamma": 0.0},
        # A prepared plan over samples of different sizes with their own parameters (serving-like
        # evaluation of many small circuits at once).
        {"name": "uneven_10_to_19", "kind": "uneven", "sizes": "10:24,13:16,16:8,19:4", "layers": 4, "model": "xxz"},
        # Energy of a large state that is already on the device.
        {"name": "expect_xxz_n26", "kind": "expect", "n": 26, "batch": 1, "model": "xxz"},
        # Readout of a final state: marginal probabilities of ten qubits and the reduced density
        # matrix of six.
        {"name": "readout_n22", "kind": "readout", "n": 22, "qubits": 10, "keep": 6, "at": 0},
    ]


def draw(rng):
    kind = rng.choice(["evaluate", "gradient", "batch_gradient", "rotations", "brickwork", "noisy", "noisy_gradient",
                       "uneven", "expect", "readout"])
    model = rng.choice(["tfim", "xxz"])
    if kind == "evaluate":
        return {"kind": kind, "n": rng.randint(4, 22), "layers": rng.randint(1, 8), "model": model}
    if kind == "gradient":
        n = rng.randint(4, 23)
        return {"kind": kind, "n": n, "layers": rng.randint(1, 12 if n < 18 else 6), "model": model,
                "checkpoint": rng.random() < 0.3}
    if kind == "batch_gradient":
        n = rng.randint(4, 14)
        batch = int(round(math.exp(rng.uniform(math.log(2), math.log(min(256, 1 << (20 - n)))))))
        return {"kind": kind, "n": n, "layers": rng.randint(1, 6), "batch": batch, "model": model,
                "weighted": rng.random() < 0.5}
    if kind == "rotations":
        return {"kind": kind, "n": rng.randint(9, 25), "layers": rng.randint(2, 20)}
    if kind == "brickwork":
        return {"kind": kind, "n": rng.randint(15, 27), "layers": rng.randint(2, 20)}
    if kind == "noisy":
        n = rng.randint(4, 12)
        batch = int(round(math.exp(rng.uniform(0, math.log(min(64, 1 << (24 - 2 * n)))))))
        return {"kind": kind, "n": n, "layers": rng.randint(1, 5), "batch": batch, "model": model}
    if kind == "noisy_gradient":
        n = rng.randint(4, 10)
        batch = int(round(math.exp(rng.uniform(0, math.log(64)))))
        return {"kind": kind, "n": n, "layers": rng.randint(1, 4), "batch": batch, "model": model,
                "gamma": rng.choice([0.0, 0.02])}
    if kind == "uneven":
        chosen = sorted(rng.sample(range(10, 21), rng.randint(2, 4)))
        return {"kind": kind, "sizes": ",".join("%d:%d" % (n, rng.randint(1, 24 if n < 16 else 6)) for n in chosen),
                "layers": rng.randint(1, 5), "model": model}
    if kind == "expect":
        n = rng.randint(10, 27)
        return {"kind": kind, "n": n, "batch": rng.randint(1, min(32, 1 << (27 - n))), "model": model}
    n = rng.randint(8, 24)
    qubits = rng.randint(1, min(n, 14))
    return {"kind": kind, "n": n, "qubits": qubits, "keep": rng.randint(2, min(9, n - 1)), "at": rng.randint(0, n - 1)}


# ---------------------------------------------------------------------------------------------
# What a program has in hand
# ---------------------------------------------------------------------------------------------
NOISE = 0.01          # depolarizing probability after every gate of the noisy circuits
GRADIENT_NOISE = 0.005
DAMPING = 0.02


class _Buffer:
    def __init__(self, state):
        self.state = state   # the tensor on this memory keeps the state alive
        count = state.nbytes // 16
        self.__cuda_array_interface__ = {"shape": (count, 2), "typestr": "<f8", "data": (state.device_ptr(), False),
                                         "version": 2, "strides": None}


def _view(state):
    """The state's amplitudes as a torch tensor on the same memory (real and imaginary parts)."""
    return torch.as_tensor(_Buffer(state), device="cuda")


class _Held:
    """A plan and its parameters; the plan's graph and buffers go with it."""

    def __init__(self, plan, thetas):
        self.plan, self.thetas = plan, thetas

    def __del__(self):
        self.plan.close()


def _rng(seed):
    return np.random.default_rng([20261203, seed])


def _observable(case):
    return (W.tfim if case["model"] == "tfim" else W.xxz)


def _sizes(case):
    return [tuple(int(x) for x in part.split(":")) for part in case["sizes"].split(",")]


def _product_states(n, batch, seed):
    """Encoded inputs: one RY(angle) per qubit on |0>, as a (2^n, batch) array."""
    half = 0.5 * _rng(seed).uniform(0, np.pi, size=(batch, n))
    v = np.ones((batch, 1))
    for q in range(n):
        one = np.stack([np.cos(half[:, q]), np.sin(half[:, q])], axis=1)
        v = (one[:, :, None] * v[:, None, :]).reshape(batch, -1)
    return np.ascontiguousarray(v.T).astype(np.complex128)


def _random_states(n, batch, seed):
    """Normalised random amplitudes, made on the GPU: (batch, 2^n, 2) doubles."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    v = torch.randn((batch, 1 << n, 2), generator=g, device="cuda", dtype=torch.float64)
    for b in range(batch):
        v[b] /= torch.linalg.vector_norm(v[b])
    return v


def _angles(count, seed):
    return _rng(seed + 1).uniform(0, 2 * np.pi, size=count)


def _weights(case, seed):
    w = _rng(seed + 2).uniform(0.5, 1.5, size=case["batch"])
    return w / w.sum()


def _picked(case):
    """1-based readout qubits: consecutive from `at`, around the register's end."""
    return [1 + (case["at"] + k) % case["n"] for k in range(case["qubits"])]


def _kept(case):
    """1-based qubits whose reduced density matrix is read: spread over the register."""
    n, keep = case["n"], case["keep"]
    return sorted({1 + (case["at"] + (k * n) // keep) % n for k in range(keep)})


def prepare(case, seed):
    mq.init(0)
    kind, layers = case["kind"], case.get("layers", 0)
    s = {"case": case}
    if kind in ("evaluate", "gradient"):
        n = case["n"]
        circuit = W.hea_circuit(n, layers)
        s["objective"] = mq.ExpectationObjective(circuit, _observable(case)(n), mq.StateVector(n))
        s["values"] = _angles(3 * n * layers, seed)
        s["method"] = mq.AdjointGradient(checkpoint_every=4 * (4 * n - 1) if case.get("checkpoint") else 0)
    elif kind == "batch_gradient":
        n = case["n"]
        states = mq.BatchStateVector(_product_states(n, case["batch"], seed))
        how = {"reduction": "weighted_sum", "weights": _weights(case, seed)} if case["weighted"] else {}
        s["objective"] = mq.BatchExpectationObjective(W.hea_circuit(n, layers), _observable(case)(n), states, **how)
        s["values"] = _angles(3 * n * layers, seed)
        s["method"] = mq.AdjointGradient()
    elif kind == "noisy_gradient":
        n = case["n"]
        states = mq.BatchDensityMatrix(mq.BatchStateVector(_product_states(n, case["batch"], seed)))
        circuit = W.hea_circuit(n, layers, noise=(GRADIENT_NOISE, case["gamma"]))
        s["objective"] = mq.BatchExpectationObjective(circuit, _observable(case)(n), states)
        s["values"] = _angles(3 * n * layers, seed)
        s["method"] = mq.AdjointGradient()
    elif kind == "rotations":
        n = case["n"]
        s["circuit"] = _rotations(n, layers)
        s["theta"] = _angles(n * layers, seed)
        s["state"] = mq.StateVector(n)
        s["view"] = _view(s["state"])
    elif kind == "brickwork":
        n = case["n"]
        s["circuit"] = W.u3_brickwork(n, layers, W.u3_params(n, layers, _rng(seed)))
        s["state"] = mq.StateVector(n)
        s["view"] = _view(s["state"])
    elif kind == "noisy":
        n, batch = case["n"], case["batch"]
        s["circuit"] = W.hea_circuit(n, layers, noise=(NOISE, DAMPING))
        s["theta"] = _angles(3 * n * layers, seed)
        s["state"] = mq.DensityMatrix(n) if batch == 1 else mq.BatchDensityMatrix(n, batch)
        s["observable"] = _observable(case)(n)
        s["view"] = _view(s["state"])
    elif kind == "uneven":
        groups = {n: (W.hea_circuit(n, layers), batch) for n, batch in _sizes(case)}
        s = _Held(BatchPlan(groups, _observable(case)), _uneven_thetas(case, seed))
    else:
        n, batch = case["n"], case.get("batch", 1)
        state = mq.StateVector(n) if batch == 1 else mq.BatchStateVector(n, batch)
        mq.synchronize()
        _view(state).copy_(_random_states(n, batch, seed).reshape(-1, 2))
        s["state"] = state
        if kind == "expect":
            s["observable"] = _observable(case)(n)
        else:
            s["qubits"] = _picked(case)
            kept = set(_kept(case))
            s["traced"] = [q for q in range(1, n + 1) if q not in kept]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return s


def _rotations(n, layers):
    """The CPU-scheduling circuit with active angles: (RX, RY, RZ)[(layer + qubit) mod 3]."""
    kinds = (mq.RxGate, mq.RyGate, mq.RzGate)
    c = mq.QCircuit()
    for layer in range(1, layers + 1):
        for q in range(1, n + 1):
            c.push(kinds[(layer + q - 1) % 3](q, 0.0, isparas=True))
        for q in range(1, n):
            c.push(mq.CNOTGate(q, q + 1))
    return c


def _uneven_thetas(case, seed):
    r = _rng(seed)
    return {n: r.uniform(0, 2 * np.pi, size=(batch, 3 * n * case["layers"])) for n, batch in _sizes(case)}


# ---------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------
def run(s):
    if isinstance(s, _Held):
        return s.plan.run(s.thetas)
    kind = s["case"]["kind"]
    if kind == "evaluate":
        return s["objective"].evaluate(s["values"])
    if kind in ("gradient", "batch_gradient", "noisy_gradient"):
        value, gradient = mq.value_and_gradient(s["method"], s["objective"], s["values"])
        return {"value": value, "gradient": gradient}
    if kind == "rotations":
        mq.apply_(s["circuit"], s["state"].set_zero(), theta=s["theta"])
        return s["view"]
    if kind == "brickwork":
        mq.apply_(s["circuit"], s["state"].set_zero())
        return s["view"]
    if kind == "noisy":
        mq.apply_(s["circuit"], s["state"].set_zero(), theta=s["theta"])
        return {"state": s["view"], "energy": mq.expectation(s["observable"], s["state"])
                if s["state"].is_batch else np.array(mq.expectation(s["observable"], s["state"]))}
    if kind == "expect":
        return np.array(mq.expectation(s["observable"], s["state"]))
    return {"probabilities": mq.probabilities(s["state"], s["qubits"]),
            "reduced": mq.partial_tr(s["state"], s["traced"]).to_numpy()}


def work(case):
    """Bytes: each state read and written once, each result written once. Flops: six per amplitude
    for every single-qubit unitary (a rotation between two phases), twelve per element of a
    density matrix for a noisy gate, eight per amplitude and flip group of an observable."""
    kind, n, layers = case["kind"], case.get("n", 0), case.get("layers", 0)
    size, batch = float(1 << n), case.get("batch", 1)
    if kind == "evaluate":
        return {"bytes": 16 * size, "flops": size * (6 * n * layers + 8 * n)}
    if kind in ("gradient", "batch_gradient"):
        return {"bytes": 16 * size * batch, "flops": batch * size * (n * layers * (6 + 3 * 16) + 16 * n)}
    if kind == "noisy_gradient":
        # the loss is linear in the state: the samples are read, their mean is reversed
        return {"bytes": 16 * size * size * batch, "flops": size * size * (2 * batch + n * layers * 5 * 12 * 4)}
    if kind == "rotations":
        return {"bytes": 16 * size, "flops": size * 4 * n * layers}
    if kind == "brickwork":
        return {"bytes": 16 * size, "flops": size * 6 * n * layers}
    if kind == "noisy":
        return {"bytes": 16 * size * size * batch, "flops": size * size * batch * n * layers * 5 * 12}
    if kind == "uneven":
        total = float(sum((1 << m) * b * m for m, b in _sizes(case)))
        amps = float(sum((1 << m) * b for m, b in _sizes(case)))
        return {"bytes": 16 * amps, "flops": total * (6 * layers + 8)}
    if kind == "expect":
        return {"bytes": 16 * size * batch, "flops": 8 * size * batch * n}
    reduced = float(1 << len(_kept(case)))
    return {"bytes": 16 * size + 8.0 * (1 << case["qubits"]) + 16 * reduced ** 2, "flops": 3 * size + 8 * size * reduced}


# ---------------------------------------------------------------------------------------------
# The same results in plain torch, 64 bits
# ---------------------------------------------------------------------------------------------
def _t(x):
    return torch.as_tensor(np.asarray(x), device="cuda")


def _rotation(axis, theta):
    """2x2 entries (m00, m01, m10, m11) of exp(-i theta P / 2); theta a float or a (B, 1, 1) tensor."""
    half = 0.5 * theta if torch.is_tensor(theta) else torch.tensor(0.5 * float(theta), dtype=torch.float64, device="cuda")
    c, s = torch.cos(half).to(torch.complex128), torch.sin(half).to(torch.complex128)
    if axis == "x":
        return c, -1j * s, -1j * s, c
    if axis == "y":
        return c, -s, s, c
    z = torch.zeros_like(c)
    return c - 1j * s, z, z, c + 1j * s


def _apply(v, q, m):
    """2x2 on bit q of a (B, 2^bits) tensor."""
    x = v.view(v.shape[0], -1, 2, 1 << q)
    out = torch.empty_like(x)
    out[:, :, 0] = m[0] * x[:, :, 0] + m[1] * x[:, :, 1]
    out[:, :, 1] = m[2] * x[:, :, 0] + m[3] * x[:, :, 1]
    return out.view_as(v)


def _dagger(m):
    return m[0].conj(), m[2].conj(), m[1].conj(), m[3].conj()


def _conj(m):
    return tuple(e.conj() for e in m)


def _cnot(v, c, t):
    """CNOT with adjacent bits t = c + 1."""
    x = v.view(v.shape[0], -1, 2, 2, 1 << c).clone()   # [.., t, c, ..]
    x[:, :, :, 1] = x[:, :, :, 1].flip(2)
    return x.view_as(v)


def _pauli(v, q, p):
    x = v.view(v.shape[0], -1, 2, 1 << q)
    if p == "x":
        return x.flip(2).reshape_as(v)
    sign = torch.tensor([1.0, -1.0], dtype=torch.float64, device="cuda").view(1, 1, 2, 1)
    if p == "z":
        return (x * sign).reshape_as(v)
    return (1j * (x * sign).flip(2)).reshape_as(v)


def _terms(model, n):
    if model == "tfim":
        return [(-1.0, [(i, "z"), (i + 1, "z")]) for i in range(n - 1)] + [(-1.0, [(i, "x")]) for i in range(n)]
    return [(c, [(i, p), (i + 1, p)]) for i in range(n - 1) for p, c in (("x", 1.0), ("y", 1.0), ("z", 0.5))]


def _hamiltonian(v, model, n):
    out = torch.zeros_like(v)
    for c, ops in _terms(model, n):
        w = v
        for q, p in ops:
            w = _pauli(w, q, p)
        out += c * w
    return out


def _dot(a, b):
    return (a.conj() * b).sum(dim=1)


def _ladder(n, layers):
    """The ansatz: per layer RX, RY, RZ on each qubit, then CNOT(i, i + 1)."""
    ops, k = [], 0
    for _ in range(layers):
        for q in range(n):
            for axis in "xyz":
                ops.append((axis, q, k))
                k += 1
        ops += [("cnot", q, -1) for q in range(n - 1)]
    return ops


def _forward(v, ops, theta):
    """theta: (P,) shared angles or (B, P) per sample."""
    for op, q, k in ops:
        if op == "cnot":
            v = _cnot(v, q, q + 1)
        else:
            v = _apply(v, q, _rotation(op, theta[k] if theta.ndim == 1 else _t(theta[:, k]).view(-1, 1, 1)))
    return v


def _ground(n, batch=1):
    v = torch.zeros((batch, 1 << n), dtype=torch.complex128, device="cuda")
    v[:, 0] = 1
    return v


def _pure_gradient(v, ops, theta, model, n, weights):
    y = _forward(v, ops, theta)
    d = _hamiltonian(y, model, n)
    value = float((weights * _dot(y, d).real).sum())
    grad = np.zeros(len(theta))
    for op, q, k in reversed(ops):
        if op == "cnot":
            y, d = _cnot(y, q, q + 1), _cnot(d, q, q + 1)
            continue
        grad[k] = float((weights * _dot(d, _pauli(y, q, op)).imag).sum())
        m = _dagger(_rotation(op, theta[k]))
        y, d = _apply(y, q, m), _apply(d, q, m)
    return {"value": value, "gradient": grad}


def _noise_entries(p, gamma):
    """Depolarizing(p) then damping(gamma) on (rho00, rho10, rho01, rho11): the population mixing
    (to 00 from 00 and 11, to 11 from 00 and 11) and the factor of the coherences."""
    a, b = 1 - p / 2, p / 2
    return a + gamma * b, b + gamma * a, (1 - gamma) * b, (1 - gamma) * a, math.sqrt(1 - gamma) * (1 - p)


def _channel(v, q, n, e, adjoint=False):
    x = v.view(v.shape[0], -1, 2, 1 << (n - 1), 2, 1 << q)   # [.., column bit, .., row bit, ..]
    m00, m01, m10, m11, c = e
    if adjoint:
        m01, m10 = m10, m01
    out = x * c
    out[:, :, 0, :, 0] = m00 * x[:, :, 0, :, 0] + m01 * x[:, :, 1, :, 1]
    out[:, :, 1, :, 1] = m10 * x[:, :, 0, :, 0] + m11 * x[:, :, 1, :, 1]
    return out.view_as(v)


def _noisy_ops(n, layers):
    ops = []
    for op in _ladder(n, layers):
        ops.append(op)
        ops += [("noise", q, -1) for q in ((op[1],) if op[0] != "cnot" else (op[1], op[1] + 1))]
    return ops


def _noisy_step(r, op, q, k, n, theta, e):
    if op == "noise":
        return _channel(r, q, n, e)
    if op == "cnot":
        return _cnot(_cnot(r, q, q + 1), q + n, q + n + 1)
    m = _rotation(op, theta[k])
    return _apply(_apply(r, q, m), q + n, _conj(m))


def _trace(r, n):
    dim = 1 << n
    return r.view(-1, dim, dim).diagonal(dim1=1, dim2=2).sum(dim=1)


def _noisy_gradient(r, n, layers, theta, model, e):
    ops = _noisy_ops(n, layers)
    kept = {}
    for i, (op, q, k) in enumerate(ops):
        r = _noisy_step(r, op, q, k, n, theta, e)
        if k >= 0:
            kept[i] = r
    value = float(_trace(_hamiltonian(r, model, n), n).real.sum())
    d = torch.eye(1 << n, dtype=torch.complex128, device="cuda").view(1, -1)
    d = _hamiltonian(d, model, n)
    grad = np.zeros(len(theta))
    for i in range(len(ops) - 1, -1, -1):
        op, q, k = ops[i]
        if op == "noise":
            d = _channel(d, q, n, e, adjoint=True)
        elif op == "cnot":
            d = _cnot(_cnot(d, q, q + 1), q + n, q + n + 1)
        else:
            grad[k] = float(_dot(d, _pauli(kept.pop(i), q, op)).imag.sum())
            m = _dagger(_rotation(op, theta[k]))
            d = _apply(_apply(d, q, m), q + n, _conj(m))
    return {"value": value, "gradient": grad}


def _brickwork(case, seed):
    """Layers of U3 as Kronecker blocks of up to seven qubits: each block multiplies the lowest
    bits and rotates them to the top, so a layer ends in the original order."""
    n, layers = case["n"], case["layers"]
    p = W.u3_params(n, layers, _rng(seed))
    v = _ground(n).view(-1)
    for layer in range(layers):
        for first in range(0, n, 7):
            block = np.ones((1, 1))
            for q in range(first, min(n, first + 7)):
                th, phi, lam = p[layer, q]
                c, s = math.cos(th / 2), math.sin(th / 2)
                u = np.array([[c, -np.exp(1j * lam) * s], [np.exp(1j * phi) * s, np.exp(1j * (phi + lam)) * c]])
                block = np.kron(u, block)
            # rows of the product are the block's bits, so they end up on top
            v = (_t(block) @ v.view(-1, block.shape[0]).T).reshape(-1)
        for q in range(layer % 2, n - 1, 2):
            v.view(-1, 2, 2, 1 << q)[:, 1, 1].neg_()
    return torch.view_as_real(v)


def exact(case, seed):
    kind = case["kind"]
    if kind == "uneven":
        got, thetas = {}, _uneven_thetas(case, seed)
        for n, batch in _sizes(case):
            y = _forward(_ground(n, batch), _ladder(n, case["layers"]), thetas[n])
            got[n] = _dot(y, _hamiltonian(y, case["model"], n)).cpu().numpy()
        return got
    n, layers, batch = case["n"], case.get("layers", 0), case.get("batch", 1)
    if kind == "evaluate":
        y = _forward(_ground(n), _ladder(n, layers), _angles(3 * n * layers, seed))
        return float(_dot(y, _hamiltonian(y, case["model"], n)).real[0])
    if kind == "gradient":
        return _pure_gradient(_ground(n), _ladder(n, layers), _angles(3 * n * layers, seed), case["model"], n, 1.0)
    if kind == "batch_gradient":
        v = _t(np.ascontiguousarray(_product_states(n, batch, seed).T))
        w = _t(_weights(case, seed)) if case["weighted"] else 1.0 / batch
        return _pure_gradient(v, _ladder(n, layers), _angles(3 * n * layers, seed), case["model"], n, w)
    if kind == "noisy_gradient":
        # the loss is linear in the state, so the mean of the inputs stands for all of them
        v = _t(_product_states(n, batch, seed))
        r = (v.conj() @ v.T).reshape(1, -1) / batch
        return _noisy_gradient(r, n, layers, _angles(3 * n * layers, seed), case["model"],
                               _noise_entries(GRADIENT_NOISE, case["gamma"]))
    if kind == "noisy":
        theta, e = _angles(3 * n * layers, seed), _noise_entries(NOISE, DAMPING)
        r = _ground(2 * n)
        for op, q, k in _noisy_ops(n, layers):
            r = _noisy_step(r, op, q, k, n, theta, e)
        energy = _trace(_hamiltonian(r, case["model"], n), n).cpu().numpy()
        energy = energy[0] if batch == 1 else np.repeat(energy, batch)
        return {"state": torch.view_as_real(r.view(-1).repeat(batch)), "energy": np.array(energy)}
    if kind == "rotations":
        theta, ops, k = _angles(n * layers, seed), [], 0
        for layer in range(1, layers + 1):
            for q in range(1, n + 1):
                ops.append(("xyz"[(layer + q - 1) % 3], q - 1, k))
                k += 1
            ops += [("cnot", q, -1) for q in range(n - 1)]
        return torch.view_as_real(_forward(_ground(n), ops, theta).view(-1))
    if kind == "brickwork":
        return _brickwork(case, seed)
    v = torch.view_as_complex(_random_states(n, batch, seed))
    if kind == "expect":
        e = _dot(v, _hamiltonian(v, case["model"], n)).cpu().numpy()
        return np.array(e[0]) if batch == 1 else e
    # bits of the picked (or kept) qubits lowest, in order: dimension of bit q is n - 1 - q
    def lowest(bits):
        rest = [b for b in range(n) if b not in bits]
        order = [n - 1 - b for b in reversed(rest)] + [n - 1 - b for b in reversed(bits)]
        return v.view([2] * n).permute(order).reshape(-1, 1 << len(bits))
    p = lowest([q - 1 for q in _picked(case)]).abs().square().sum(dim=0)
    m = lowest([q - 1 for q in _kept(case)])
    return {"probabilities": (p / p.sum()).cpu().numpy(), "reduced": (m.T @ m.conj()).cpu().numpy()}
