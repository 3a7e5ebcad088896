"""Performance cases: the work that programs using this engine have it do.

``listed()`` are the cases that stand for the range, ``draw(rng)`` gives more
of the same ranges. ``prepare`` builds what a program holds before the call
(a circuit, a plan, a resident state, parameter values), ``run`` is one pass
through the public entry points, ``work`` the bytes and operations that pass
cannot do without, and ``exact`` the same result in 64 bits from plain torch.

Kinds:

* ``run``     ``ParameterizedCircuit.run`` at new parameters, amplitudes to the host
* ``sweep``   ``Circuit.run`` on a resident state
* ``shots``   ``Circuit.run_shots_packed``: simulate, then seeded terminal sampling
* ``noisy``   ``run_shots_packed(noise=True)``: one Kraus trajectory per shot
* ``density`` ``Circuit.run_density`` from a pure state, entries to the host
* ``grad``    ``gradient_with_inputs`` (adjoint): energy and the whole gradient
* ``train``   ``torch_ops.expectation`` forward and backward
* ``qaoa``    ``QaoaBatch.run``: cost and gradient of many MaxCut instances
"""
import math

import numpy as np
import torch

import quantumforge_gb300 as qf
from quantumforge_gb300 import _abi, gradients, torch_ops
from quantumforge_gb300 import workloads as W
from quantumforge_gb300._native import check, load
from quantumforge_gb300.qaoa import QaoaBatch

import ctypes

_AMP_BYTES = {"c64": 8, "c128": 16}


def listed():
    return [
        # the smallest call: a few-qubit variational circuit evaluated at new angles, all amplitudes read back
        {"name": "run_6q_c128", "kind": "run", "qubits": 6, "layers": 4, "dtype": "c128"},
        # the classic job: a 20-qubit depth-20 random circuit, every qubit measured, 10^5 seeded shots
        {"name": "shots_20q_c128", "kind": "shots", "qubits": 20, "depth": 20, "circuit": 1, "two_qubit": "ladder",
         "shots": 100000, "dtype": "c128"},
        # an ordinary single-precision simulation that stays inside L2
        {"name": "sweep_21q_c64", "kind": "sweep", "qubits": 21, "depth": 40, "circuit": 1, "two_qubit": "mixed",
         "dtype": "c64"},
        # the same in the default (double) precision, beyond L2
        {"name": "sweep_25q_c128", "kind": "sweep", "qubits": 25, "depth": 40, "circuit": 1, "two_qubit": "mixed",
         "dtype": "c128"},
        # the headline: the largest sweep, 8 GiB of amplitudes
        {"name": "sweep_30q_c64", "kind": "sweep", "qubits": 30, "depth": 40, "circuit": 1, "two_qubit": "mixed",
         "dtype": "c64"},
        # one optimiser step of a small variational model in the default precision
        {"name": "grad_9q_c128", "kind": "grad", "model": "tfim", "qubits": 9, "layers": 3, "checkpoint": 0,
         "dtype": "c128"},
        # one training step through the autograd binding, odd width, default precision of that binding
        {"name": "train_17q_c64", "kind": "train", "model": "tfim", "qubits": 17, "layers": 6, "checkpoint": 0,
         "dtype": "c64"},
        # the variational workload: 24 qubits, 384 parameters
        {"name": "grad_24q_c64", "kind": "grad", "model": "tfim", "qubits": 24, "layers": 8, "checkpoint": 4,
         "dtype": "c64"},
        # the large checkpointed adjoint: XXZ ring, a checkpoint per layer
        {"name": "grad_28q_c64", "kind": "grad", "model": "xxz", "qubits": 28, "layers": 4, "checkpoint": 1,
         "dtype": "c64"},
        # a batch of MaxCut instances of uneven width, cost and gradient of each
        {"name": "qaoa_512", "kind": "qaoa", "count": 512, "smallest": 12, "largest": 20, "depth": 4},
        # a noise study by trajectories: damping and depolarizing after every layer
        {"name": "noisy_12q_c128", "kind": "noisy", "qubits": 12, "layers": 4, "circuit": 7, "shots": 20000,
         "dtype": "c128"},
        # the same kind of study as a density matrix
        {"name": "density_10q_c128", "kind": "density", "qubits": 10, "layers": 6, "circuit": 7, "dtype": "c128"},
    ]


def draw(rng):
    """One more case of these ranges, none of the listed ones."""
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in known:
            return case


def _draw(rng):
    """A kind by how often programs call it, sizes over its range."""
    kind = rng.choice(["run", "sweep", "sweep", "shots", "noisy", "density", "grad", "grad", "train", "qaoa"])
    circuit = rng.randrange(2, 10**6)
    dtype = rng.choice(["c64", "c128"])
    if kind == "run":
        return {"kind": kind, "qubits": rng.randint(3, 18), "layers": rng.randint(1, 8), "dtype": dtype}
    if kind == "sweep":
        return {"kind": kind, "qubits": rng.randint(10, 28 if dtype == "c64" else 24), "depth": rng.randint(5, 40),
                "circuit": circuit, "two_qubit": rng.choice(["mixed", "ladder"]), "dtype": dtype}
    if kind == "shots":
        return {"kind": kind, "qubits": rng.randint(5, 22), "depth": rng.randint(5, 20), "circuit": circuit,
                "two_qubit": rng.choice(["mixed", "ladder"]), "shots": int(10 ** rng.uniform(2, 5)), "dtype": dtype}
    if kind == "noisy":
        return {"kind": kind, "qubits": rng.randint(4, 12), "layers": rng.randint(1, 4), "circuit": circuit,
                "shots": int(10 ** rng.uniform(2, 4.3)), "dtype": dtype}
    if kind == "density":
        return {"kind": kind, "qubits": rng.randint(3, 11), "layers": rng.randint(1, 6), "circuit": circuit,
                "dtype": dtype}
    if kind == "grad":
        return {"kind": kind, "model": rng.choice(["tfim", "xxz"]),
                "qubits": rng.randint(4, 26 if dtype == "c64" else 19), "layers": rng.randint(1, 5),
                "checkpoint": rng.choice([0, 0, 1, 2]), "dtype": dtype}
    if kind == "train":
        return {"kind": kind, "model": rng.choice(["tfim", "xxz"]), "qubits": rng.randint(4, 22),
                "layers": rng.randint(1, 6), "checkpoint": 0, "dtype": "c64"}
    smallest = 2 * rng.randint(2, 9)
    return {"kind": kind, "count": int(2 ** rng.uniform(3, 9)), "smallest": smallest,
            "largest": min(20, smallest + 2 * rng.randint(0, 5)), "depth": rng.randint(1, 4)}


# ---------------------------------------------------------------------------
# the circuits and inputs of a case
# ---------------------------------------------------------------------------
def _circuit(case):
    """The random circuit of a sweep or shots case."""
    return W.random_circuit(case["qubits"], case["depth"], case["circuit"], case["two_qubit"])


def _noisy_circuit(case):
    """Random layers, each followed by amplitude damping on every qubit and depolarizing on every other one."""
    n, c = case["qubits"], qf.Circuit()
    for layer in range(case["layers"]):
        for r in W.random_circuit(n, 1, case["circuit"] + layer):
            c.operations.append((int(r["kind"]), int(r["gate"]), int(r["q0"]), int(r["q1"]), 0, float(r["theta"]), 0))
        for q in range(n):
            c.channel(q, qf.NoiseChannel.AmplitudeDamping(0.02))
        for q in range(0, n, 2):
            c.channel(q, qf.NoiseChannel.Depolarizing(0.01))
    return c


def _ansatz(case):
    """(op records, parameter count) of the hardware-efficient ansatz of a case."""
    if case.get("model", "tfim") == "xxz":
        ops, params = W.hea_vqe(case["qubits"], case["layers"], 1, axes=(_abi.PAULI_X, _abi.PAULI_Y), entangler="cnot")
    else:
        ops, params = W.hea_vqe(case["qubits"], case["layers"], 1)
    return ops, params.size


def _hamiltonian(case):
    return (qf.PauliSum.xxz_ring if case["model"] == "xxz" else qf.PauliSum.tfim_ring)(case["qubits"])


def _angles(count, seed):
    return np.random.default_rng(seed).uniform(-math.pi, math.pi, count)


def _random_state(n, seed, dtype):
    """A normalised random state (complex Gaussian amplitudes) on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(2 << n, generator=g, device="cuda", dtype=torch.float32 if dtype == "c64" else torch.float64)
    x /= torch.sqrt((x.view(-1, 256) if n > 7 else x.view(1, -1)).square().sum(1, dtype=torch.float64).sum()).to(x.dtype)
    return torch.view_as_complex(x.view(-1, 2))


def _qaoa_inputs(case, seed):
    """Random 3-regular MaxCut instances of even widths, with their angles."""
    sizes = tuple(range(case["smallest"], case["largest"] + 1, 2))
    return W.qaoa_batch_problems(case["count"], sizes, case["depth"], seed % 1_000_003 + 1)


class _DeviceArray:
    """A resident state's amplitudes for ``torch.as_tensor`` (no copy); the tensor keeps this object, and so the
    state, alive."""

    def __init__(self, sv, dtype):
        self.state = sv
        p = ctypes.c_void_p()
        check(load().qf_sv_device_ptr(sv._h, ctypes.byref(p)))
        self.__cuda_array_interface__ = {"shape": (1 << sv.qubits,), "typestr": "<c8" if dtype == "c64" else "<c16",
                                         "data": (p.value, False), "version": 3}


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind, s = case["kind"], {"case": case, "seed": int(seed)}
    if kind in ("run", "grad", "train"):
        ops, count = _ansatz(case)
        s["circuit"] = qf.ParameterizedCircuit.from_ops(ops, count)
        s["params"] = _angles(count, seed)
        if kind != "run":
            s["hamiltonian"] = _hamiltonian(case)
            s["every"] = case["checkpoint"] * (3 * case["qubits"])  # operations of one layer
        if kind == "train":
            s["theta"] = torch.tensor(s["params"], requires_grad=True)
    elif kind == "sweep":
        s["circuit"] = qf.Circuit.from_ops(_circuit(case))
        s["state"] = qf.StateVector.zero(case["qubits"], dtype=case["dtype"])
        qf.default_backend().synchronize()
        s["amplitudes"] = torch.as_tensor(_DeviceArray(s["state"], case["dtype"]), device="cuda")
        s["amplitudes"].copy_(_random_state(case["qubits"], seed, case["dtype"]))
        torch.cuda.synchronize()  # the engine runs on a stream of its own
    elif kind == "shots":
        s["circuit"] = qf.Circuit.from_ops(W.with_terminal_measurements(_circuit(case), case["qubits"]))
    elif kind == "noisy":
        s["circuit"] = _noisy_circuit(case)
        for q in range(case["qubits"]):
            s["circuit"].measure(q, q)
    elif kind == "density":
        s["circuit"] = _noisy_circuit(case)
        psi = _random_state(case["qubits"], seed, case["dtype"]).to(torch.complex128).cpu().numpy()
        s["state"] = qf.StateVector.from_amplitudes(psi, dtype=case["dtype"])
    else:
        problems, s["gammas"], s["betas"] = _qaoa_inputs(case, seed)
        s["batch"] = QaoaBatch(problems, case["depth"])
    return s


def run(state):
    case = state["case"]
    kind, n = case["kind"], case.get("qubits")
    if kind == "run":
        return state["circuit"].run(state["params"], n, dtype=case["dtype"]).amplitudes()
    if kind == "sweep":
        state["circuit"].run(state["state"])
        return state["amplitudes"]
    if kind in ("shots", "noisy"):
        outcomes, _, ties = state["circuit"].run_shots_packed(n, case["shots"], state["seed"], dtype=case["dtype"],
                                                              noise=kind == "noisy")
        return outcomes.view(np.int64), ties
    if kind == "density":
        return state["circuit"].run_density(qf.DensityMatrix.from_state(state["state"])).entries()
    if kind == "grad":
        est = gradients.gradient_with_inputs(state["circuit"], gradients.GradientOptions(), [], state["params"], n,
                                             state["hamiltonian"], dtype=case["dtype"], checkpoint_every=state["every"])
        return est.expectation, est.gradient
    if kind == "train":
        theta = state["theta"]
        theta.grad = None
        energy = torch_ops.expectation(theta, state["circuit"], n, state["hamiltonian"], dtype=case["dtype"])
        energy.backward()
        return energy.detach(), theta.grad
    return state["batch"].run(state["gammas"], state["betas"])


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _gate_flops(ops):
    """Operations per amplitude of a gate list: two real multiplies and an add per component of a real or RX-type
    2x2, one complex multiply for a diagonal gate, nothing for permutations and signs."""
    dense = {_abi.GATE_H, _abi.GATE_RX, _abi.GATE_RY}
    flops = 0
    for r in ops:
        kind, gate = int(r["kind"]), int(r["gate"])
        if kind in (_abi.OP_ROTATION, _abi.OP_ENCODING):
            flops += 6
        elif kind == _abi.OP_GATE:
            flops += 6 if gate in dense or gate == _abi.GATE_RZ else 0
        elif kind == _abi.OP_CHANNEL:
            flops += 3
    return flops


def work(case):
    kind = case["kind"]
    if kind == "qaoa":
        sizes = range(case["smallest"], case["largest"] + 1, 2)
        amps = case["count"] * sum(2.0**n for n in sizes) / len(sizes)
        edges = case["count"] * sum(1.5 * n for n in sizes) / len(sizes)
        # per layer: the phase and n mixers forward, the same twice in reverse, and the two gradient terms
        per_amp = sum((3 * case["depth"] * (6 + 6 * n) + case["depth"] * (8 + 4 * n)) * 2.0**n for n in sizes) / sum(
            2.0**n for n in sizes)
        return {"bytes": 8 * edges + 8 * case["count"] * (4 * case["depth"] + 1), "flops": amps * per_amp}
    n = case["qubits"]
    amps, b = 2.0**n, _AMP_BYTES[case["dtype"]]
    if kind in ("run", "grad", "train"):
        ops, count = _ansatz(case)
        if kind == "run":
            return {"bytes": 8.0 * count + 16 * amps, "flops": amps * _gate_flops(ops)}
        terms = len(_hamiltonian(case))
        # forward, psi and lambda backward, an overlap (4 operations) per parameter, H psi
        return {"bytes": 16.0 * count + 32 * terms, "flops": amps * (3 * _gate_flops(ops) + 4 * count + 4 * terms)}
    if kind == "sweep":
        return {"bytes": 2 * b * amps, "flops": amps * _gate_flops(_circuit(case))}
    if kind == "shots":
        return {"bytes": 16 * amps + 8.0 * case["shots"], "flops": amps * _gate_flops(_circuit(case))}
    if kind == "noisy":
        return {"bytes": 16 * amps + 8.0 * case["shots"],
                "flops": case["shots"] * amps * _gate_flops(_noisy_circuit(case).ops())}
    return {"bytes": b * amps + 16 * amps * amps, "flops": 2 * amps * amps * _gate_flops(_noisy_circuit(case).ops())}


# ---------------------------------------------------------------------------
# exact: the same results in 64 bits from plain torch
# ---------------------------------------------------------------------------
_PAULI = {_abi.PAULI_X: [[0, 1], [1, 0]], _abi.PAULI_Y: [[0, -1j], [1j, 0]], _abi.PAULI_Z: [[1, 0], [0, -1]]}


def _matrix(op, params=None):
    kind, gate, theta = int(op["kind"]), int(op["gate"]), float(op["theta"])
    if kind == _abi.OP_ROTATION:
        gate, theta = (_abi.GATE_RX, _abi.GATE_RY, _abi.GATE_RZ)[gate], float(params[int(op["param"])])
    c, s, h = math.cos(theta / 2), math.sin(theta / 2), math.sqrt(0.5)
    return {_abi.GATE_H: [[h, h], [h, -h]], _abi.GATE_RX: [[c, -1j * s], [-1j * s, c]],
            _abi.GATE_RY: [[c, -s], [s, c]], _abi.GATE_RZ: [[complex(c, -s), 0], [0, complex(c, s)]]}[gate]


def _apply_matrix(v, q, m):
    """v <- m on bit q, in place."""
    w = v.view(-1, 2, 1 << q)
    a, b = w[:, 0], w[:, 1]
    if m[0][1] == 0 and m[1][0] == 0:
        a.mul_(m[0][0])
        b.mul_(m[1][1])
        return
    x = a * m[0][0] + b * m[0][1]
    y = a * m[1][0] + b * m[1][1]
    a.copy_(x)
    b.copy_(y)


def _apply_pair(v, kind, a, b):
    """CNOT (control a), CZ or SWAP of bits a, b, in place."""
    lo, hi = min(a, b), max(a, b)
    w = v.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)  # [rest, hi, between, lo, low]
    at = lambda bit_a, bit_b: w[:, bit_b, :, bit_a] if a == lo else w[:, bit_a, :, bit_b]  # noqa: E731
    if kind == _abi.OP_CZ:
        at(1, 1).neg_()
        return
    x, y = (at(1, 0), at(1, 1)) if kind == _abi.OP_CNOT else (at(1, 0), at(0, 1))
    t = x.clone()
    x.copy_(y)
    y.copy_(t)


def _apply(v, op, params=None):
    kind = int(op["kind"])
    if kind in (_abi.OP_GATE, _abi.OP_ROTATION):
        _apply_matrix(v, int(op["q0"]), _matrix(op, params))
    else:
        _apply_pair(v, kind, int(op["q0"]), int(op["q1"]))


def _apply_inverse(v, op, params):
    if int(op["kind"]) == _abi.OP_ROTATION:
        m = np.array(_matrix(op, params)).conj().T.tolist()
        _apply_matrix(v, int(op["q0"]), m)
    else:
        _apply(v, op, params)


def _times_pauli_sum(v, hamiltonian):
    """H v for real coefficients; Y = both masks set."""
    n = int(v.numel()).bit_length() - 1
    out = torch.zeros_like(v)
    for x, z, coeff in hamiltonian.terms:
        t = v.clone()
        for q in range(n):
            xq, zq = (x >> q) & 1, (z >> q) & 1
            if xq or zq:
                axis = _abi.PAULI_Y if xq and zq else _abi.PAULI_X if xq else _abi.PAULI_Z
                _apply_matrix(t, q, _PAULI[axis])
        out.add_(t, alpha=coeff.real)
    return out


def _zero_state(n):
    v = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    v[0] = 1
    return v


def _exact_gradient(case, params):
    ops, hamiltonian = _ansatz(case)[0], _hamiltonian(case)
    psi = _zero_state(case["qubits"])
    for op in ops:
        _apply(psi, op, params)
    lam = _times_pauli_sum(psi, hamiltonian)
    energy = torch.vdot(psi, lam).real.item()
    grad = np.zeros(len(params))
    for op in ops[::-1]:
        if int(op["kind"]) == _abi.OP_ROTATION:
            p, l = psi.view(-1, 2, 1 << int(op["q0"])), lam.view(-1, 2, 1 << int(op["q0"]))
            axis = int(op["gate"])
            if axis == _abi.PAULI_Z:
                d = (l[:, 0].conj() * p[:, 0]).sum() - (l[:, 1].conj() * p[:, 1]).sum()
            elif axis == _abi.PAULI_X:
                d = (l[:, 0].conj() * p[:, 1]).sum() + (l[:, 1].conj() * p[:, 0]).sum()
            else:
                d = 1j * ((l[:, 1].conj() * p[:, 0]).sum() - (l[:, 0].conj() * p[:, 1]).sum())
            grad[int(op["param"])] += d.imag.item()
        _apply_inverse(psi, op, params)
        _apply_inverse(lam, op, params)
    return energy, grad


def _exact_density(case, seed):
    n = case["qubits"]
    psi = _random_state(n, seed, case["dtype"]).to(torch.complex128)
    rho = torch.outer(psi, psi.conj()).reshape(-1)  # row-major: the row's qubit q is bit n + q
    for op in _noisy_circuit(case).ops():
        kind, q = int(op["kind"]), int(op["q0"])
        if kind == _abi.OP_GATE:
            m = _matrix(op)
            _apply_matrix(rho, n + q, m)
            _apply_matrix(rho, q, np.conj(m).tolist())
        elif kind == _abi.OP_CHANNEL:
            w = rho.view(-1, 2, 1 << (n - 1), 2, 1 << q)
            p = float(op["theta"])
            r00, r11 = w[:, 0, :, 0].clone(), w[:, 1, :, 1].clone()
            if int(op["gate"]) == _abi.CHANNEL_AMPLITUDE_DAMPING:
                w[:, 0, :, 0] = r00 + p * r11
                w[:, 1, :, 1] = (1 - p) * r11
                keep = math.sqrt(1 - p)
            else:
                w[:, 0, :, 0] = (1 - 2 * p / 3) * r00 + 2 * p / 3 * r11
                w[:, 1, :, 1] = (1 - 2 * p / 3) * r11 + 2 * p / 3 * r00
                keep = 1 - 4 * p / 3
            w[:, 0, :, 1] *= keep
            w[:, 1, :, 0] *= keep
        else:
            _apply_pair(rho, kind, n + q, n + int(op["q1"]))
            _apply_pair(rho, kind, q, int(op["q1"]))
    return rho.view(1 << n, 1 << n).cpu().numpy()


def _exact_qaoa(case, seed):
    problems, gammas, betas = _qaoa_inputs(case, seed)
    depth = case["depth"]
    cost, grad = np.zeros(len(problems)), np.zeros((len(problems), 2 * depth))
    for n in sorted({p[0] for p in problems}):
        every = [i for i, p in enumerate(problems) if p[0] == n]
        for begin in range(0, len(every), 64):
            rows = every[begin:begin + 64]
            index = torch.arange(1 << n, device="cuda")
            cut = torch.zeros(len(rows), 1 << n, dtype=torch.float64, device="cuda")
            for k, i in enumerate(rows):
                for u, v, _ in problems[i][1]:
                    cut[k] += ((index >> u) ^ (index >> v)) & 1
            edges = torch.tensor([len(problems[i][1]) for i in rows], dtype=torch.float64, device="cuda")[:, None]
            zz = edges - 2 * cut
            g, b = (torch.tensor(x[rows], device="cuda") for x in (gammas, betas))

            def mixer(v, angle):
                c, s = torch.cos(angle)[:, None, None], -1j * torch.sin(angle)[:, None, None]
                for q in range(n):
                    w = v.view(len(rows), -1, 2, 1 << q)
                    x, y = w[:, :, 0].clone(), w[:, :, 1].clone()
                    w[:, :, 0] = c * x + s * y
                    w[:, :, 1] = s * x + c * y

            psi = torch.full((len(rows), 1 << n), 2.0 ** (-n / 2), dtype=torch.complex128, device="cuda")
            for layer in range(depth):
                psi *= torch.exp(-1j * g[:, layer, None] * zz)
                mixer(psi, b[:, layer])
            lam = cut * psi
            cost[rows] = (psi.conj() * lam).real.sum(1).cpu().numpy()
            for layer in reversed(range(depth)):
                flipped = torch.zeros_like(psi)
                for q in range(n):
                    flipped += psi.view(len(rows), -1, 2, 1 << q).flip(2).reshape(len(rows), -1)
                grad[rows, depth + layer] = 2 * (lam.conj() * flipped).imag.sum(1).cpu().numpy()
                mixer(psi, -b[:, layer])
                mixer(lam, -b[:, layer])
                grad[rows, layer] = 2 * (lam.conj() * psi * zz).imag.sum(1).cpu().numpy()
                back = torch.exp(1j * g[:, layer, None] * zz)
                psi *= back
                lam *= back
    return cost, grad


def exact(case, seed):
    kind = case["kind"]
    if kind in ("shots", "noisy"):
        return None  # whole numbers
    if kind == "run":
        ops, count = _ansatz(case)
        params, v = _angles(count, seed), _zero_state(case["qubits"])
        for op in ops:
            _apply(v, op, params)
        return v.cpu().numpy()
    if kind == "sweep":
        if case["qubits"] > 27:
            return None  # over 20 seconds
        v = _random_state(case["qubits"], seed, case["dtype"]).to(torch.complex128)
        for op in _circuit(case):
            _apply(v, op)
        return v
    if kind in ("grad", "train"):
        if case["qubits"] > 25:
            return None  # over 20 seconds
        energy, grad = _exact_gradient(case, _angles(_ansatz(case)[1], seed))
        return energy, (torch.from_numpy(grad) if kind == "train" else grad)
    if kind == "density":
        return _exact_density(case, seed)
    return _exact_qaoa(case, seed)
