"""Noisy complex128 shots (one trajectory per shot, register-tile kernels) against
the oracle's literal trajectories, shot by shot: every channel and measurement
kind in one circuit, runs of decisions broken by gates and by repeated qubits,
weak noise (most shots share the no-event trajectory) and strong noise, and
every register and warp split of the state (2 to 12 qubits)."""
import numpy as np
import pytest

import oracle as O
from quantumforge_gb300 import Circuit, Gate, NoiseChannel
from quantumforge_gb300 import _abi as A

pytestmark = pytest.mark.gpu


def noisy_circuit(rng, n, layers, strength, mid):
    c = Circuit()
    bit = 0
    for _ in range(layers):
        for q in range(n):
            code = int(rng.integers(0, 12))
            c.push(Gate(code, float(rng.uniform(-3, 3))), q)
        for q in range(n - 1):
            (c.cnot, c.cz, c.swap)[int(rng.integers(0, 3))](q, (q + 1 + int(rng.integers(0, n - 1))) % n if n > 2 else 1 - q)
        for q in rng.permutation(n):
            p = float(strength * rng.uniform(0.2, 1.0))
            kind = int(rng.integers(0, 5))
            if kind == 0:
                c.channel(int(q), NoiseChannel.AmplitudeDamping(p))
            elif kind == 1:
                c.channel(int(q), NoiseChannel.PhaseDamping(p))
            elif kind == 2:
                c.channel(int(q), NoiseChannel.ThermalDamping(p, 0.7))
            elif kind == 3:
                c.channel(int(q), NoiseChannel.Depolarizing(p))
                c.channel(int(q), NoiseChannel.AmplitudeDamping(p))  # populations may have flipped before it
            else:
                c.channel(int(q), NoiseChannel.AmplitudeDamping(p))
                c.channel(int(q), NoiseChannel.AmplitudeDamping(0.5 * p))  # the same qubit twice
                c.channel(int(q), NoiseChannel.Depolarizing(p))
        if mid and bit < 20:
            q = int(rng.integers(0, n))
            c.measure(q, bit)
            bit += 1
    for q in rng.permutation(n)[: max(1, n - 1)]:
        c.measure(int(q), 40 + int(q))
    return c


@pytest.mark.parametrize("strength", [0.02, 0.6])
@pytest.mark.parametrize("n,layers,mid", [(2, 4, True), (3, 3, False), (5, 3, True), (6, 3, False), (7, 3, True), (8, 2, False),
                                          (9, 2, True), (10, 2, False), (11, 2, True), (12, 2, False)])
def test_shots_match_literal_trajectories(backend, n, layers, mid, strength):
    rng = np.random.default_rng(10 * n + layers)
    c = noisy_circuit(rng, n, layers, strength, mid)
    shots = 300 if n < 9 else 60
    got, width, ties = c.run_shots_packed(n, shots, 17 + n, backend=backend, noise=True, tie_eps=1e-11,
                                          exec_opts={"shots_engine": "trajectories"})
    want, _ = O.run_shots(c.ops(), n, shots, 17 + n, noise=True)
    assert ties == 0 and np.array_equal(got, want)


def test_certain_events_and_idle_channels(backend):
    """Probabilities 0 and 1: the no-event branch of a step has no weight, or every draw follows it."""
    c = Circuit()
    for q in range(4):
        c.push(Gate.X, q)
    c.channel(0, NoiseChannel.AmplitudeDamping(1.0))
    c.channel(1, NoiseChannel.AmplitudeDamping(0.0))
    c.channel(2, NoiseChannel.Depolarizing(1.0))
    c.channel(3, NoiseChannel.Depolarizing(0.0))
    for q in range(4):
        c.measure(q, q)
    got, _, _ = c.run_shots_packed(4, 400, 5, backend=backend, noise=True)
    want, _ = O.run_shots(c.ops(), 4, 400, 5, noise=True)
    assert np.array_equal(got, want)
    assert np.all((got & 1) == 0) and np.all((got >> 1) & 1 == 1) and np.all((got >> 3) & 1 == 1)
