"""Noisy complex128 shots of more trajectories than fit the GPU at once, which walk
one shared trajectory up to their first deviation from it, against the oracle's
literal trajectories, shot by shot, for every register and warp split of the state."""
import numpy as np
import pytest

import oracle as O
from quantumforge_gb300 import Circuit, Gate, NoiseChannel
from test_gpu_trajectories import noisy_circuit

pytestmark = pytest.mark.gpu


def shared_shots(n):
    """More than the CTAs of 32 << W threads that a GPU of 160 SMs holds."""
    return 5200 if n <= 9 else {10: 2600, 11: 1300, 12: 700}[n]


def check(c, n, shots, seed, backend):
    got, _, ties = c.run_shots_packed(n, shots, seed, backend=backend, noise=True, tie_eps=1e-11,
                                      exec_opts={"shots_engine": "trajectories"})
    want, _ = O.run_shots(c.ops(), n, shots, seed, noise=True)
    assert ties == 0 and np.array_equal(got, want)
    return got


@pytest.mark.parametrize("n", [2, 3, 6, 7, 8, 9, 10, 11, 12])
def test_no_event_branch_without_weight(backend, n):
    """Resets: damping of probability 1 on an excited qubit leaves the no-event branch
    nothing, and channels, gates and measurements follow."""
    c = Circuit()
    a, b, d = 0, n - 1, n // 2
    c.push(Gate.X, a)
    c.channel(a, NoiseChannel.AmplitudeDamping(1.0))
    c.push(Gate.H, a)
    c.channel(a, NoiseChannel.AmplitudeDamping(0.1))
    c.push(Gate.Rx(0.9), b)
    c.measure(b, 0)
    c.push(Gate.X, d)
    c.channel(d, NoiseChannel.ThermalDamping(1.0, 0.0))  # down and up with certainty
    c.push(Gate.Ry(0.7), d)
    c.channel(d, NoiseChannel.ThermalDamping(0.2, 0.5))
    for q in range(n - 1):
        c.cnot(q, q + 1)
    c.channel(b, NoiseChannel.PhaseDamping(1.0))
    c.push(Gate.Rx(1.3), b)
    c.channel(b, NoiseChannel.PhaseDamping(0.2))
    for q in range(n):
        c.push(Gate.Ry(0.4 + q), q)
        c.channel(q, NoiseChannel.AmplitudeDamping(0.05))
    for q in range(n):
        c.measure(q, 1 + q)
    check(c, n, shared_shots(n), 3 + n, backend)


@pytest.mark.parametrize("n,shots", [(2, 60), (2, 5200), (4, 60), (4, 5200), (9, 60), (12, 60), (12, 400)])
def test_depth_with_depolarizing_noise_alone(backend, n, shots):
    """No channel depends on the state, so nothing but the gates' own factors tells how far
    the stored amplitudes have grown: 1400 Hadamards."""
    c = Circuit()
    for _ in range(1400 // n):
        for q in range(n):
            c.push(Gate.H, q)
            c.channel(q, NoiseChannel.Depolarizing(0.01))
    for q in range(n):
        c.push(Gate.Ry(0.5 + q), q)
        c.measure(q, q)
    check(c, n, shots, 1 + n, backend)


@pytest.mark.parametrize("every", [1, 40, 300])
def test_depth_with_a_damping_channel_now_and_then(backend, every):
    """Runs that find the norm from the amplitudes between stretches that do not."""
    n = 5
    c = Circuit()
    for i in range(1600):
        q = i % n
        c.push(Gate.H if i % 3 else Gate.Ry(0.1 * i), q)
        c.channel(q, NoiseChannel.Depolarizing(0.005))
        if i % every == every - 1:
            c.channel(q, NoiseChannel.AmplitudeDamping(0.01))
    for q in range(n):
        c.measure(q, q)
    check(c, n, shared_shots(n), 9, backend)


@pytest.mark.parametrize("strength", [0.01, 0.5])
@pytest.mark.parametrize("n,layers,mid", [(2, 4, True), (3, 3, False), (5, 3, True), (6, 3, False), (7, 3, True), (8, 2, False),
                                          (9, 2, True), (10, 2, False), (11, 2, True), (12, 2, False), (12, 2, True)])
def test_shared_shots_match_literal_trajectories(backend, n, layers, mid, strength):
    c = noisy_circuit(np.random.default_rng(7 * n + layers), n, layers, strength, mid)
    check(c, n, shared_shots(n), 23 + n, backend)


def test_more_runs_than_snapshots(backend):
    """1100 runs (each iteration's CNOT acts on the qubit of the channel before it) of
    64 KB each: shots start from every second run's amplitudes."""
    n = 12
    c = Circuit()
    for i in range(1100):
        q, before = 7 * i % n, 7 * (i - 1) % n
        c.cnot(before, q)
        c.push(Gate.Ry(0.3 + i), q)
        c.channel(q, NoiseChannel.AmplitudeDamping(1e-3))
        if i % 100 == 50:
            c.measure(q, 20 + i // 100)
    for q in range(n):
        c.measure(q, q)
    check(c, n, 400, 4, backend)
