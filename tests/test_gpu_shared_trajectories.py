"""Noisy complex128 shots of more trajectories than fit the GPU at once, which walk
one shared trajectory up to their first deviation from it, against the oracle's
literal trajectories, shot by shot, for every register and warp split of the state."""
import numpy as np
import pytest

import oracle as O
from quantumforge_gb300 import Circuit, Gate, NoiseChannel

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
