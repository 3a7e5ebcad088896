"""Damping so weak that its Kraus operators are unitary to nine digits, in complex128
shots on the branch tree: the engine must not take them for unitary. The seed is
worked back from the draw it has to give: one just below and one just above the
measured qubit's probability, which the state of the no-event branch gives to
1e-15; the two draws lie 1e-11 from it, the damping moves it by about 1e-9."""
import numpy as np
import pytest

from quantumforge_gb300 import Circuit, Gate, NoiseChannel

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1


def unshift_right(y, k):
    x = y
    for _ in range(64 // k + 1):
        x = y ^ (x >> k)
    return x


def unshift_left(y, k):
    x = y
    for _ in range(64 // k + 1):
        x = y ^ ((x << k) & M64)
    return x


def seed_of_draw(u, draw):
    """A seed whose draw number `draw` (from 0) is u to 2^-53."""
    x = (int(u * 2.0**53) << 11) | 1
    for _ in range(draw + 1):  # xorshift64 undone
        x = unshift_right(unshift_left(x, 17), 7)
        x = unshift_left(x, 13)
    x = unshift_right(x, 31)  # splitmix64 undone
    x = x * pow(0x94D049BB133111EB, -1, 1 << 64) & M64
    x = unshift_right(x, 27)
    x = x * pow(0xBF58476D1CE4E5B9, -1, 1 << 64) & M64
    x = unshift_right(x, 30)
    return (x - 0x9E3779B97F4A7C15) & M64


def matrix(gate):
    from oracle import gate_matrix

    return np.asarray(gate_matrix(gate.code, gate.theta), dtype=complex).reshape(2, 2)


def apply(a, m, q):
    a = a.reshape(-1, 2, 1 << q)
    return np.einsum("ij,ajb->aib", m, a).reshape(-1)


def cnot(a, c, t):
    i = np.arange(a.size)
    return a[i ^ (((i >> c) & 1) << t)]


GAMMA = 1.5e-9
BEHIND = {"nothing": [], "x": [Gate.X], "phase": [Gate.Rz(0.4)], "real": [Gate.Ry(0.3)], "complex": [Gate.Rz(0.4), Gate.Rx(0.7)],
          "flipped phase": [Gate.X, Gate.Rz(0.4), Gate.X], "x then real": [Gate.X, Gate.Ry(0.3)]}


@pytest.mark.parametrize("channel", ["amplitude", "phase", "thermal"])
@pytest.mark.parametrize("flip", [False, True])
@pytest.mark.parametrize("behind", list(BEHIND))
@pytest.mark.parametrize("n", [2, 5, 13])
def test_kraus_factors_near_one(backend, n, behind, flip, channel):
    q, other = 1, n - 1 if n > 2 else 0
    kind = {"amplitude": NoiseChannel.AmplitudeDamping(GAMMA), "phase": NoiseChannel.PhaseDamping(GAMMA),
            "thermal": NoiseChannel.ThermalDamping(GAMMA, 1.0)}[channel]
    up = GAMMA * np.exp(-1.0) if channel == "thermal" else 0.0
    c = Circuit()
    a = np.zeros(1 << n, dtype=complex)
    a[0] = 1
    for gate, at in ((Gate.Ry(1.2), q), (Gate.Ry(0.5), other)):
        c.push(gate, at)
        a = apply(a, matrix(gate), at)
    c.channel(q, kind)
    a = apply(a, np.diag([np.sqrt(1 - up), np.sqrt(1 - GAMMA)]), q)
    a /= np.linalg.norm(a)
    if flip:  # the damped bit as the other qubit sees it
        c.cnot(other, q)
        a = cnot(a, other, q)
    for gate in BEHIND[behind]:
        c.push(gate, q)
        a = apply(a, matrix(gate), q)
    c.measure(q, 0)
    p = float((np.abs(a.reshape(-1, 2, 1 << q)[:, 1]) ** 2).sum())
    for u, outcome in ((p - 1e-11, 1), (p + 1e-11, 0)):
        got, _, _ = c.run_shots_packed(n, 1, seed_of_draw(u, 1), backend=backend, noise=True, exec_opts={"shots_engine": "tree"})
        assert got[0] == outcome
