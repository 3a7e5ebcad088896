"""Register-tile passes (complex128 states, complex64 states below the compiled
passes' size) against the CPU oracle: every tile width, states smaller than a
tile and of many tiles, circuits long enough to be cut into several launches,
and the gates that the lowering keeps symbolic (X, Y, Z, S, CZ, CNOT, SWAP)
between dense ones.

Tolerance: an operation rounds each component at most twice (factor and sum),
so after m operations an amplitude of a normalised state is off by at most
2 sqrt(2) u m with u = 2^-24 (complex64) or 2^-53 (complex128)."""
import math

import numpy as np
import pytest

import oracle as O
from quantumforge_gb300 import ParameterizedCircuit, PauliSum, StateVector
from quantumforge_gb300 import _abi as A
from quantumforge_gb300.gradients import GradientOptions, GradientStrategy, gradient_with_inputs

pytestmark = pytest.mark.gpu


def bound(dtype, ops):
    return 2.0 * math.sqrt(2.0) * (2.0**-24 if dtype == "c64" else 2.0**-53) * (ops + 8)


def mixed_ops(rng, n, count, rotations=False):
    """Random gates: every kind, two-qubit gates on any pair, angles that include exact quarter turns."""
    recs, params = [], []
    for _ in range(count):
        kind = rng.integers(0, 10)
        q0, q1 = int(rng.integers(0, n)), int(rng.integers(0, n))
        theta = float(rng.choice([rng.uniform(-math.pi, math.pi), math.pi / 2, math.pi, 0.0], p=[0.85, 0.05, 0.05, 0.05]))
        if kind < 4 and q0 != q1:
            recs.append(((A.OP_CNOT, A.OP_CZ, A.OP_SWAP)[int(rng.integers(0, 3))], 0, q0, q1, 0, 0.0))
        elif rotations and kind < 8:
            recs.append((A.OP_ROTATION, int(rng.integers(0, 3)), q0, 0, len(params), 0.0))
            params.append(theta)
        else:
            recs.append((A.OP_GATE, int(rng.integers(0, 12)), q0, 0, 0, theta))
    return A.ops_array(recs), np.array(params)


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n,tile,count", [(1, 0, 12), (2, 0, 30), (3, 0, 40), (5, 0, 60), (6, 0, 60), (7, 6, 80), (8, 0, 80),
                                          (9, 7, 90), (10, 0, 100), (11, 8, 100), (12, 9, 120), (13, 10, 120),
                                          (14, 11, 120), (14, 12, 120), (17, 0, 150), (9, 0, 900), (13, 0, 900)])
def test_states_match_oracle(backend, n, tile, count, dtype):
    rng = np.random.default_rng(1000 * n + tile)
    ops, _ = mixed_ops(rng, n, count)
    init = rng.normal(size=2 << n).view(np.complex128)
    init /= np.linalg.norm(init)
    sv = StateVector.from_amplitudes(init, dtype=dtype, backend=backend)
    sv.apply_ops(ops, exec_opts={"tile_qubits": tile})
    want = O.run(ops, n, init=init)
    assert np.abs(sv.amplitudes() - want).max() <= bound(dtype, count)


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n,tile,count,every", [(1, 0, 10, 0), (4, 0, 40, 0), (6, 0, 60, 25), (9, 0, 120, 0), (9, 7, 120, 40),
                                                (12, 9, 120, 0), (13, 11, 120, 50), (14, 0, 120, 0), (7, 0, 500, 0)])
def test_gradients_match_oracle(backend, n, tile, count, every, dtype):
    rng = np.random.default_rng(77 * n + tile)
    ops, params = mixed_ops(rng, n, count, rotations=True)
    H = PauliSum.xxz_ring(n) if n > 2 else PauliSum([(1, 0, 0.7), (0, 1, -0.4)])
    pc = ParameterizedCircuit.from_ops(ops, params.size)
    est = gradient_with_inputs(pc, GradientOptions(strategy=GradientStrategy.Adjoint), [], params, n, H, dtype=dtype,
                               checkpoint_every=every, exec_opts={"tile_qubits": tile}, backend=backend)
    e, g = O.adjoint_uncompute(ops, n, params, H.array())
    # psi and lambda = H psi each carry the state's bound; |H| <= the sum of its coefficients
    tol = 4.0 * bound(dtype, 2 * count) * sum(abs(c) for _, _, c in H.terms)
    assert abs(est.expectation - e) <= tol and np.abs(est.gradient - g).max() <= tol
