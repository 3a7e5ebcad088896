"""Backward complex64 passes in groups of ops against the shared-memory
interpreter: tiles of every width (one pair a thread up to 16 amplitudes a
thread), all overlap kinds inside and outside the tile, SWAPs between groups,
more overlaps in a pass than one batch holds.

Tolerance: below 12 qubits both run the same forward passes and every gate
and every thread's partial overlap is the same float32 operation, so only the
order of the final sums differs: 256 partial sums a tile in 53 bits or more,
each at most 4 |H| in sum. From 12 qubits on the forward passes differ too,
and the bound of a complex64 gradient holds: an operation rounds each
component at most twice."""
import math

import numpy as np
import pytest

from quantumforge_gb300 import ParameterizedCircuit, PauliSum
from quantumforge_gb300 import _abi as A
from quantumforge_gb300.gradients import GradientOptions, GradientStrategy, gradient_with_inputs

pytestmark = pytest.mark.gpu


def circuit(rng, n, count):
    recs, params = [], []
    for _ in range(count):
        q0, q1 = int(rng.integers(0, n)), int(rng.integers(0, n))
        kind = rng.integers(0, 10)
        theta = float(rng.uniform(-math.pi, math.pi))
        if kind < 3 and q0 != q1:
            recs.append(((A.OP_CNOT, A.OP_CZ, A.OP_SWAP)[int(rng.integers(0, 3))], 0, q0, q1, 0, 0.0))
        elif kind < 8:
            recs.append((A.OP_ROTATION, int(rng.integers(0, 3)), q0, 0, len(params), 0.0))
            params.append(theta)
        else:
            recs.append((A.OP_GATE, int(rng.integers(0, 12)), q0, 0, 0, theta))
    return A.ops_array(recs), np.array(params)


@pytest.mark.parametrize("n,count,every", [(1, 20, 0), (2, 40, 0), (3, 60, 0), (4, 60, 0), (5, 80, 0), (7, 120, 0), (8, 120, 30),
                                           (9, 160, 0), (10, 160, 0), (11, 160, 50), (12, 160, 0), (13, 200, 0), (16, 200, 90),
                                           (18, 240, 0), (9, 700, 0), (11, 700, 0)])
def test_matches_interpreter(backend, n, count, every):
    rng = np.random.default_rng(31 * n + count)
    ops, params = circuit(rng, n, count)
    H = PauliSum.xxz_ring(n) if n > 2 else PauliSum([(1, 0, 0.7), (0, 1, -0.4)])
    pc = ParameterizedCircuit.from_ops(ops, params.size)

    def grad(**opts):
        return gradient_with_inputs(pc, GradientOptions(strategy=GradientStrategy.Adjoint), [], params, n, H, dtype="c64",
                                    checkpoint_every=every, exec_opts=opts, backend=backend)

    got, want = grad(), grad(smem_tiles=True)
    size = sum(abs(c) for _, _, c in H.terms)
    tol = 4.0 * size * (2.0**-53 * 256 if n < 12 else 8.0 * math.sqrt(2.0) * 2.0**-24 * (2 * count + 8))
    assert abs(got.expectation - want.expectation) <= tol
    assert np.abs(got.gradient - want.gradient).max() <= tol
