"""Lists whose SWAPs the planner takes out (more qubits than a tile, at least
twice as many SWAPs as the permutation left) against the CPU oracle: compiled
and register-tile passes, both precisions, states and gradients.

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


def swap_list(rng, n, count, rotations=False):
    """Half SWAPs (cyclic runs, repeated pairs, long range), CNOTs and CZs among one-qubit gates."""
    recs, params = [], []
    for i in range(count):
        a, b = (int(q) for q in rng.permutation(n)[:2])
        kind = rng.integers(0, 8)
        if kind < 4:
            recs.append((A.OP_SWAP, 0, *((a, b) if kind < 3 else (i % n, (i + 1) % n)), 0, 0.0))
        elif kind < 6:
            recs.append(((A.OP_CNOT, A.OP_CZ)[int(kind) - 4], 0, a, b, 0, 0.0))
        elif rotations:
            recs.append((A.OP_ROTATION, int(rng.integers(0, 3)), a, 0, len(params), 0.0))
            params.append(float(rng.uniform(-math.pi, math.pi)))
        else:
            recs.append((A.OP_GATE, int(rng.integers(0, 12)), a, 0, 0, float(rng.uniform(-math.pi, math.pi))))
    return A.ops_array(recs), np.array(params)


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n,count,opts", [(12, 100, {}), (13, 40, {}), (14, 300, {}), (16, 200, {"plan": "first_come"}),
                                          (17, 400, {}), (15, 300, {"jit": True}), (18, 200, {"jit": True})])
def test_states_match_oracle(backend, n, count, opts, dtype):
    rng = np.random.default_rng(10 * n + count)
    ops, _ = swap_list(rng, n, count)
    init = rng.normal(size=2 << n).view(np.complex128)
    init /= np.linalg.norm(init)
    sv = StateVector.from_amplitudes(init, dtype=dtype, backend=backend)
    sv.apply_ops(ops, exec_opts=opts)
    assert np.abs(sv.amplitudes() - O.run(ops, n, init=init)).max() <= bound(dtype, count)


@pytest.mark.parametrize("n,count,every", [(10, 150, 0), (13, 200, 0), (14, 200, 70)])
def test_gradients_match_oracle(backend, n, count, every):
    rng = np.random.default_rng(n)
    ops, params = swap_list(rng, n, count, rotations=True)
    H = PauliSum.xxz_ring(n)
    pc = ParameterizedCircuit.from_ops(ops, params.size)
    est = gradient_with_inputs(pc, GradientOptions(strategy=GradientStrategy.Adjoint), [], params, n, H, dtype="c128",
                               checkpoint_every=every, backend=backend)
    e, g = O.adjoint_uncompute(ops, n, params, H.array())
    tol = 4.0 * bound("c128", 2 * count) * sum(abs(c) for _, _, c in H.terms)
    assert abs(est.expectation - e) <= tol and np.abs(est.gradient - g).max() <= tol
