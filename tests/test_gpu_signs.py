"""In-order complex64 passes (parameterised runs) whose CZ signs wait: CZ between
lane, register, warp and outside qubits in a row, before and after diagonal,
dense and moving gates, at a pass's end, and passes without any, against the
CPU oracle.

Tolerance: an operation rounds each component at most twice, so after m
operations an amplitude of a normalised state is off by at most 2 sqrt(2) u m,
u = 2^-24."""
import math

import numpy as np
import pytest

import oracle as O
from quantumforge_gb300 import ParameterizedCircuit
from quantumforge_gb300 import _abi as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,share", [(12, 0.0), (12, 0.6), (13, 0.3), (14, 0.8), (16, 0.5), (18, 0.7)])
def test_runs_match_oracle(backend, n, share):
    rng = np.random.default_rng(n + int(100 * share))
    recs, params = [(A.OP_GATE, A.GATE_H, q, 0, 0, 0.0) for q in range(n)], []
    for _ in range(200):
        a, b = (int(q) for q in rng.permutation(n)[:2])
        kind = rng.uniform()
        if kind < share:
            recs.append((A.OP_CZ, 0, a, b, 0, 0.0))
        elif kind < share + 0.3 * (1 - share):
            recs.append(((A.OP_CNOT, A.OP_SWAP)[int(rng.integers(0, 2))], 0, a, b, 0, 0.0))
        elif rng.uniform() < 0.7:
            recs.append((A.OP_ROTATION, int(rng.integers(0, 3)), a, 0, len(params), 0.0))
            params.append(float(rng.uniform(-math.pi, math.pi)))
        else:
            recs.append((A.OP_GATE, int(rng.integers(0, 12)), a, 0, 0, float(rng.uniform(-math.pi, math.pi))))
    recs.append((A.OP_CZ, 0, 0, n - 1, 0, 0.0))
    ops, params = A.ops_array(recs), np.array(params)
    got = ParameterizedCircuit.from_ops(ops, params.size).run(params, n, dtype="c64", backend=backend).amplitudes()
    fixed = ops.copy()
    for r in fixed:
        if int(r["kind"]) == A.OP_ROTATION:
            r["theta"] = params[int(r["param"])]
            r["gate"] = (A.GATE_RX, A.GATE_RY, A.GATE_RZ)[int(r["gate"])]
            r["kind"], r["param"] = A.OP_GATE, 0
    want = O.run(fixed, n)
    assert np.abs(got - want).max() <= 2.0 * math.sqrt(2.0) * 2.0**-24 * (len(recs) + 8)
