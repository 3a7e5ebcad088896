"""Cut values of batched QAOA instances whose edges all lie above a tile's low 12
bits, where each tile adds one constant: more instances than a CTA's run of tiles
covers, and fewer, against the oracle.

Tolerance: an operation rounds each component at most twice (u = 2^-24), a layer
has n mixer gates and one phase, there and back, and C is at most W: 16 sqrt(2) u p
(n + 1) W on the energy, W more on dE/dgamma, n on dE/dbeta."""
import numpy as np
import pytest

import oracle as O
from quantumforge_gb300 import PauliSum
from quantumforge_gb300 import workloads as W
from quantumforge_gb300.qaoa import QaoaBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count", [(14, 200), (15, 90), (17, 40), (18, 3)])
def test_edges_above_the_low_bits(backend, n, count):
    rng = np.random.default_rng(n)
    pairs = [(u, v) for u in range(12, n) for v in range(12, u)]
    problems = [(n, [(*pairs[i], 1.0) for i in rng.permutation(len(pairs))[: int(rng.integers(1, len(pairs) + 1))]])
                for _ in range(count)]
    assert all(problems[i][1] for i in range(count))
    gam, bet = rng.uniform(0, np.pi, (count, 1)), rng.uniform(-np.pi, np.pi, (count, 1))
    cost, grad = QaoaBatch(problems, 1, backend=backend).run(gam, bet)
    for i in sorted({0, 1, count // 2, count - 2, count - 1}):
        ed = problems[i][1]
        e, g = O.adjoint_uncompute(W.qaoa_param_circuit(n, ed, 1), n, np.array([2 * gam[i, 0], 2 * bet[i, 0]]),
                                   PauliSum.maxcut(ed).array())
        tol = 16.0 * np.sqrt(2.0) * 2.0**-24 * (n + 1) * (len(ed) + 1)
        assert abs(cost[i] - e) <= tol and np.abs(grad[i] - 2 * g).max() <= tol * (len(ed) + n + 1)
