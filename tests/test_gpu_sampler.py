"""Terminal measurements against the CPU oracle, outcome by outcome: trees of
one fold, of two and of a remainder, fewer low indices than a run, shot counts
around a warp and a block, outcomes that are certain, skewed or a tie away, and
states whose norm is not 1.

Whole numbers: a shot differs only where a uniform falls within the rounding of
its probability (about 1e-15, none in these 10^6 draws)."""
import numpy as np
import pytest

import oracle as O
from quantumforge_gb300 import StateVector
from quantumforge_gb300 import _abi as A

pytestmark = pytest.mark.gpu


def measure(qubits):
    return A.ops_array([(A.OP_MEASURE, 0, int(q), 0, j, 0.0) for j, q in enumerate(qubits)])


@pytest.mark.parametrize("n,m,shots", [(1, 1, 1), (2, 2, 31), (3, 1, 33), (5, 5, 1000), (9, 9, 4097), (10, 10, 129), (11, 11, 5000),
                                       (13, 12, 3000), (14, 13, 127), (20, 20, 20000), (21, 21, 1025), (16, 3, 40000)])
@pytest.mark.parametrize("kind", ["dense", "skewed"])
def test_shots_match_the_oracle(backend, n, m, shots, kind):
    rng = np.random.default_rng(1000 * n + m)
    psi = rng.normal(size=2 << n).view(np.complex128)
    if kind == "skewed":  # outcomes near certainty on half of the qubits
        for q in range(0, n, 2):
            psi.reshape(-1, 2, 1 << q)[:, q % 4 // 2, :] *= 1e-3
    psi /= np.linalg.norm(psi)
    qubits = rng.permutation(n)[:m]
    sv = StateVector.from_amplitudes(psi, backend=backend)
    got, ties = sv.sample(qubits, np.arange(m), shots, 7 + n)
    want, _ = O.run_shots(measure(qubits), n, shots, 7 + n, init=psi)
    assert ties == 0 and (got == want).all()


def test_ties_within_a_wide_margin(backend):
    """|u - p| < tie_eps is counted over every draw, however far from the float32 margin."""
    n, shots = 6, 2000
    psi = np.full(1 << n, 2.0 ** (-n / 2), dtype=complex)
    sv = StateVector.from_amplitudes(psi, backend=backend)
    for eps in (0.0, 1e-7, 1e-3, 0.25, 2.0):
        got, ties = sv.sample(range(n), range(n), shots, 11, tie_eps=eps)
        draws = np.zeros(shots * n)
        x = O.Rng(11)
        for i in range(draws.size):
            draws[i] = x.next_f64()
        assert ties == int((np.abs(draws - 0.5) < eps).sum())
        assert (got == ((draws.reshape(shots, n) < 0.5) << np.arange(n)).sum(1)).all()
