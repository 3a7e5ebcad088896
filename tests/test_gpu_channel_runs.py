"""Runs of channels on complex128 density matrices against the CPU oracle's one
channel at a time: every tile width and register split, runs that need one to
four passes, qubits with several channels, and the strengths at which a row of
a channel's map is zero, the identity, or led by the other population.

Tolerance: entries of a density matrix are at most 1 in modulus; a channel
rounds an entry at most four times in the oracle and four times here (two in its
composition, one shear, one factor), the factors at most twice per qubit."""
import numpy as np
import pytest

import oracle as O
from quantumforge_gb300 import Circuit, DensityMatrix, NoiseChannel

pytestmark = pytest.mark.gpu

KINDS = (NoiseChannel.AmplitudeDamping, NoiseChannel.Depolarizing, NoiseChannel.PhaseDamping,
         lambda p: NoiseChannel.ThermalDamping(p, 0.1))


@pytest.mark.parametrize("n,which", [(1, "all"), (2, "all"), (3, "all"), (4, "all"), (5, "high"), (6, "all"), (7, "all"), (7, "ends"),
                                     (8, "all"), (9, "high"), (9, "all"), (10, "ends"), (10, "all"), (10, "high"), (11, "six")])
def test_runs_match_the_oracle(backend, n, which):
    rng = np.random.default_rng(100 * n + len(which))
    qubits = {"all": range(n), "high": range(n // 2, n), "ends": (0, n - 1), "six": range(2, 8)}[which]
    a = rng.normal(size=(2**n, 2, 2)) @ np.array([1.0, 1j])
    rho = a @ a.conj().T
    rho /= np.trace(rho).real
    c, count = Circuit(), 0
    for repeat in range(2):
        for q in rng.permutation(list(qubits)):
            if repeat == 0 or rng.uniform() < 0.5:
                p = float(rng.choice([rng.uniform(0.0, 0.9), 0.0, 1.0], p=[0.8, 0.1, 0.1]))
                c.channel(int(q), KINDS[int(rng.integers(0, 4))](p))
                count += 1
    d = DensityMatrix.from_entries(rho, backend=backend)
    c.run_density(d)
    want = O.run_density(c.ops(), n, rho=rho)
    assert np.abs(d.entries() - want).max() <= 2.0**-53 * (8 * count + 2 * n + 4)
