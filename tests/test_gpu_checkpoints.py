"""Checkpoints that take over the state's memory: gradients with segments of
every length (one gate, uneven, longer than the list, empty ones behind it)
against the CPU oracle, with compiled passes (which read the checkpoint) and
the others (which copy it), twice in a row over the kept states, and a circuit
without a checkpoint in between.

Tolerance: an operation rounds each component at most twice, so after m
operations an amplitude of a normalised state is off by at most 2 sqrt(2) u m;
psi and lambda = H psi each carry that, |H| at most the sum of its coefficients."""
import math

import numpy as np
import pytest

import oracle as O
from quantumforge_gb300 import ParameterizedCircuit, PauliSum
from quantumforge_gb300 import workloads as W
from quantumforge_gb300.gradients import GradientOptions, GradientStrategy, gradient_with_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n,opts", [("c64", 13, {"jit": True}), ("c64", 12, {"jit": True}), ("c64", 13, {"jit": False}),
                                          ("c64", 9, {}), ("c128", 10, {}), ("c64", 13, {"smem_tiles": True})])
@pytest.mark.parametrize("every", [1, 17, 40, 1000])
def test_gradients_with_checkpoints(backend, dtype, n, opts, every):
    layers = 1 if every == 1 else 2
    ops, params = W.hea_vqe(n, layers, 3 + n)
    H = PauliSum.tfim_ring(n)
    pc = ParameterizedCircuit.from_ops(ops, params.size)
    e, g = O.adjoint_uncompute(ops, n, params, H.array())
    u = 2.0**-24 if dtype == "c64" else 2.0**-53
    tol = 4.0 * 2.0 * math.sqrt(2.0) * u * (2 * len(ops) + 8) * sum(abs(c) for _, _, c in H.terms)

    def grad(every):
        return gradient_with_inputs(pc, GradientOptions(strategy=GradientStrategy.Adjoint), [], params, n, H, dtype=dtype,
                                    checkpoint_every=every, exec_opts=opts, backend=backend)

    first = grad(every)
    for est in (first, grad(0), grad(every)):
        assert abs(est.expectation - e) <= tol and np.abs(est.gradient - g).max() <= tol
    again = grad(every)
    assert again.expectation == first.expectation and (again.gradient == first.gradient).all()
