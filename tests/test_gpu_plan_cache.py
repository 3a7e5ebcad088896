"""Plans that one call leaves behind for the next: a noisy circuit of many unitary
parts must not push out the searched plans of other circuits."""
import ctypes as C
import time

import numpy as np
import pytest

from quantumforge_gb300 import Circuit, Gate, NoiseChannel, _native
from quantumforge_gb300 import _abi as A
from quantumforge_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def planned(lib, ops, n):
    npass, ngate = C.c_uint64(), C.c_uint64()
    t = time.perf_counter()
    st = lib.qf_plan_stats(n, A.C64, _native.ptr(ops), len(ops), None, 0, None, 0, None, C.byref(npass), C.byref(ngate))
    assert st == 0
    return time.perf_counter() - t


def test_noisy_parts_leave_searched_plans_alone(backend, engine_lib):
    rng = np.random.default_rng(1)
    c = Circuit()
    for i in range(200):  # parts of different structure
        for _ in range(1 + i % 7):
            a, b = rng.permutation(5)[:2]
            (c.cnot, c.cz, c.swap)[int(rng.integers(0, 3))](int(a), int(b))
            c.push(Gate.Ry(0.1 + i), int(a))
        for q in range(5):
            c.channel(q, NoiseChannel.AmplitudeDamping(0.01))
    c.measure(0, 0)
    ops = W.random_circuit(30, 40, 77, two_qubit="mixed")
    searched = planned(engine_lib, ops, 30)  # hundreds of times a replay
    assert planned(engine_lib, ops, 30) < 0.1 * searched
    c.run_shots_packed(5, 10, 1, backend=backend, noise=True)
    assert planned(engine_lib, ops, 30) < 0.1 * searched
