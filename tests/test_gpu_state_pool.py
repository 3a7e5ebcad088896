"""Memory of destroyed states taken up by new ones: every new state is |0...0>
whatever its memory held, sizes above and below what is kept, states whose
address was given out, threads with contexts of their own, and shots from a
qubit count against shots from the amplitudes of |0...0>. Exact results."""
import threading

import numpy as np
import pytest

from quantumforge_gb300 import Circuit, CudaBackend, DensityMatrix, NoiseChannel, StateVector
from quantumforge_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def use(backend, n, dtype):
    sv = StateVector.zero(n, dtype=dtype, backend=backend)
    a = sv.amplitudes()
    assert a[0] == 1 and np.count_nonzero(a) == 1
    sv.apply_ops(W.random_circuit(n, 2, n))
    return sv


@pytest.mark.parametrize("dtype", ["c64", "c128"])
def test_new_states_are_zero_states(backend, dtype):
    for n in (1, 2, 3, 10, 1, 3, 17, 10, 24, 25, 17, 24):
        use(backend, n, dtype)
    held = [use(backend, n, dtype) for n in (5, 5, 5)]
    first = [h.amplitudes() for h in held]
    use(backend, 5, dtype)
    assert all((h.amplitudes() == f).all() for h, f in zip(held, first))
    rho = DensityMatrix.zero(3, dtype=dtype, backend=backend)
    rho.apply_channel(NoiseChannel.Depolarizing(0.1), 1)
    del rho
    assert DensityMatrix.zero(3, dtype=dtype, backend=backend).entries()[0, 0] == 1


def test_threads_with_contexts_of_their_own():
    errors = []

    def work(seed):
        try:
            be = CudaBackend()
            for i in range(30):
                use(be, 4 + (seed + i) % 9, "c128")
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


@pytest.mark.parametrize("n", [1, 6, 12])
@pytest.mark.parametrize("noise", [False, True])
def test_shots_from_a_qubit_count(backend, n, noise):
    c = Circuit.from_ops(W.random_circuit(n, 3, 5))
    if noise:
        c.channel(0, NoiseChannel.AmplitudeDamping(0.2))
    for q in range(n):
        c.measure(q, q)
    zero = np.zeros(1 << n, dtype=complex)
    zero[0] = 1
    a = c.run_shots_packed(n, 500, 3, backend=backend, noise=noise)
    b = c.run_shots_packed(zero, 500, 3, backend=backend, noise=noise)
    assert (a[0] == b[0]).all() and a[1:] == b[1:]
