"""Recorded plans and the engines they are for: small complex128 states have one
tile on either engine, but register-tile passes merge every product of one-qubit
gates and the in-order ones only some, so a pass of either holds other gates."""
import ctypes as C

import numpy as np
import pytest

from quantumforge_gb300 import _abi as A
from quantumforge_gb300 import _native


def passes(lib, n, ops, params, flags):
    npass, ngate = C.c_uint64(), C.c_uint64()
    o = A.ExecOpts(A.EXEC_AUTO, 0, 0, flags)
    st = lib.qf_plan_stats(n, A.C128, _native.ptr(ops), len(ops), _native.ptr(params), params.size, None, 0, C.byref(o),
                           C.byref(npass), C.byref(ngate))
    assert st == 0
    return npass.value


@pytest.mark.parametrize("n", [1, 2, 3])
def test_engines_do_not_share_plans(engine_lib, n):
    for length, order in ((1600, (0, A.EXEC_FLAG_SMEM_TILES)), (1800, (A.EXEC_FLAG_SMEM_TILES, 0))):
        ops = np.zeros(length, dtype=A.OP_DTYPE)
        ops["kind"] = A.OP_ROTATION
        ops["gate"] = np.where(np.arange(length) // n % 2, A.PAULI_X, A.PAULI_Z)
        ops["q0"] = np.arange(length) % n
        ops["param"] = np.arange(length)
        params = np.linspace(0.1, 3.0, length)
        got = {f: passes(engine_lib, n, ops, params, f) for f in order}
        assert got[0] == 1                             # one product per qubit
        assert got[A.EXEC_FLAG_SMEM_TILES] == -(-length // 768)  # gate by gate, 768 of them in a pass
