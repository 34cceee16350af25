"""GPU: long chains of rotations that no phase interrupts, forward and backward.

complex128 sweeps defer the rotations' cosines to phase tables; sums over the
two states are formed from what the sweep holds, so a chain without a table
would leave single precision's range (its products stood 2^128 above the
state's).  Tolerances as the other tile tests: complex128 states 1e-12 and Jacobians
1e-10, complex64 5e-6 and 1e-4.
"""
import numpy as np
import pytest

import oracle as O
from abi import State, make_ops
from pennylane_lightning_kokkos import _native as N
from test_gpu_adjoint import gpu_adjoint
from test_oracle_golden import rand_state
from test_tile_growth_cpu import chains

pytestmark = pytest.mark.gpu

STOL = {N.PLK_C64: 5e-6, N.PLK_C128: 1e-12}
JTOL = {N.PLK_C64: 1e-4, N.PLK_C128: 1e-10}


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
@pytest.mark.parametrize("kind,nq", [("one wire", 12), ("two wires", 5), ("two wires", 13), ("four wires", 12)])
def test_chains(kind, nq, dtype):
    rng = np.random.default_rng(nq)
    ops = chains(nq, kind, 100)
    psi = rand_state(nq, rng)
    s = State.from_array(psi, dtype)
    arr, keep = make_ops(ops)
    N.check(N.lib.plk_apply_ops(s.h, arr, len(ops)))
    np.testing.assert_allclose(s.get(), O.run_ops(psi.copy(), ops), atol=STOL[dtype], rtol=0)
    s.close()
    del keep
    trainable = list(range(0, len(ops), 16)) # few sums, so that they do not end the passes early
    obs = [("named", "PauliX", [1]), ("named", "PauliZ", [0])]
    ref = O.adjoint_jacobian(psi, obs, ops, trainable)
    for k in (1, 2):
        np.testing.assert_allclose(gpu_adjoint(psi, obs[:k], ops, trainable, dtype), ref[:k], atol=JTOL[dtype], rtol=0)
