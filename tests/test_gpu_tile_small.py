"""GPU: tiles of fewer threads than a warp, where several lanes hold the same
amplitudes: lists of many rounds give the oracle's state and Jacobian (tolerances
as test_gpu_tile.py), and the same bits every time.
"""
import numpy as np
import pytest

import oracle as O
from abi import State, make_ops
from pennylane_lightning_kokkos import _native as N
from test_gpu_adjoint import gpu_adjoint
from test_oracle_golden import rand_state
from test_tile_program_cpu import random_ops

pytestmark = pytest.mark.gpu

STOL = {N.PLK_C64: 5e-6, N.PLK_C128: 1e-12}
JTOL = {N.PLK_C64: 1e-4, N.PLK_C128: 1e-10}


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
@pytest.mark.parametrize("nq", [4, 5, 6, 7, 8, 9])
def test_reruns(nq, dtype):
    rng = np.random.default_rng(40 + nq)
    ops = random_ops(nq, 150, rng, single_param=True)
    psi = rand_state(nq, rng)
    arr, keep = make_ops(ops)
    first = None
    for _ in range(20):
        s = State.from_array(psi, dtype)
        N.check(N.lib.plk_apply_ops(s.h, arr, len(ops)))
        got = s.get()
        s.close()
        first = got if first is None else first
        np.testing.assert_array_equal(got, first)
    np.testing.assert_allclose(first, O.run_ops(psi.copy(), ops), atol=STOL[dtype], rtol=0)
    del keep
    trainable = list(range(0, sum(1 for o in ops if o[3]), 2))
    obs = [("named", "PauliX", [1]), ("named", "PauliZ", [0])]
    jac = gpu_adjoint(psi, obs, ops, trainable, dtype)
    np.testing.assert_allclose(jac, O.adjoint_jacobian(psi, obs, ops, trainable), atol=JTOL[dtype], rtol=0)
    for _ in range(5):
        np.testing.assert_array_equal(gpu_adjoint(psi, obs, ops, trainable, dtype), jac)
