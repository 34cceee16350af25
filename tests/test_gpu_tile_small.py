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


@pytest.mark.parametrize("nq", [4, 5, 8, 11, 13, 15])
def test_index_maps_move_doubles_exactly(nq):
    """CNOT, X and SWAP alone, one pass or several: every bit of a double arrives, also
    of what double-float cannot hold."""
    rng = np.random.default_rng(nq)
    ops = []
    for _ in range(50 if nq < 13 else 80):
        name = str(rng.choice(["CNOT", "PauliX", "SWAP"]))
        ops.append((name, [int(w) for w in rng.choice(nq, 1 if name == "PauliX" else 2, replace=False)], False, []))
    psi = rand_state(nq, rng)
    psi[: 4] = [1e-200 + 3e-310j, -1e200j, complex(np.inf, 0.1), complex(np.nan, -0.0)]
    ref = psi.copy()
    for name, w, _, _ in ops: # by index, so that no arithmetic meets inf and nan
        i = np.arange(1 << nq)
        bit = [i >> (nq - 1 - x) & 1 for x in w]
        if name == "PauliX":
            src = i ^ (1 << (nq - 1 - w[0]))
        elif name == "CNOT":
            src = i ^ (bit[0] << (nq - 1 - w[1]))
        else:
            d = bit[0] ^ bit[1]
            src = i ^ (d << (nq - 1 - w[0])) ^ (d << (nq - 1 - w[1]))
        ref = ref[src]
    s = State.from_array(psi, N.PLK_C128)
    arr, keep = make_ops(ops)
    N.check(N.lib.plk_apply_ops(s.h, arr, len(ops)))
    got = s.get()
    s.close()
    del keep
    np.testing.assert_array_equal(got.view(np.uint64), ref.view(np.uint64))
