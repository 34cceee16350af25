"""GPU: tile sweeps (op lists and adjoint Jacobians without dense matrices)
against the oracle, at the sizes where tiles change: fewer amplitudes than a
warp holds, one tile, one tile and a bit, several.

Tolerances: complex128 states 1e-12 and Jacobians 1e-10 (double-float, about
2^-45 per op); complex64 states 5e-6 and Jacobians 1e-4 (200 ops of 2^-24 in
random walk, doubled), as the other op-list tests.
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
@pytest.mark.parametrize("nq", [4, 5, 8, 9, 10, 11, 12, 13, 14, 16])
def test_forward_and_backward(nq, dtype):
    rng = np.random.default_rng(700 + nq)
    ops = random_ops(nq, 200, rng)
    psi = rand_state(nq, rng)
    s = State.from_array(psi, dtype)
    arr, keep = make_ops(ops)
    N.check(N.lib.plk_apply_ops(s.h, arr, len(ops)))
    np.testing.assert_allclose(s.get(), O.run_ops(psi.copy(), ops), atol=STOL[dtype], rtol=0)
    s.close()
    del keep
    ops = random_ops(nq, 120, rng, single_param=True)
    npar = sum(1 for o in ops if o[3])
    trainable = sorted(int(x) for x in rng.choice(npar, npar * 3 // 4, replace=False))
    obs = [("named", "PauliX", [1]), ("named", "PauliZ", [nq - 1]), ("named", "PauliY", [0])]
    ref = O.adjoint_jacobian(psi, obs, ops, trainable)
    for k in (1, 3): # one sweep, several in the same launches
        np.testing.assert_allclose(gpu_adjoint(psi, obs[:k], ops, trainable, dtype), ref[:k], atol=JTOL[dtype], rtol=0)


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
def test_index_maps_only(dtype):
    """CNOTs, X and SWAP move amplitudes and change none."""
    nq = 15
    rng = np.random.default_rng(3)
    ops = []
    for _ in range(60):
        name = str(rng.choice(["CNOT", "PauliX", "SWAP"]))
        ops.append((name, [int(w) for w in rng.choice(nq, 1 if name == "PauliX" else 2, replace=False)], False, []))
    psi = rand_state(nq, rng)
    s = State.from_array(psi, dtype)
    start = s.get()
    arr, keep = make_ops(ops)
    N.check(N.lib.plk_apply_ops(s.h, arr, len(ops)))
    got = s.get()
    s.close()
    ref = O.run_ops(start.astype(np.complex128), ops)
    if dtype == N.PLK_C64:
        np.testing.assert_array_equal(got, ref.astype(np.complex64))
    else: # 48 of a double's 53 bits pass through the sweep
        np.testing.assert_allclose(got, ref, rtol=2.0 ** -46, atol=0)
    del keep


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
@pytest.mark.parametrize("nq", [4, 8, 11, 12, 14])
def test_jacobian_of_pauli_words(nq, dtype):
    """Sweeps that read H lambda off lambda: words with every letter, none, and
    more than one launch holds (32)."""
    import ctypes as C

    from abi import f64, i64

    rng = np.random.default_rng(900 + nq)
    ops = random_ops(nq, 60, rng, single_param=True)
    npar = sum(1 for o in ops if o[3])
    trainable = sorted(int(x) for x in rng.choice(npar, npar // 2 + 1, replace=False))
    words = [(1.0, [w], "Z") for w in range(nq)] + [(0.7, [], "")]
    while len(words) < (35 if nq == 8 else nq + 6):
        k = int(rng.integers(1, nq + 1))
        words.append((float(rng.standard_normal()), [int(w) for w in rng.choice(nq, k, replace=False)],
                      "".join(str(x) for x in rng.choice(list("XYZI"), k))))
    name = {"X": "PauliX", "Y": "PauliY", "Z": "PauliZ", "I": "Identity"}
    obs = [("hamiltonian", [c], [("tensor", [("named", name[l], [w]) for w, l in zip(ws, ls)] or
                                  [("named", "Identity", [0])])]) for c, ws, ls in words]
    psi = rand_state(nq, rng)
    ref = O.adjoint_jacobian(psi, obs, ops, trainable)
    s = State.from_array(psi, dtype)
    before = s.get()
    arr, keep = make_ops(ops)
    c, cp = f64([w[0] for w in words])
    off, offp = i64(np.cumsum([0] + [len(w[1]) for w in words]))
    wi, wp = i64([x for w in words for x in w[1]])
    tp, tpp = i64(trainable)
    jac = np.zeros((len(words), len(trainable)))
    N.check(N.lib.plk_adjoint_jacobian_pauli(s.h, len(words), cp, offp, wp, "".join(w[2] for w in words).encode(), arr,
                                             len(ops), tpp, len(tp), jac.ctypes.data_as(C.POINTER(C.c_double))))
    np.testing.assert_allclose(jac, ref, atol=JTOL[dtype], rtol=0)
    np.testing.assert_array_equal(s.get(), before)
    s.close()
    del keep
