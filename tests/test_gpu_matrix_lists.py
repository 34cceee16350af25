"""GPU: op lists, Jacobians and complex64 batches with a dense matrix in them, which
keep the register windows and the batch engine: without one they run on tiles.

A SWAP is given as its matrix, so that the oracle's named gate is the reference.
Tolerances as test_gpu_windows.py and test_gpu_batch.py: states 1e-12 (complex128)
and 5e-6 (complex64), Jacobians 1e-10 and 1e-4, batches 1e-4.
"""
import numpy as np
import pytest

import oracle as O
from abi import State, make_ops
from pennylane_lightning_kokkos import _native as N
from test_gpu_adjoint import gpu_adjoint, random_circuit
from test_gpu_batch import check_against_oracle, make_cases, run_batch
from test_gpu_batch_tune import matrix_circuit
from test_gpu_windows import diagonal_heavy_circuit, window_switch  # noqa: F401

pytestmark = pytest.mark.gpu

STOL = {N.PLK_C64: 5e-6, N.PLK_C128: 1e-12}
JTOL = {N.PLK_C64: 1e-4, N.PLK_C128: 1e-10}
SWAP = np.eye(4, dtype=np.complex128)[[0, 2, 1, 3]]


def with_matrices(ops, nq, rng, count=3):
    """(for the library, for the oracle): the list with SWAPs, as matrices and by name"""
    mine, theirs = list(ops), list(ops)
    for _ in range(count):
        at, w = int(rng.integers(len(mine) + 1)), [int(x) for x in rng.choice(nq, 2, replace=False)]
        mine.insert(at, ("Matrix", w, False, [], SWAP))
        theirs.insert(at, ("SWAP", w, False, []))
    return mine, theirs


def observables(nobs, nq):
    return [("named", "PauliZ", [o % nq]) for o in range(nobs - 1)] + [
        ("hamiltonian", [0.5, -1.2], [("named", "PauliX", [2]),
                                      ("tensor", [("named", "PauliY", [0]), ("named", "PauliZ", [nq - 1])])])]


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
@pytest.mark.parametrize("nobs", [1, 2, 5])
@pytest.mark.parametrize("nq", [7, 10])
def test_windows_backward(nq, nobs, dtype, window_switch): # noqa: F811
    rng = np.random.default_rng(600 + 10 * nq + nobs)
    mine, theirs = with_matrices(random_circuit(nq, 90, rng), nq, rng)
    npar = sum(1 for o in mine if o[3])
    trainable = sorted(int(x) for x in rng.choice(npar, npar * 3 // 4, replace=False))
    obs = observables(nobs, nq)
    psi = O.run_ops(O.zero_state(nq), theirs)
    ref = O.adjoint_jacobian(psi, obs, theirs, trainable)
    window_switch(True)
    jac = gpu_adjoint(psi, obs, mine, trainable, dtype)
    np.testing.assert_allclose(jac, ref, atol=JTOL[dtype], rtol=0)
    np.testing.assert_array_equal(gpu_adjoint(psi, obs, mine, trainable, dtype), jac)


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
@pytest.mark.parametrize("nq", [7, 10, 13])
def test_windows_diagonal_runs(nq, dtype, window_switch): # noqa: F811
    rng = np.random.default_rng(800 + nq)
    mine, theirs = with_matrices(diagonal_heavy_circuit(nq, 3, rng), nq, rng)
    window_switch(True)
    s = State(nq, dtype)
    arr, keep = make_ops(mine)
    N.check(N.lib.plk_apply_ops(s.h, arr, len(mine)))
    psi = O.run_ops(O.zero_state(nq), theirs)
    np.testing.assert_allclose(s.get(), psi, atol=STOL[dtype], rtol=0)
    s.close()
    del keep
    trainable = list(range(0, sum(1 for o in mine if o[3]), 2))
    for nobs in (1, 3):
        obs = observables(nobs, nq)
        np.testing.assert_allclose(gpu_adjoint(psi, obs, mine, trainable, dtype),
                                   O.adjoint_jacobian(psi, obs, theirs, trainable), atol=JTOL[dtype], rtol=0)


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
def test_windows_one_observable_after_another(dtype, window_switch): # noqa: F811
    """Above 22 qubits the observables' sweeps run in turn, not on streams of their own;
    the reference is the op-at-a-time path on the same states."""
    nq, rng = 23, np.random.default_rng(23)
    ops = [o for w in range(5) for o in (("RY", [w], False, [0.3 + w]), ("RZ", [w], False, [0.2 * w]))] * 2
    ops += [("CNOT", [0, 1], False, []), ("CRX", [3, 2], False, [0.7])]
    mine, _ = with_matrices(ops, 5, rng, 1)
    psi = np.zeros(1 << nq, dtype=np.complex128)
    psi[: 1 << nq: 1 << 18] = O.run_ops(O.zero_state(5), ops)
    obs = [("named", "PauliZ", [0]), ("named", "PauliX", [1]), ("named", "PauliY", [2])]
    trainable = list(range(sum(1 for o in mine if o[3])))
    window_switch(True)
    jac = gpu_adjoint(psi, obs, mine, trainable, dtype)
    window_switch(False)
    np.testing.assert_allclose(jac, gpu_adjoint(psi, obs, mine, trainable, dtype), atol=JTOL[dtype], rtol=0)


@pytest.mark.parametrize("config", [
    dict(cluster=1, ctas_per_sm=2),
    dict(cluster=4, ctas_per_sm=2, cluster_min_qubits=13),
    dict(cluster=4, smem_qubits=13, cluster_min_qubits=14),
    dict(cluster=2, smem_qubits=11, cluster_min_qubits=12),
    dict(cluster=8, smem_qubits=12, cluster_min_qubits=15),
    dict(cluster=1, smem_qubits=4, cluster_min_qubits=30),
])
def test_engine_configurations_c64(config):
    cases = make_cases("engine", [4, 9, 11, 12, 13, 14, 15, 16], 50)
    mine, theirs = matrix_circuit(14, 9)
    ev, grads = run_batch(cases + [mine], "c64", config)
    check_against_oracle(cases + [theirs], ev, grads, 1e-4)
