"""GPU: more tiles than the chip holds CTAs, so that a CTA walks several and uses
its shared tile and its sums again, and batches whose circuits' states take turns.

Pauli sums: 21 qubits are 512 tiles against at most 456 CTAs; tolerances as
test_gpu_pauli_tile.py, 1e-12 (complex128) and 2e-6 (complex64) of the sum of
|coefficients|.  Op lists: 22 qubits are 1024 (complex128) and 2048 tiles against
304 and 1216 CTAs; states 1e-12 and, for 60 ops, sqrt(60) 2^-24 of the largest amplitude's
neighbourhood, 5e-7, doubled.  Jacobians: the CTAs are shared by the observables, 20 of
them leave 15 to 30 for 32 tiles; complex128 1e-10, complex64 1e-5 (two states, each
within sqrt(120) 2^-24 of unit norm after 120 ops, doubled, and sums of 32 products).
"""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from abi import State, make_ops
from pennylane_lightning_kokkos import _native as N
from test_gpu_adjoint import gpu_adjoint
from test_gpu_batch import oracle_ref
from test_gpu_dynamic_range import mode, wide_state  # noqa: F401
from test_gpu_pauli_modes import applied, packed
from test_oracle_golden import rand_state
from test_tile_program_cpu import random_ops

pytestmark = pytest.mark.gpu

TOL = {N.PLK_C64: 2e-6, N.PLK_C128: 1e-12}


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
@pytest.mark.parametrize("weights", [(1, 2), (1, 2, 9)]) # all on tiles; the wide ones in plain passes
def test_pauli_sum(weights, dtype):
    nq, rng = 21, np.random.default_rng(len(weights))
    psi = rand_state(nq, rng)
    words = []
    for k in range(30):
        w = weights[k % len(weights)]
        words.append((float(rng.standard_normal()), [int(x) for x in rng.choice(nq, w, replace=False)],
                      "".join(str(x) for x in rng.choice(list("XYZ"), w))))
    s, o, v = State.from_array(psi, dtype), State(nq, dtype), C.c_double()
    have = s.get().astype(np.complex128)
    ref = applied(have, nq, words)
    keep, args = packed(words)
    tol = TOL[dtype] * float(np.sum(np.abs(keep[0])))
    N.check(N.lib.plk_apply_pauli_sum(o.h, s.h, *args))
    np.testing.assert_allclose(o.get(), ref, atol=tol, rtol=0)
    N.check(N.lib.plk_expval_pauli_sum(s.h, *args, C.byref(v)))
    assert abs(v.value - float(np.vdot(have, ref).real)) < tol
    s.close()
    o.close()


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
def test_op_list(dtype):
    nq, rng = 22, np.random.default_rng(22)
    ops = random_ops(nq, 60, rng)
    psi = rand_state(nq, rng)
    s = State.from_array(psi, dtype)
    arr, keep = make_ops(ops)
    N.check(N.lib.plk_apply_ops(s.h, arr, len(ops)))
    np.testing.assert_allclose(s.get(), O.run_ops(psi.copy(), ops), atol=1e-12 if dtype == N.PLK_C128 else 1e-6, rtol=0)
    s.close()
    del keep


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
def test_jacobian_of_many_observables(dtype):
    nq, rng = 16, np.random.default_rng(16)
    ops = random_ops(nq, 120, rng, single_param=True)
    psi = rand_state(nq, rng)
    obs = [("named", ("PauliX", "PauliY", "PauliZ")[k % 3], [k % nq]) for k in range(20)]
    trainable = list(range(0, sum(1 for o in ops if o[3]), 3))
    np.testing.assert_allclose(gpu_adjoint(psi, obs, ops, trainable, dtype), O.adjoint_jacobian(psi, obs, ops, trainable),
                               atol=1e-10 if dtype == N.PLK_C128 else 1e-5, rtol=0)


def test_jacobian_on_wide_state(mode): # noqa: F811
    """Amplitudes of thirty decades, complex128 in both arithmetic modes."""
    nq, rng = 13, np.random.default_rng(13)
    ops = random_ops(nq, 100, rng, single_param=True)
    psi = wide_state(nq, rng)
    obs = [("named", "PauliX", [1]), ("named", "PauliZ", [0]), ("named", "PauliY", [nq - 1])]
    trainable = list(range(0, sum(1 for o in ops if o[3]), 2))
    ref = O.adjoint_jacobian(psi, obs, ops, trainable)
    for k in (1, 3):
        np.testing.assert_allclose(gpu_adjoint(psi, obs[:k], ops, trainable, N.PLK_C128), ref[:k], atol=1e-10, rtol=0)


def test_batch_in_waves():
    """Three circuits of 29 qubits have 8 GiB of states each, two of them at a time; the
    ops are on five wires, so that a five-qubit circuit has the same results."""
    from pennylane_lightning_kokkos.batch import CircuitBatch

    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GiB of device memory")
    nq, at = 29, [0, 3, 14, 27, 28]
    b, want = CircuitBatch("c64"), []
    for k, n in enumerate([nq, 7, nq, nq, 12]):
        rng = np.random.default_rng(k)
        ops = [o for o in random_ops(5, 40, rng, single_param=True) if o[0] != "Identity"]
        words = [(0.7, [0, 2], "XY"), (-0.4, [4], "Z"), (0.3, [1, 3], "ZX")]
        wires = at if n == nq else [0, 1, 3, 4, 6]
        tp = list(range(sum(1 for o in ops if o[3])))
        b.add(n, [(g, [wires[w] for w in ws], inv, p) for g, ws, inv, p in ops],
              [(c, [wires[w] for w in ws], l) for c, ws, l in words], tp)
        want.append(oracle_ref(5, ops, words, tp))
    for _ in range(2):
        ev, jac = b.run()
        for (e, g), e2, g2 in zip(want, ev, b.gradients(jac)):
            assert abs(e - e2) < 1e-5
            np.testing.assert_allclose(g2, g, atol=1e-5, rtol=0)
    b.close()
