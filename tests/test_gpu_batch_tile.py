"""GPU: complex64 batches on tiles (csrc/batch_tile.cu) against the oracle at the
sizes where tiles and CTAs change, with circuits that have no ops, no
trainable parameter or no Hamiltonian term, and over repeated runs with other
parameters.  Tolerance 1e-4 as the other complex64 batch tests; a rerun of the
same parameters gives the same bits.
"""
import numpy as np
import pytest

from test_gpu_batch import check_against_oracle, make_cases, oracle_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[4, 5, 8], [9, 10, 11], [12, 13, 15], [4, 16, 7, 11, 12, 8]])
def test_sizes_and_reruns(sizes):
    from pennylane_lightning_kokkos.batch import CircuitBatch

    cases = make_cases("tile", sizes, 70)
    b = CircuitBatch("c64")
    for nq, ops, words, tp in cases:
        b.add(nq, ops, words, tp)
    ev, jac = b.run()
    check_against_oracle(cases, ev, b.gradients(jac), 1e-4)
    rng = np.random.default_rng(len(sizes))
    other = rng.uniform(-np.pi, np.pi, b.info()[1])
    # special angles: runs that multiply to diagonals, flips and the identity
    other[: len(other) // 2] = rng.choice([0.0, np.pi, -np.pi, np.pi / 2, 2 * np.pi], len(other) // 2)
    ev2, jac2 = b.run(other)
    changed, k = [], 0
    for nq, ops, words, tp in cases:
        new = []
        for name, wires, inv, prm in ops:
            new.append((name, wires, inv, [float(x) for x in other[k:k + len(prm)]]))
            k += len(prm)
        changed.append((nq, new, words, tp))
    check_against_oracle(changed, ev2, b.gradients(jac2), 1e-4)
    ev3, jac3 = b.run(np.concatenate([[x for o in ops for x in o[3]] for _, ops, _, _ in cases]))
    np.testing.assert_array_equal(ev3, ev)
    np.testing.assert_array_equal(jac3, jac)
    b.close()


def test_empty_pieces():
    from pennylane_lightning_kokkos.batch import CircuitBatch

    b = CircuitBatch("c64")
    b.add(6, [], [(0.5, [1], "Z"), (0.25, [0], "X")])
    b.add(5, [("RY", [0], False, [0.3]), ("CNOT", [0, 1], False, [])], [(1.0, [1], "Z")], [])
    b.add(12, [("RX", [3], False, [0.7])], [])
    ev, jac = b.run()
    np.testing.assert_allclose(ev, [0.5, np.cos(0.3), 0.0], atol=1e-6)
    np.testing.assert_allclose(jac, [0.0], atol=1e-7)
    b.close()
