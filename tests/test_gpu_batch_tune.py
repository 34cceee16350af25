"""GPU: tuning a batch.  Tile programs have no launch configuration: the report says
so, the settings stay as the caller set them and results do not change.  A
batch with a dense matrix runs on the engine, whose configurations are timed.
"""
import numpy as np
import pytest

from test_gpu_batch import check_against_oracle, make_cases

pytestmark = pytest.mark.gpu


def matrix_circuit(nq, seed):
    """(as added, for the oracle): a circuit with a named gate given as a matrix"""
    from pennylane_lightning_kokkos import _native as N
    import ctypes as C

    m = np.zeros(16, dtype=np.complex128)
    N.check(N.lib.plk_gate_matrix(N.GATE_ID["SWAP"], None, 0, 0, 2, m.ctypes.data_as(C.POINTER(C.c_double))))
    (nq, ops, words, tp), = make_cases("with a matrix", [nq], 40, seed)
    at = len(ops) // 2
    mine = ops[:at] + [("Matrix", [1, nq - 1], False, [], m.reshape(4, 4))] + ops[at:]
    theirs = ops[:at] + [("SWAP", [1, nq - 1], False, [])] + ops[at:]
    return (nq, mine, words, tp), (nq, theirs, words, tp)


def test_tiles_have_nothing_to_tune():
    from pennylane_lightning_kokkos.batch import CircuitBatch

    cases = make_cases("untuned", [8, 12, 14, 9], 50)
    for compiled in (False, True):
        b = CircuitBatch("c64")
        for c in cases:
            b.add(*c)
        b.set_config(cluster=2, smem_qubits=11, cluster_min_qubits=15)
        want = b.get_config()
        first = b.run() if compiled else None
        report = b.tune(reps=2)
        assert "nothing to tune" in report and len(report.strip().splitlines()) == 1
        assert b.get_config() == want
        again = b.run()
        if compiled:
            np.testing.assert_array_equal(first[0], again[0])
            np.testing.assert_array_equal(first[1], again[1])
        check_against_oracle(cases, again[0], b.gradients(again[1]), 1e-4)
        b.close()


@pytest.mark.parametrize("dtype,tol", [("c64", 1e-4), ("c128", 1e-10)])
def test_engine_is_tuned(dtype, tol):
    from pennylane_lightning_kokkos.batch import CircuitBatch

    cases = make_cases("tuned", [8, 14, 15, 9], 50)
    mine, theirs = matrix_circuit(13, 3)
    b = CircuitBatch(dtype)
    for c in cases + [mine]:
        b.add(*c)
    lines = b.tune(reps=1).strip().splitlines()
    assert len(lines) > 3 and all("ctas_per_sm" in x for x in lines)
    assert any(x.startswith("ctas_per_sm=2") for x in lines) == (dtype == "c64")
    ev, jac = b.run()
    check_against_oracle(cases + [theirs], ev, b.gradients(jac), tol)
    b.close()
