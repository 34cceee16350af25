"""Long lists of gates that commute on a wire compile in time linear in their length
(csrc/tile_program.hpp): 40000 gates in well under two seconds, where a dependency
for each pair of them took six.
"""
import ctypes as C
import time

import numpy as np
import pytest

from abi import make_ops
from test_tile_growth_cpu import growth  # noqa: F401

N = 40000


@pytest.mark.parametrize("kind", ["controls, then targets", "phases on all pairs"])
def test_linear_time(growth, kind): # noqa: F811
    nq, rng = 20, np.random.default_rng(1)
    if kind == "phases on all pairs":
        ops = [("CZ", [int(w) for w in rng.choice(nq, 2, replace=False)], False, []) for _ in range(N)]
    else: # half of them wait for the other half
        ops = [("CRZ", [0, 1 + i % (nq - 1)], False, [0.1]) for i in range(N // 2)]
        ops += [("CNOT", [1 + i % (nq - 1), 0], False, []) for i in range(N // 2)]
    arr, keep = make_ops(ops)
    slots, left = np.full(N, -1, dtype=np.int64), C.c_double()
    t = time.perf_counter()
    assert growth(nq, 12, 4, 2, 0, arr, N, slots.ctypes.data_as(C.c_void_p), C.byref(left)) >= 0
    took = time.perf_counter() - t
    assert took < 2.0, took
    del keep
