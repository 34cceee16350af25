"""Copies of an AdjointCircuit (host side of the torch op, no GPU): the tape that
a call hands to the library points into the copy's own arrays and holds the same
ops, also once the original is gone.
"""
import copy
import ctypes as C
import gc
import pickle

import numpy as np
import pytest

pytest.importorskip("torch")

OPS = [("RY", [3]), ("CNOT", [0, 2]), ("Rot", [1]), ("MultiRZ", [4, 0, 2]), ("CRX", [2, 4], True), ("Hadamard", [0])]


def addresses(tape, n):
    return [C.cast(tape[i].wires, C.c_void_p).value for i in range(n)]


def contents(tape, n):
    return [(tape[i].gate, [tape[i].wires[k] for k in range(tape[i].num_wires)], tape[i].adjoint,
             [tape[i].params[k] for k in range(tape[i].num_params)]) for i in range(n)]


@pytest.mark.parametrize("how", ["deepcopy", "pickle"])
def test_copies_own_what_their_tape_points_to(how):
    from pennylane_lightning_kokkos.torch_adjoint import AdjointCircuit

    original = AdjointCircuit(5, OPS, [[(1.0, [0], "Z")]])
    params = np.arange(1.0, original.num_params + 1)
    n = len(original.ops)
    tape, keep = original._tape(params)
    want, theirs = contents(tape, n), set(addresses(tape, n))
    clone = copy.deepcopy(original) if how == "deepcopy" else pickle.loads(pickle.dumps(original))
    mine, keep2 = clone._tape(params)
    assert not theirs & set(addresses(mine, n)) # before anything is read through them
    del original, tape, keep
    gc.collect()
    assert contents(mine, n) == want
    del keep2


def test_empty_tape():
    from pennylane_lightning_kokkos.torch_adjoint import AdjointCircuit

    c = copy.deepcopy(AdjointCircuit(2, [], [[(1.0, [0], "Z")]]))
    c._tape(np.zeros(0))
    assert c.num_params == 0 and len(c.ops) == 0
