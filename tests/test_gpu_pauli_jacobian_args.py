"""GPU: what plk_adjoint_jacobian_pauli refuses, and with which message: malformed
words, as the Pauli-sum entry points refuse them, and tapes and modes whose
sweeps do not start from words.  A refused call writes no Jacobian.
"""
import ctypes as C

import numpy as np
import pytest

from abi import State, f64, i64, make_ops
from pennylane_lightning_kokkos import _native as N
from test_oracle_golden import rand_state

pytestmark = pytest.mark.gpu

NQ = 6
OPS = [("RX", [w], False, [0.1 + w]) for w in range(NQ)] + [("CNOT", [w, w + 1], False, []) for w in range(NQ - 1)]
NO_WORDS = "does not start from Pauli words"


def call(offsets, wires, letters, ops=OPS, dtype=N.PLK_C128, coeffs=None):
    s = State.from_array(rand_state(NQ, np.random.default_rng(1)), dtype)
    arr, keep = make_ops(ops)
    n = len(offsets) - 1
    c, cp = f64(coeffs or [1.0] * max(n, 1))
    off, offp = i64(offsets)
    w, wp = i64(wires or [0])
    tp, tpp = i64([0, 2])
    jac = np.full((max(n, 1), 2), 7.0)
    try:
        N.check(N.lib.plk_adjoint_jacobian_pauli(s.h, n, cp, offp, wp, letters.encode(), arr, len(ops), tpp, len(tp),
                                                 jac.ctypes.data_as(C.POINTER(C.c_double))))
    except N.NativeError:
        np.testing.assert_array_equal(jac, 7.0)
        raise
    finally:
        s.close()
        del keep
    return jac


@pytest.mark.parametrize("offsets,wires,letters,message", [
    ([0, 2, 1], [0, 1], "XY", "offsets must be non-decreasing"),
    ([1, 0], [0], "X", "offsets must be non-decreasing"),
    ([0, 1], [NQ], "X", "wire out of range"),
    ([0, 1], [-1], "Z", "wire out of range"),
    ([0, 2], [3, 3], "XZ", "repeated wire"),
    ([0, 1], [0], "Q", "bad Pauli letter"),
    ([0], [0], "X", "bad Pauli-word arguments"),
])
def test_malformed_words(offsets, wires, letters, message):
    with pytest.raises(N.NativeError, match=message):
        call(offsets, wires, letters)


def test_unsupported_tapes_and_modes():
    good = ([0, 1, 3], [0, 1, 2], "XYZ")
    assert np.isfinite(call(*good)).all()
    with pytest.raises(N.NativeError, match=NO_WORDS):
        call(*good, ops=OPS + [("Matrix", [0], False, [], np.eye(2))])
    N.check(N.lib.plk_set_window_path(0))
    try:
        with pytest.raises(N.NativeError, match=NO_WORDS):
            call(*good, dtype=N.PLK_C64)
    finally:
        N.check(N.lib.plk_set_window_path(1))
    before = N.c128_arithmetic()
    N.set_c128_arithmetic("fp64")
    try:
        with pytest.raises(N.NativeError, match=NO_WORDS):
            call(*good)
    finally:
        N.set_c128_arithmetic(before)
