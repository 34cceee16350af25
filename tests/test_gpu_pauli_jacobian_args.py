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


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
def test_tapes_that_are_cheaper_gate_by_gate(dtype):
    """Large states under DoubleExcitation (csrc/sweep_cost.hpp): words with every letter
    and coefficient, against the states formed outside, gate by gate."""
    nq, rng = 21, np.random.default_rng(2)
    ops = [("RX", [w], False, [0.2 + w]) for w in range(4)]
    ops += [("DoubleExcitation", [int(w) for w in rng.choice(nq, 4, replace=False)], False, [0.3 + k]) for k in range(24)]
    words = [(0.7, [0, 5, 20], "XYZ"), (-1.3, [], ""), (1.0, [3], "Z"), (2.0, [7, 8], "YI"), (0.0, [1], "X")]
    s = State.from_array(rand_state(nq, rng), dtype)
    before = s.get()
    arr, keep = make_ops(ops)
    c, cp = f64([w[0] for w in words])
    off, offp = i64(np.cumsum([0] + [len(w[1]) for w in words]))
    wi, wp = i64([x for w in words for x in w[1]])
    tp, tpp = i64(range(0, len(ops), 3))
    jac = np.zeros((len(words), len(tp)))
    ref = np.zeros_like(jac)
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    N.check(N.lib.plk_adjoint_jacobian_pauli(s.h, len(words), cp, offp, wp, "".join(w[2] for w in words).encode(), arr,
                                             len(ops), tpp, len(tp), ptr(jac)))
    np.testing.assert_array_equal(s.get(), before)
    hls = []
    for k, w in enumerate(words):
        h = State(nq, dtype)
        o1, o1p = i64([0, len(w[1])])
        w1, w1p = i64(w[1] or [0])
        N.check(N.lib.plk_apply_pauli_sum(h.h, s.h, 1, f64([w[0]])[1], o1p, w1p, w[2].encode()))
        hls.append(h)
    harr = (C.c_void_p * len(hls))(*[h.h.value for h in hls])
    N.check(N.lib.plk_set_window_path(0))
    try:
        N.check(N.lib.plk_adjoint_jacobian(s.h, harr, len(hls), arr, len(ops), tpp, len(tp), ptr(ref)))
    finally:
        N.check(N.lib.plk_set_window_path(1))
    np.testing.assert_allclose(jac, ref, atol=1e-5 if dtype == N.PLK_C64 else 1e-11, rtol=0)
    for x in hls + [s]:
        x.close()
    del keep
