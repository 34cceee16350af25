"""GPU: Pauli sums of complex128 states in both arithmetic modes, on amplitudes of
thirty decades and, in native FP64, beyond single precision's exponents.

Expectation values and applied sums: within 1e-12 of the sum of |coefficients|
(double-float, as test_gpu_pauli_tile.py).  The huge and tiny amplitudes multiply
to 1 exactly.
"""
import ctypes as C

import numpy as np
import pytest

from abi import State, f64, i64
from pennylane_lightning_kokkos import _native as N
from test_gpu_dynamic_range import mode, wide_state  # noqa: F401
from test_gpu_pauli_tile import words_for

pytestmark = pytest.mark.gpu


def packed(words):
    c, cp = f64([w[0] for w in words])
    off, offp = i64(np.cumsum([0] + [len(w[1]) for w in words]))
    wi, wp = i64([x for w in words for x in w[1]] or [0])
    return (c, off, wi), (len(words), cp, offp, wp, "".join(w[2] for w in words).encode())


def parity(v):
    v = v.copy()
    for s in (16, 8, 4, 2, 1):
        v ^= v >> s
    return v & 1


def applied(psi, nq, words):
    out, idx = np.zeros_like(psi), np.arange(1 << nq)
    for c, wires, letters in words:
        x = sum(1 << (nq - 1 - w) for w, l in zip(wires, letters) if l in "XY")
        z = sum(1 << (nq - 1 - w) for w, l in zip(wires, letters) if l in "YZ")
        src = idx ^ x
        out += c * 1j ** letters.count("Y") * (1 - 2 * parity(src & z)) * psi[src]
    return out


@pytest.mark.parametrize("kind", ["narrow", "shared"])
@pytest.mark.parametrize("nq", [5, 13, 18])
def test_wide_state(nq, kind, mode): # noqa: F811
    rng = np.random.default_rng(17 * nq)
    psi = wide_state(nq, rng)
    words = words_for(nq, rng, kind)
    ref = applied(psi, nq, words)
    keep, args = packed(words)
    scale = float(np.sum(np.abs(keep[0])))
    s, o, v = State.from_array(psi, N.PLK_C128), State(nq, N.PLK_C128), C.c_double()
    N.check(N.lib.plk_expval_pauli_sum(s.h, *args, C.byref(v)))
    assert abs(v.value - float(np.vdot(psi, ref).real)) < 1e-12 * scale
    N.check(N.lib.plk_apply_pauli_sum(o.h, s.h, *args))
    np.testing.assert_allclose(o.get(), ref, atol=1e-12 * scale, rtol=0)
    s.close()
    o.close()


@pytest.mark.parametrize("nq", [4, 8, 12, 14])
def test_fp64_products_keep_their_exponents(nq):
    before = N.c128_arithmetic()
    N.set_c128_arithmetic("fp64")
    try:
        psi = np.zeros(1 << nq, dtype=np.complex128)
        psi[0], psi[1 << (nq - 1)] = 2.0**150, 2.0**-150
        psi[1] = 1j * 2.0**-150
        keep, args = packed([(0.25, [0], "X"), (0.5, [nq - 1], "Y"), (4.0, [1, 2], "XX")])
        s, v = State.from_array(psi, N.PLK_C128), C.c_double()
        N.check(N.lib.plk_expval_pauli_sum(s.h, *args, C.byref(v)))
        assert v.value == 2 * 0.25 + 2 * 0.5
        s.close()
    finally:
        N.set_c128_arithmetic(before)
