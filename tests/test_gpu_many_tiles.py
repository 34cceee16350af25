"""GPU: more tiles than the chip holds CTAs, so that a CTA walks several and uses
its shared tile and its sums again.  21 qubits are 512 tiles of a Pauli sum
against at most 456 CTAs.

Tolerances as test_gpu_pauli_tile.py: 1e-12 (complex128) and 2e-6 (complex64) of
the sum of |coefficients|.
"""
import ctypes as C

import numpy as np
import pytest

from abi import State
from pennylane_lightning_kokkos import _native as N
from test_gpu_pauli_modes import applied, packed
from test_oracle_golden import rand_state

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
