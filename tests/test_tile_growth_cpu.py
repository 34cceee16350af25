"""complex128 sweeps leave the cosines of rotations to a later phase table.  What
they hold must stay near the state's own size, whatever the list: a sum's
products are twice as many powers of two above it, and single precision ends at 2^127.

A stage turns at most R bits, by at most sqrt(2) each, and none is opened 2^8 or
more above the state without a table: 2^(8 + R / 2), at most 2^10.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from abi import make_ops
from conftest import ROOT
from test_tile_program_cpu import emulate, emulator, random_ops  # noqa: F401
from test_oracle_golden import rand_state
import oracle as O

QUARTER = np.pi / 2 - 1e-3 # the largest tangents, and each rotation needs its cosine


def chains(nq, kind, count):
    """Rotations that neither merge nor meet a phase: controlled rotations keep them apart."""
    ops = []
    for k in range(count):
        if kind == "one wire":
            ops += [("RY", [0], False, [QUARTER]), ("CRY", [1, 0], False, [0.3])]
        elif kind == "two wires":
            ops += [("RY", [0], False, [QUARTER]), ("RY", [1], False, [-QUARTER]), ("CRY", [k % 2, 1 - k % 2], False, [0.3])]
        else:
            ops += [("RY", [w], False, [QUARTER]) for w in range(4)] + [("CRY", [w, (w + 1) % 4], False, [0.2]) for w in range(4)]
    return ops


@pytest.fixture(scope="module")
def growth(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("tile") / "libtile_growth.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "pennylane-lightning-kokkos_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "tile_growth.cpp"), "-o", out], check=True)
    fn = C.CDLL(out).tile_growth
    fn.restype = C.c_double
    return fn


@pytest.mark.parametrize("bwd", [False, True])
@pytest.mark.parametrize("T,R", [(12, 4), (11, 3)])
@pytest.mark.parametrize("kind", ["one wire", "two wires", "four wires", "random"])
def test_growth_is_bounded(growth, kind, T, R, bwd):
    nq = 14
    ops = random_ops(nq, 600, np.random.default_rng(5), single_param=True) if kind == "random" else chains(nq, kind, 150)
    slots = np.full(len(ops), -1, dtype=np.int64)
    par = [i for i, o in enumerate(ops) if o[3]][:5] # few sums, so that they do not end the passes early
    slots[par] = np.arange(len(par))
    arr, keep = make_ops(ops)
    left = C.c_double()
    most = growth(nq, T, R, 2, int(bwd), arr, len(ops), slots.ctypes.data_as(C.c_void_p), C.byref(left))
    del keep
    assert 0 <= most <= 8 + R / 2 + 1e-6
    assert abs(left.value) < 1e-6


@pytest.mark.parametrize("R", [3, 4])
@pytest.mark.parametrize("kind", ["one wire", "two wires", "four wires"])
def test_chains_match_the_oracle(emulator, kind, R): # noqa: F811
    nq, T = 9, 8
    ops = chains(nq, kind, 40)
    rng = np.random.default_rng(R)
    lam = rand_state(nq, rng)
    got, _, _, _ = emulate(emulator, nq, ops, T, R, 2, 16, lam)
    np.testing.assert_allclose(got, O.run_ops(lam.copy(), ops), atol=1e-11, rtol=0)
    hl = lam.copy()
    O.apply(hl, "PauliX", [1])
    par = [i for i, o in enumerate(ops) if o[3]]
    slots = np.full(len(ops), -1)
    slots[par] = np.arange(len(par))
    _, _, jac, _ = emulate(emulator, nq, ops, T, R, 2, 16, lam, hl, slots)
    np.testing.assert_allclose(jac, O.adjoint_jacobian(lam, [("named", "PauliX", [1])], ops, list(range(len(par))))[0],
                               atol=1e-10, rtol=0)
