"""Tile programs (csrc/tile_program.hpp) on the CPU against the oracle.

tests/cpp/tile_emulator.cpp compiles an op list with the product's own program
compiler and runs the programs thread by thread in double precision, checking
that every slot of a tile is read exactly once per round.  Programs with
double-float coefficients (48 bits) agree with the oracle within
ops x 2^-45 ~ 1e-11 at 300 ops; with single-precision ones within
ops x 2^-23 ~ 4e-5.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import oracle as O
from abi import make_ops
from conftest import ROOT
from test_oracle_golden import ALL_GATES, rand_state

TOL = {16: 1e-11, 8: 4e-5}


@pytest.fixture(scope="module")
def emulator(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("tile") / "libtile_emulator.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "pennylane-lightning-kokkos_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "tile_emulator.cpp"), "-o", out], check=True)
    return C.CDLL(out).tile_emulate


def emulate(fn, nq, ops, T, R, low, amp, lam, hl=None, slots=None):
    arr, keep = make_ops(ops)
    lam = np.array(lam, dtype=np.complex128)
    h = np.array(lam if hl is None else hl, dtype=np.complex128)
    sl = np.array(slots if slots is not None else [-1] * len(ops), dtype=np.int64)
    ns = int(sl.max()) + 1 if len(sl) else 0
    jac = np.zeros(max(ns, 1))
    rounds = C.c_int()
    p = fn(nq, T, R, low, amp, int(hl is not None), arr, len(ops), sl.ctypes.data_as(C.c_void_p),
           lam.ctypes.data_as(C.c_void_p), h.ctypes.data_as(C.c_void_p), jac.ctypes.data_as(C.c_void_p), ns,
           C.byref(rounds))
    assert p >= 0, f"program check {p}"
    del keep
    return lam, h, jac[:ns], p


def random_ops(nq, count, rng, single_param=False):
    names = sorted(ALL_GATES) + ["MultiRZ"]
    ops = []
    while len(ops) < count:
        name = str(rng.choice(names))
        nw, npar = ALL_GATES.get(name, (-1, 1))
        if nw < 0:
            nw, npar = int(rng.integers(1, nq + 1)), 1
        if nw > nq or (single_param and npar > 1):
            continue
        ops.append((name, [int(w) for w in rng.choice(nq, nw, replace=False)], bool(rng.integers(2)),
                    [float(x) for x in rng.uniform(0, 2 * np.pi, npar)]))
    return ops


# (qubits, T, R, low): whole state in one tile, tiles with outer bits, the fewest free bits of a tile
SHAPES = [(4, 12, 4, 3), (4, 12, 3, 2), (5, 12, 4, 2), (7, 9, 4, 3), (9, 8, 4, 3), (9, 8, 3, 2), (10, 7, 3, 2),
          (11, 9, 4, 3)]


@pytest.mark.parametrize("amp", [8, 16])
@pytest.mark.parametrize("nq,T,R,low", SHAPES)
def test_forward(emulator, nq, T, R, low, amp):
    rng = np.random.default_rng(nq * 100 + T)
    ops = random_ops(nq, 300, rng)
    psi = rand_state(nq, rng)
    got, _, _, _ = emulate(emulator, nq, ops, T, R, low, amp, psi)
    np.testing.assert_allclose(got, O.run_ops(psi.copy(), ops), atol=TOL[amp], rtol=0)


@pytest.mark.parametrize("amp", [8, 16])
@pytest.mark.parametrize("nq,T,R,low", SHAPES)
def test_backward(emulator, nq, T, R, low, amp):
    rng = np.random.default_rng(nq * 100 + T + 1)
    ops = random_ops(nq, 200, rng, single_param=True)
    lam = rand_state(nq, rng)
    obs = [("named", "PauliX", [1])]
    hl = lam.copy()
    O.apply(hl, "PauliX", [1])
    par = [i for i, o in enumerate(ops) if o[3]]
    slots = np.full(len(ops), -1)
    slots[par] = np.arange(len(par))
    got, goth, jac, _ = emulate(emulator, nq, ops, T, R, low, amp, lam, hl, slots)
    np.testing.assert_allclose(jac, O.adjoint_jacobian(lam, obs, ops, list(range(len(par))))[0], atol=TOL[amp] * 10,
                               rtol=0)
    inverse = [(o[0], o[1], not o[2], o[3]) for o in reversed(ops)]
    np.testing.assert_allclose(got, O.run_ops(lam.copy(), inverse), atol=TOL[amp], rtol=0)
    np.testing.assert_allclose(goth, O.run_ops(hl.copy(), inverse), atol=TOL[amp], rtol=0)


@pytest.mark.parametrize("R", [3, 4])
def test_special_angles(emulator, R):
    """Runs that multiply to diagonals, to X, and to the identity, with gradients."""
    nq = 7
    rng = np.random.default_rng(R)
    angles = [0.0, np.pi, -np.pi, 2 * np.pi, np.pi / 2, 3 * np.pi, 1e-9, np.pi + 1e-9]
    ops = []
    for _ in range(150):
        name = str(rng.choice(["RX", "RY", "RZ", "PhaseShift", "Hadamard", "PauliX", "PauliY", "S", "CNOT", "CRY",
                               "IsingXX"]))
        nw, npar = ALL_GATES[name]
        ops.append((name, [int(w) for w in rng.choice(nq, nw, replace=False)], bool(rng.integers(2)),
                    [float(rng.choice(angles)) for _ in range(npar)]))
    lam = rand_state(nq, rng)
    got, _, _, _ = emulate(emulator, nq, ops, 6, R, 2, 16, lam)
    np.testing.assert_allclose(got, O.run_ops(lam.copy(), ops), atol=1e-11, rtol=0)
    hl = lam.copy()
    O.apply(hl, "PauliY", [2])
    par = [i for i, o in enumerate(ops) if o[3]]
    slots = np.full(len(ops), -1)
    slots[par] = np.arange(len(par))
    _, _, jac, _ = emulate(emulator, nq, ops, 6, R, 2, 16, lam, hl, slots)
    ref = O.adjoint_jacobian(lam, [("named", "PauliY", [2])], ops, list(range(len(par))))[0]
    np.testing.assert_allclose(jac, ref, atol=1e-10, rtol=0)


def test_layers_take_few_passes(emulator):
    from pennylane_lightning_kokkos.circuits import hardware_efficient_ansatz

    nq = 12
    rng = np.random.default_rng(1)
    ops = hardware_efficient_ansatz(nq, 4, seed=3)
    psi = rand_state(nq, rng)
    got, _, _, passes = emulate(emulator, nq, ops, 9, 4, 3, 16, psi)
    np.testing.assert_allclose(got, O.run_ops(psi.copy(), ops), atol=1e-11, rtol=0)
    assert passes <= 12
