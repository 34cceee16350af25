"""When the adjoint sweeps of several observables run on tiles
(csrc/sweep_cost.hpp): tapes of 8 or 60 gates of one kind on random wires, as the
compiler makes programs of them, against what was measured on a GB300 with the
path switched on and off (us on tiles, us op by op).
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from abi import make_ops
from conftest import ROOT
from test_oracle_golden import ALL_GATES

MEASURED = [
    ("c128", 22, "DoubleExcitation", 60, 16, 27938, 9940),
    ("c128", 22, "DoubleExcitation", 60, 2, 4052, 2162),
    ("c128", 22, "CSWAP", 60, 3, 6291, 2953),
    ("c128", 22, "Toffoli", 60, 6, 10425, 5099),
    ("c128", 24, "CSWAP", 8, 6, 8639, 4427),
    ("c128", 24, "Toffoli", 8, 3, 4160, 2271),
    ("c128", 24, "DoubleExcitation", 8, 2, 2764, 1675),
    ("c64", 22, "DoubleExcitation", 60, 16, 11908, 7023),
    ("c128", 20, "DoubleExcitation", 60, 6, 3169, 1933),
    ("c128", 22, "CSWAP", 8, 16, 6031, 3481),
    ("c64", 24, "Toffoli", 8, 6, 2971, 2138),
    ("c64", 22, "CSWAP", 60, 16, 10725, 8725),
    ("c128", 24, "CZ", 8, 6, 5847, 4596),
    ("c128", 24, "ControlledPhaseShift", 8, 6, 7332, 5172),
    ("c128", 22, "RX", 60, 3, 1795, 9357),
    ("c128", 22, "IsingXX", 60, 3, 5162, 8892),
    ("c64", 22, "RX", 60, 16, 2576, 19834),
    ("c128", 24, "RZ", 8, 6, 4984, 10030),
    ("c128", 22, "CNOT", 60, 16, 5026, 17452),
    ("c64", 24, "CRX", 8, 3, 1168, 1534),
    ("c128", 18, "DoubleExcitation", 60, 16, 2558, 2947),
    ("c128", 18, "Toffoli", 8, 2, 209, 405),
    ("c64", 20, "SingleExcitation", 60, 6, 1117, 2778),
    ("c128", 22, "DoubleExcitationPlus", 60, 3, 9590, 24154),
    ("c128", 22, "SingleExcitation", 60, 6, 8481, 9290),
    ("c64", 14, "CSWAP", 60, 16, 921, 4984),
    ("c128", 10, "Toffoli", 60, 3, 396, 1188),
]


@pytest.fixture(scope="module")
def chosen(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("cost") / "libsweep_cost.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "pennylane-lightning-kokkos_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "sweep_cost.cpp"), "-o", out], check=True)
    return C.CDLL(out).tiles_chosen


def tape(nq, name, count):
    rng = np.random.default_rng(nq * 100 + count)
    nw, npar = ALL_GATES[name]
    ops = [(name, [int(x) for x in rng.choice(nq, nw, replace=False)], False, [float(rng.uniform(0, 6)) for _ in range(npar)])
           for _ in range(count)]
    ops[0] = ("RX", [0], False, [0.3]) # something to differentiate
    return ops


@pytest.mark.parametrize("dtype,nq,name,count,nobs,tiles,plain", MEASURED)
def test_the_cheaper_way(chosen, dtype, nq, name, count, nobs, tiles, plain):
    ops = tape(nq, name, count)
    arr, keep = make_ops(ops)
    assert chosen(nq, int(dtype == "c64"), nobs, arr, len(ops)) == int(tiles < plain)
    assert chosen(nq, int(dtype == "c64"), 1, arr, len(ops)) == 1
    del keep


def test_layers_of_rotations_stay_on_tiles(chosen):
    from pennylane_lightning_kokkos.circuits import hardware_efficient_ansatz

    for nq in (4, 12, 20, 26):
        ops = hardware_efficient_ansatz(nq, 3, seed=1)
        arr, keep = make_ops(ops)
        for c64 in (0, 1):
            for nobs in (2, 20, 100):
                assert chosen(nq, c64, nobs, arr, len(ops)) == 1
        del keep
