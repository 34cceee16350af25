"""Which words of an applied Pauli sum go to tiles (csrc/pauli_plan.hpp).

The passes are compared with a plain restatement of the rule that finds them.
The split between tiles and the plain kernel is compared with what was measured
on a GB300: sums of random words, times in us of the whole call, on tiles (every
pass that the rule for 24 qubits would have kept) and in plain passes.
"""
import ctypes as C
import os
import subprocess
from collections import Counter

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("plan") / "libpauli_plan.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "pennylane-lightning-kokkos_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "pauli_plan.cpp"), "-o", out], check=True)
    return C.CDLL(out)


def patterns(nq, weight, words):
    """X patterns and their numbers of words in a sum of random words of one weight."""
    rng = np.random.default_rng(nq * 1000 + weight * 10 + words)
    wires = [(float(rng.standard_normal()), [int(x) for x in rng.choice(nq, weight, replace=False)])[1] for _ in range(words)]
    xs = Counter(sum(1 << (nq - 1 - w) for w, l in zip(ws, rng.choice(list("XYZ"), weight)) if l in "XY") for ws in wires)
    return sorted(xs.items())


def arrays(groups):
    x = np.array([g[0] for g in groups], dtype=np.uint64)
    n = np.array([g[1] for g in groups], dtype=np.int32)
    return x, n, x.ctypes.data_as(C.c_void_p), n.ctypes.data_as(C.c_void_p)


def passes_of(nq, T, low, groups):
    """Restated: the widest pattern left, then whichever needs the fewest more bits."""
    mask, done, out = (1 << low) - 1, set(), []
    order = sorted(range(len(groups)), key=lambda i: -bin(groups[i][0] & ~mask).count("1"))
    for seed in order:
        if seed in done:
            continue
        bits = mask | groups[seed][0]
        if T < nq and bin(bits).count("1") > T:
            done.add(seed)
            continue
        while True:
            more = [(bin(bits | groups[i][0]).count("1"), k, i) for k, i in enumerate(order)
                    if i not in done and groups[i][0] & ~bits]
            more = [m for m in more if m[0] <= T]
            if not more:
                break
            bits |= groups[min(more)[2]][0]
        b = 0
        while b < nq and bin(bits).count("1") < T:
            bits |= 1 << b
            b += 1
        inside = [i for i in range(len(groups)) if i not in done and not groups[i][0] & ~bits]
        done |= set(inside)
        if not (len(inside) == 1 and T < nq):
            out.append((bits, inside))
    return out


@pytest.mark.parametrize("low", [2, 3])
@pytest.mark.parametrize("nq,weight,words", [(6, 3, 40), (12, 5, 60), (13, 1, 30), (13, 4, 100), (18, 3, 100), (20, 9, 80),
                                             (32, 2, 100), (32, 14, 30)])
def test_passes(lib, nq, weight, words, low):
    groups = patterns(nq, weight, words)
    T = min(12, nq)
    x, n, xp, np_ = arrays(groups)
    of, bits = np.zeros(len(groups), dtype=np.int32), np.zeros(len(groups), dtype=np.uint32)
    k = lib.plan_passes(nq, T, low, len(groups), xp, np_, of.ctypes.data_as(C.c_void_p), bits.ctypes.data_as(C.c_void_p))
    want = passes_of(nq, T, low, groups)
    assert k == len(want)
    for p, (b, inside) in enumerate(want):
        assert int(bits[p]) == b
        assert [int(i) for i in np.flatnonzero(of == p)] == inside


# (dtype, qubits, weight, words, us on tiles, us plain)
MEASURED = [
    ("c64", 18, 8, 100, 115, 73), ("c64", 18, 3, 10, 32, 21), ("c64", 18, 4, 10, 33, 21), ("c64", 18, 6, 100, 114, 78),
    ("c64", 18, 4, 40, 60, 41), ("c64", 18, 6, 40, 58, 40), ("c64", 18, 4, 100, 93, 80), ("c64", 19, 3, 10, 33, 23),
    ("c64", 19, 6, 100, 124, 93), ("c64", 19, 8, 100, 121, 92), ("c64", 19, 8, 40, 60, 46), ("c64", 19, 4, 40, 61, 48),
    ("c64", 20, 2, 10, 35, 28), ("c64", 20, 8, 40, 77, 64), ("c64", 21, 8, 40, 117, 103),
    ("c128", 18, 8, 40, 113, 74), ("c128", 18, 6, 10, 46, 31), ("c128", 18, 3, 10, 45, 30), ("c128", 18, 8, 100, 227, 161),
    ("c128", 18, 6, 40, 90, 74), ("c128", 19, 8, 10, 54, 40),
    ("c64", 18, 1, 100, 53, 77), ("c64", 20, 1, 100, 62, 212), ("c64", 24, 2, 40, 336, 753), ("c64", 24, 4, 100, 888, 1621),
    ("c128", 18, 1, 100, 81, 123), ("c128", 18, 2, 40, 58, 83), ("c128", 20, 4, 100, 223, 463), ("c128", 24, 4, 40, 1220, 2522),
]


@pytest.mark.parametrize("dtype,nq,weight,words,tiles,plain", MEASURED)
def test_split_follows_what_was_measured(lib, dtype, nq, weight, words, tiles, plain):
    groups = patterns(nq, weight, words)
    x, n, xp, np_ = arrays(groups)
    on = lib.plan_words_on_tiles(nq, int(dtype == "c64"), len(groups), xp, np_)
    if tiles < plain:
        assert on >= words // 2
    else: # none, or a part that the model expects to gain from
        assert on <= words // 2


@pytest.mark.parametrize("c64", [0, 1])
@pytest.mark.parametrize("nq", [18, 22, 32])
def test_edges(lib, nq, c64):
    for groups in ([(0, 1), (1, 1)], [((1 << nq) - 1, 1), (1, 1)], [(0, 100), (3, 1)], [(1 << (nq - 1), 50), (1, 50)]):
        x, n, xp, np_ = arrays(groups)
        assert 0 <= lib.plan_words_on_tiles(nq, c64, len(groups), xp, np_) <= sum(g[1] for g in groups)
