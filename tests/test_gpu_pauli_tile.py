"""GPU: Pauli sums on tiles (expectation value and application) against dense
numpy evaluation, at sizes where tiles change (fewer amplitudes than a block
holds, one tile, several) and for words that share an X pattern, have none, or
are too wide for a tile.

Tolerances, relative to the sum of |coefficients|: complex128 1e-12
(double-float sums, 2^-45 per product, random signs); complex64 2e-6 (2^-24 per
amplitude of a normalised state, eight products per single-precision sum).
"""
import ctypes as C

import numpy as np
import pytest

from abi import State, f64, i64
from pennylane_lightning_kokkos import _native as N
from test_oracle_golden import rand_state

pytestmark = pytest.mark.gpu

TOL = {N.PLK_C64: 2e-6, N.PLK_C128: 1e-12}


def dense(psi, nq, words):
    out = np.zeros_like(psi)
    idx = np.arange(1 << nq)
    for c, wires, letters in words:
        x = z = ny = 0
        for w, l in zip(wires, letters):
            bit = 1 << (nq - 1 - w)
            x |= bit if l in "XY" else 0
            z |= bit if l in "YZ" else 0
            ny += l == "Y"
        par = np.array([bin(int(k)).count("1") & 1 for k in range(1 << 8)])
        src = idx ^ x
        s = src & z
        sign = 1 - 2 * (par[s & 255] ^ par[(s >> 8) & 255])
        out += c * (1j) ** ny * sign * psi[src]
    return out


def words_for(nq, rng, kind):
    words = []
    for k in range(40):
        if kind == "shared": # few X patterns, many sign patterns
            wires = list(range(min(nq, 4)))
            letters = "".join(rng.choice(["XXYZ", "YYXI", "ZZII", "IZZI"])[: len(wires)])
            extra = [int(w) for w in rng.choice(nq, 2, replace=False) if w >= len(wires)]
            wires, letters = wires + extra, letters + "Z" * len(extra)
        else:
            wt = int(rng.integers(1, min(nq, 5) + 1)) if kind == "narrow" else int(rng.integers(1, nq + 1))
            wires = [int(w) for w in rng.choice(nq, wt, replace=False)]
            letters = "".join(str(x) for x in rng.choice(list("XYZ"), wt))
        words.append((float(rng.standard_normal()), wires, letters))
    return words


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
@pytest.mark.parametrize("kind", ["narrow", "wide", "shared"])
@pytest.mark.parametrize("nq", [4, 5, 8, 9, 11, 12, 13, 15])
def test_pauli_sum(nq, kind, dtype):
    rng = np.random.default_rng(31 * nq + len(kind))
    psi = rand_state(nq, rng)
    words = words_for(nq, rng, kind)
    s, o = State.from_array(psi, dtype), State(nq, dtype)
    ref = dense(s.get().astype(np.complex128), nq, words)
    c, cp = f64([w[0] for w in words])
    off, offp = i64(np.cumsum([0] + [len(w[1]) for w in words]))
    wi, wp = i64([x for w in words for x in w[1]])
    letters = "".join(w[2] for w in words).encode()
    scale = float(np.sum(np.abs(c)))
    v = C.c_double()
    N.check(N.lib.plk_expval_pauli_sum(s.h, len(words), cp, offp, wp, letters, C.byref(v)))
    want = float(np.vdot(s.get().astype(np.complex128), ref).real)
    assert abs(v.value - want) < TOL[dtype] * scale
    first = v.value
    N.check(N.lib.plk_expval_pauli_sum(s.h, len(words), cp, offp, wp, letters, C.byref(v)))
    assert v.value == first
    N.check(N.lib.plk_apply_pauli_sum(o.h, s.h, len(words), cp, offp, wp, letters))
    np.testing.assert_allclose(o.get(), ref, atol=TOL[dtype] * scale, rtol=0)
    s.close()
    o.close()


@pytest.mark.parametrize("nq", [9, 13, 16])
def test_cancelling_energy_keeps_low_bits(nq):
    """complex128 energies of many words whose terms cancel, on a state with a few
    large amplitudes.  Coefficients carry 48 bits (2^-49 each), products 2^-48,
    sums are settled after each word: within 2^-46 of the sum of |coefficients|."""
    rng = np.random.default_rng(7 * nq)
    psi = np.ones(1)
    for a in rng.uniform(0.2, 0.6, nq): # product state, probabilities over many decades
        psi = np.kron(psi, [np.cos(a), np.sin(a) * np.exp(1j * a)])
    words = []
    for _ in range(60):
        wt = int(rng.integers(1, 5))
        wires = [int(w) for w in rng.choice(nq, wt, replace=False)]
        letters = "".join(str(x) for x in rng.choice(list("XYZ"), wt))
        c = float(rng.standard_normal())
        words += [(c, wires, letters), (-c * (1 + 1e-9), wires, letters)]
    s = State.from_array(psi, N.PLK_C128)
    want = sum(float(np.vdot(psi, dense(psi, nq, [w])).real) for w in words)
    c, cp = f64([w[0] for w in words])
    off, offp = i64(np.cumsum([0] + [len(w[1]) for w in words]))
    wi, wp = i64([x for w in words for x in w[1]])
    v = C.c_double()
    N.check(N.lib.plk_expval_pauli_sum(s.h, len(words), cp, offp, wp, "".join(w[2] for w in words).encode(), C.byref(v)))
    assert abs(v.value - want) < 2.0**-46 * float(np.sum(np.abs(c)))
    s.close()


@pytest.mark.parametrize("dtype", [N.PLK_C64, N.PLK_C128])
@pytest.mark.parametrize("wt", [2, 7])
def test_application_splits_between_tiles_and_plain_passes(wt, dtype):
    """Narrow words go to tiles, wide ones to the plain kernel, some sums to both
    (18 qubits, the smallest state whose applications use tiles)."""
    nq, rng = 18, np.random.default_rng(wt)
    psi = rand_state(nq, rng)
    words = []
    for k in range(40):
        w = wt if k % 2 else 1
        words.append((float(rng.standard_normal()), [int(x) for x in rng.choice(nq, w, replace=False)],
                      "".join(str(x) for x in rng.choice(list("XYZ"), w))))
    s, o = State.from_array(psi, dtype), State(nq, dtype)
    idx = np.arange(1 << nq)
    par = np.array([bin(k).count("1") & 1 for k in range(1 << 9)])
    have, ref = s.get().astype(np.complex128), np.zeros(1 << nq, dtype=np.complex128)
    for c, wires, letters in words:
        x = sum(1 << (nq - 1 - w) for w, l in zip(wires, letters) if l in "XY")
        z = sum(1 << (nq - 1 - w) for w, l in zip(wires, letters) if l in "YZ")
        t = (idx ^ x) & z
        ref += c * 1j ** letters.count("Y") * (1 - 2 * (par[t & 511] ^ par[t >> 9])) * have[idx ^ x]
    c, cp = f64([w[0] for w in words])
    off, offp = i64(np.cumsum([0] + [len(w[1]) for w in words]))
    wi, wp = i64([x for w in words for x in w[1]])
    N.check(N.lib.plk_apply_pauli_sum(o.h, s.h, len(words), cp, offp, wp, "".join(w[2] for w in words).encode()))
    np.testing.assert_allclose(o.get(), ref, atol=TOL[dtype] * float(np.sum(np.abs(c))), rtol=0)
    s.close()
    o.close()
