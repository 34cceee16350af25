"""The work a user of this simulator has it do, as cases that can be timed.

A case is one pass through the public entry points: a circuit given as an op
list and its PauliZ expectation values, gates called one by one, the Jacobian
of several observables, the gradient of one Hamiltonian through the torch op,
a batch of independent circuits, a Hamiltonian's expectation value, and
marginal probabilities with samples.  complex128 is the default precision of
the device layer, complex64 its other one.  Results of complex64 states are
returned in single precision, which is what they carry.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "pennylane-lightning-kokkos_gb300"))

ANSATZE = ("hea", "rot", "qaoa", "givens")
ROTATIONS = {"hea": ("RY", "RZ"), "rot": ("RX", "RY", "RZ")}
# real floating-point operations per amplitude of the state
FLOPS = {"RX": 6, "RY": 6, "RZ": 6, "Hadamard": 4, "IsingZZ": 6, "IsingXX": 6, "CRY": 3, "SingleExcitation": 3,
         "DoubleExcitation": 0.75, "Haar2q": 30, "CNOT": 0, "PauliX": 0}


def listed():
    return [
        # a small variational circuit, evaluated over and over: launches and host time
        {"name": "circuit_6q_c128", "kind": "circuit", "dtype": "c128", "qubits": 6, "ansatz": "rot", "layers": 2},
        # an ordinary circuit of an odd size in single precision, the state well inside the L2 cache
        {"name": "circuit_15q_c64", "kind": "circuit", "dtype": "c64", "qubits": 15, "ansatz": "hea", "layers": 8},
        # chemistry: excitation gates on a Hartree-Fock state
        {"name": "circuit_19q_c128", "kind": "circuit", "dtype": "c128", "qubits": 19, "ansatz": "givens", "layers": 4},
        # a large hardware-efficient circuit in the default precision
        {"name": "circuit_25q_c128", "kind": "circuit", "dtype": "c128", "qubits": 25, "ansatz": "hea", "layers": 4},
        # QAOA on a large ring in single precision
        {"name": "circuit_27q_c64", "kind": "circuit", "dtype": "c64", "qubits": 27, "ansatz": "qaoa", "layers": 2},
        # gates called one at a time, as a device without op lists does: the nine gates of the repository's sweep
        {"name": "gates_26q_c128", "kind": "gates", "dtype": "c128", "qubits": 26, "reps": 1},
        # a training step of a small model: forward and the Jacobian of a PauliZ on every wire
        {"name": "jacobian_8q_c64", "kind": "jacobian", "dtype": "c64", "qubits": 8, "ansatz": "rot", "layers": 3},
        # the repository's plain workload: 20 qubits, 600 parameters, 20 observables
        {"name": "jacobian_20q_c128", "kind": "jacobian", "dtype": "c128", "qubits": 20, "ansatz": "rot",
         "layers": 10},
        # gradients of a Hamiltonian through the torch op, both precisions (the repository's adjoint workload, shallower)
        {"name": "gradient_25q_c128", "kind": "gradient", "dtype": "c128", "qubits": 25, "ansatz": "hea", "layers": 4,
         "words": 100},
        {"name": "gradient_26q_c64", "kind": "gradient", "dtype": "c64", "qubits": 26, "ansatz": "hea", "layers": 6,
         "words": 100},
        # many uneven circuits at once (the repository's batch workload, fewer circuits)
        {"name": "batch_128_c64", "kind": "batch", "dtype": "c64", "circuits": 128, "min_qubits": 8, "max_qubits": 20,
         "max_layers": 30},
        # energy of a prepared state
        {"name": "hamiltonian_26q_c128", "kind": "hamiltonian", "dtype": "c128", "qubits": 26, "words": 100},
    ]


def draw(rng):
    kind = rng.choice(["circuit"] * 5 + ["gates", "jacobian", "jacobian", "gradient", "gradient", "batch",
                                         "hamiltonian"])
    dtype = rng.choice(["c64", "c128"])
    top = 26 if dtype == "c64" else 25
    if kind == "circuit":
        n = rng.randint(5, top)
        a = rng.choice(ANSATZE)
        most = max(1, min(12, 300 * (1 << 25) // (len(_shape(n, a, 1)) << n)))
        return {"kind": kind, "dtype": dtype, "qubits": n, "ansatz": a, "layers": rng.randint(1, most)}
    if kind == "gates":
        return {"kind": kind, "dtype": dtype, "qubits": rng.randint(8, top), "reps": rng.randint(1, 2)}
    if kind == "jacobian":
        n = rng.randint(5, 20)
        a = rng.choice(ANSATZE)
        most = max(1, min(10, 800 * 20 * (1 << 20) // (n * len(_shape(n, a, 1)) << n)))
        return {"kind": kind, "dtype": dtype, "qubits": n, "ansatz": a, "layers": rng.randint(1, most)}
    if kind == "gradient":
        n = rng.randint(6, top)
        a = rng.choice(ANSATZE)
        most = max(1, min(12, 300 * (1 << 25) // (len(_shape(n, a, 1)) << n)))
        return {"kind": kind, "dtype": dtype, "qubits": n, "ansatz": a, "layers": rng.randint(1, most),
                "words": rng.randint(5, 100)}
    if kind == "batch":
        hi = rng.randint(10, 20)
        return {"kind": kind, "dtype": "c64", "circuits": rng.randint(24, 128), "min_qubits": rng.randint(4, 8),
                "max_qubits": hi, "max_layers": rng.randint(6, 30)}
    return {"kind": kind, "dtype": dtype, "qubits": rng.randint(10, top), "words": rng.randint(10, 100)}


# ------------------------------------------------------------------ circuits
def _shape(n, ansatz, layers):
    """[(gate name, wires, number of parameters)] of a circuit on n wires."""
    ops = []
    if ansatz == "qaoa":
        ops += [("Hadamard", (w,), 0) for w in range(n)]
    elif ansatz == "givens":
        ops += [("PauliX", (w,), 0) for w in range(n // 2)]
    for _ in range(layers):
        if ansatz in ROTATIONS:
            ops += [(r, (w,), 1) for w in range(n) for r in ROTATIONS[ansatz]]
            ops += [("CNOT", (w, (w + 1) % n), 0) for w in range(n if ansatz == "rot" else n - 1)]
        elif ansatz == "qaoa":
            ops += [("IsingZZ", (w, (w + 1) % n), 1) for w in range(n)]
            ops += [(r, (w,), 1) for r in ("RZ", "RX") for w in range(n)]
        else:
            ops += [("SingleExcitation", (w, w + 1), 1) for p in (0, 1) for w in range(p, n - 1, 2)]
            ops += [("DoubleExcitation", (w, w + 1, w + 2, w + 3), 1) for w in range(0, n - 3, 2)]
    return ops


def _circuit(case, seed):
    """[(gate name, wires, inverse, parameters)]; angles uniform, small ones for the excitations."""
    rng = np.random.default_rng(seed)
    span = 0.6 if case["ansatz"] == "givens" else 2 * np.pi
    return [(g, list(w), False, [float(rng.uniform(0, span)) for _ in range(k)])
            for g, w, k in _shape(case["qubits"], case["ansatz"], case["layers"])]


def _words(case, seed):
    """Pauli words of weight 1 to 4 with normal coefficients, as the repository's own Hamiltonians."""
    rng = np.random.default_rng(seed + 7)
    words = []
    for _ in range(case["words"]):
        k = int(rng.integers(1, 5))
        words.append((float(rng.standard_normal()), [int(w) for w in rng.choice(case["qubits"], k, replace=False)],
                      "".join(str(x) for x in rng.choice(list("XYZ"), k))))
    return words


def _haar(dim, rng):
    z = rng.standard_normal((dim, dim)) + 1j * rng.standard_normal((dim, dim))
    q, r = np.linalg.qr(z)
    return q * (np.diag(r) / np.abs(np.diag(r)))


def _gate_calls(case, seed):
    """[(gate name, wires, parameters, matrix)]: nine gates on low, middle and high wires."""
    rng = np.random.default_rng(seed)
    n = case["qubits"]
    pools = (range(0, 5), range(n // 2 - 3, n // 2 + 3), range(n - 5, n))
    calls = []
    for g, k, p in (("PauliX", 1, 0), ("Hadamard", 1, 0), ("RX", 1, 1), ("CNOT", 2, 0), ("CRY", 2, 1),
                    ("IsingXX", 2, 1), ("SingleExcitation", 2, 1), ("DoubleExcitation", 4, 1), ("Haar2q", 2, 0)):
        for pool in pools:
            for _ in range(case["reps"]):
                w = [int(x) for x in rng.choice(list(pool), k, replace=False)]
                calls.append((g, w, [float(rng.uniform(0, 2 * np.pi)) for _ in range(p)],
                              _haar(4, rng) if g == "Haar2q" else None))
    return calls


def _batch(case, seed):
    """[(qubits, ops, words)] of uneven circuits: RX, RY, RZ on every wire and a CNOT ladder, 5 layers and more."""
    size = np.random.default_rng(5)  # the circuits' sizes belong to the case
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["circuits"]):
        n = int(size.integers(case["min_qubits"], case["max_qubits"] + 1))
        ops = []
        for _ in range(int(size.integers(5, case["max_layers"] + 1))):
            angles = rng.uniform(0, 2 * np.pi, (n, 3))
            ops += [(r, [w], False, [float(angles[w, k])]) for w in range(n) for k, r in enumerate(ROTATIONS["rot"])]
            ops += [("CNOT", [w, w + 1], False, []) for w in range(n - 1)]
        out.append((n, ops, _words({"qubits": n, "words": 10}, int(rng.integers(1 << 30)))))
    return out


def _random_state(n, seed, product=0.0):
    """Random amplitudes, or a random product state with some of them added."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.view_as_complex(torch.randn(1 << n, 2, generator=g, device="cuda", dtype=torch.float64))
    v /= torch.linalg.vector_norm(v)
    if product:
        rng = np.random.default_rng(seed)
        u = torch.ones(1, dtype=torch.complex128, device="cuda")
        for t, f in rng.uniform(0, np.pi, (n, 2)):
            q = torch.tensor([math.cos(t), math.sin(t) * complex(math.cos(f), math.sin(f))], dtype=u.dtype, device="cuda")
            u = torch.outer(u, q).reshape(-1)
        v.mul_(1 - product).add_(u, alpha=product)
        v /= torch.linalg.vector_norm(v)
    return v


# ------------------------------------------------------------------- prepare
class _View:
    """The state's own device buffer as an array of (re, im) pairs; it keeps the state."""

    def __init__(self, sv, n, dtype):
        self.sv = sv
        self.__cuda_array_interface__ = {"shape": (1 << n, 2), "typestr": "<f4" if dtype == "c64" else "<f8",
                                         "data": (sv.device_ptr(), False), "version": 2}


def _state(case):
    import pennylane_lightning_kokkos.lightning_kokkos_qubit_ops as m

    sv = getattr(m, "LightningKokkos_C" + case["dtype"][1:])(case["qubits"])
    return m, sv, torch.as_tensor(_View(sv, case["qubits"], case["dtype"]), device="cuda")


def _set(view, psi):
    view.copy_(torch.view_as_real(psi))
    torch.cuda.synchronize()


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    c64 = case["dtype"] == "c64"
    s["real"] = np.float32 if c64 else np.float64
    cplx = np.complex64 if c64 else np.complex128
    if kind == "gradient":
        from pennylane_lightning_kokkos.torch_adjoint import AdjointCircuit

        ops = _circuit(case, seed)
        s["circuit"] = AdjointCircuit(case["qubits"], [o[:3] for o in ops], [_words(case, seed)], dtype=case["dtype"])
        s["params"] = torch.tensor([x for o in ops for x in o[3]], device="cuda",
                                   dtype=torch.float32 if c64 else torch.float64)
        return s
    if kind == "batch":
        from pennylane_lightning_kokkos.batch import CircuitBatch

        s["batch"] = CircuitBatch(case["dtype"])
        work = _batch(case, seed)
        for n, ops, words in work:
            s["batch"].add(n, ops, words)
        s["params"] = np.array([x for _, ops, _ in work for o in ops for x in o[3]])
        return s
    m, sv, view = _state(case)
    s.update(sv=sv, view=view, none=np.array([], dtype=cplx))
    if kind in ("circuit", "jacobian"):
        ops = _circuit(case, seed)
        s["ops"] = ([o[0] for o in ops], [o[1] for o in ops], [o[2] for o in ops], [o[3] for o in ops])
    if kind == "jacobian":
        bits = case["dtype"][1:]
        s["adjoint"] = getattr(m, "AdjointJacobianKokkos_C" + bits)()
        s["obs"] = [getattr(m, "NamedObsKokkos_C" + bits)("PauliZ", [w]) for w in range(case["qubits"])]
        s["tape"] = s["adjoint"].create_ops_list(s["ops"][0], [np.array(p, dtype=s["real"]) for p in s["ops"][3]],
                                                 s["ops"][1], s["ops"][2], [s["none"]] * len(ops))
        s["trainable"] = list(range(sum(len(o[3]) for o in ops)))
    elif kind == "gates":
        _set(view, _random_state(case["qubits"], seed))
        s["calls"] = [(g, w, p, None if u is None else u.astype(cplx)) for g, w, p, u in _gate_calls(case, seed)]
    elif kind == "hamiltonian":
        _set(view, _random_state(case["qubits"], seed, 0.7))
        words = _words(case, seed)
        s["words"] = ([c for c, _, _ in words], [w for _, w, _ in words], [l for _, _, l in words])
    return s


# ----------------------------------------------------------------------- run
def run(s):
    kind = s["case"]["kind"]
    if kind == "circuit":
        sv = s["sv"]
        sv.resetKokkos()
        sv.apply(*s["ops"])
        z = [sv.ExpectationValue("PauliZ", [w], [], s["none"]) for w in range(s["case"]["qubits"])]
        return {"state": s["view"], "z": np.array(z, dtype=s["real"])}
    if kind == "jacobian":
        sv = s["sv"]
        sv.resetKokkos()
        sv.apply(*s["ops"])
        return {"state": s["view"],
                "jacobian": s["adjoint"].adjoint_jacobian(sv, s["obs"], s["tape"], s["trainable"])}
    if kind == "gates":
        sv = s["sv"]
        for g, w, p, u in s["calls"]:
            if u is not None:
                sv.apply("QubitUnitary", w, False, [], u)
            else:
                getattr(sv, g)(w, False, p)
        return s["view"]
    if kind == "hamiltonian":
        return s["real"](s["sv"].ExpectationValuePauliSum(*s["words"]))
    if kind == "gradient":
        p = s["params"].detach().requires_grad_()
        value = s["circuit"](p)
        value.sum().backward()
        return {"value": value.detach().to(p.dtype), "gradient": p.grad}
    values, jac = s["batch"].run(s["params"])
    return {"values": values.astype(s["real"]), "jacobian": jac.astype(s["real"])}


# ---------------------------------------------------------------------- work
def _flops(n, names):
    return sum(FLOPS[g] for g in names) * float(1 << n)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        mean = [_shape(n, "hea", 1) for n in range(case["min_qubits"], case["max_qubits"] + 1)]
        depth = (5 + case["max_layers"]) / 2
        f = sum(1.5 * 3 * depth * _flops(case["min_qubits"] + i, [o[0] for o in ops]) for i, ops in enumerate(mean))
        npar = sum(3 * depth * (case["min_qubits"] + i) for i in range(len(mean)))
        return {"bytes": 16.0 * npar / len(mean) * case["circuits"], "flops": f / len(mean) * case["circuits"]}
    n = case["qubits"]
    state = float(1 << n) * (8 if case["dtype"] == "c64" else 16)
    if kind == "hamiltonian":
        return {"bytes": state, "flops": 4.0 * case["words"] * (1 << n)}
    if kind == "gates":
        names = [c[0] for c in _gate_calls(case, 0)]
        return {"bytes": 2 * state, "flops": _flops(n, names)}
    shape = _shape(n, case["ansatz"], case["layers"])
    f = _flops(n, [o[0] for o in shape])
    npar = sum(o[2] for o in shape)
    if kind == "circuit":
        return {"bytes": state, "flops": f + 3.0 * n * (1 << n)}
    if kind == "jacobian":
        # forward, then the sweep of lambda and of every observable's state with the inner products
        return {"bytes": state + 8.0 * npar * n, "flops": f * (2 + n) + 4.0 * npar * n * (1 << n)}
    return {"bytes": state, "flops": 3 * f + 4.0 * npar * (1 << n) + 8.0 * case["words"] * (1 << n)}


# --------------------------------------------------------------------- exact
def _sel(psi, n, wires, bits):
    """View of the amplitudes whose `wires` have the given bits."""
    order = sorted(range(len(wires)), key=lambda i: wires[i])
    shape, at, last = [], [], -1
    for i in order:
        shape += [1 << (wires[i] - last - 1), 2]
        at += [slice(None), bits[i]]
        last = wires[i]
    return psi.view(shape + [1 << (n - 1 - last)])[tuple(at)]


def _mix(a, b, m):
    """(a, b) <- m (a, b)"""
    x = a * m[0][0]
    x.add_(b, alpha=m[0][1])
    b.mul_(m[1][1])
    b.add_(a, alpha=m[1][0])
    a.copy_(x)


PAIRS = {"SingleExcitation": ((0, 1), (1, 0)), "DoubleExcitation": ((0, 0, 1, 1), (1, 1, 0, 0))}


def _apply(psi, n, name, wires, params, inverse=False, matrix=None):
    t = (-params[0] if inverse else params[0]) if params else 0.0
    c, s, r = math.cos(t / 2), math.sin(t / 2), math.sqrt(0.5)
    if matrix is not None:
        q = [_sel(psi, n, wires, b) for b in ((0, 0), (0, 1), (1, 0), (1, 1))]
        old = [x.clone() for x in q]
        for i in range(4):
            q[i].zero_()
            for j in range(4):
                q[i].add_(old[j], alpha=complex(matrix[i, j]))
        return
    if name in ("RZ", "IsingZZ"):
        for i in range(2 ** len(wires)):
            bits = [(i >> j) & 1 for j in range(len(wires))]
            _sel(psi, n, wires, bits).mul_(complex(c, s if sum(bits) & 1 else -s))
        return
    if name == "IsingXX":
        for p, q in (((0, 0), (1, 1)), ((0, 1), (1, 0))):
            _mix(_sel(psi, n, wires, p), _sel(psi, n, wires, q), [[c, -1j * s], [-1j * s, c]])
        return
    if name in PAIRS:
        a, b, m = *(_sel(psi, n, wires, k) for k in PAIRS[name]), [[c, -s], [s, c]]
    elif name in ("CNOT", "CRY"):
        a, b = (_sel(psi, n, wires, (1, k)) for k in (0, 1))
        m = [[0, 1], [1, 0]] if name == "CNOT" else [[c, -s], [s, c]]
    else:
        a, b = (_sel(psi, n, wires, (k,)) for k in (0, 1))
        m = {"RX": [[c, -1j * s], [-1j * s, c]], "RY": [[c, -s], [s, c]], "Hadamard": [[r, r], [r, -r]],
             "PauliX": [[0, 1], [1, 0]]}[name]
    _mix(a, b, m)


def _dot(h, v):
    return (h.conj() * v).sum()


def _generator(h, v, n, name, wires):
    """Im <h|G|v> of the gate exp(-i t G / 2)."""
    if name in ("RZ", "IsingZZ"):
        out = 0
        for i in range(2 ** len(wires)):
            bits = [(i >> j) & 1 for j in range(len(wires))]
            out = out + _dot(_sel(h, n, wires, bits), _sel(v, n, wires, bits)).imag * (-1 if sum(bits) & 1 else 1)
        return out
    k = PAIRS.get(name, ((0,), (1,)))
    x = _dot(_sel(h, n, wires, k[0]), _sel(v, n, wires, k[1]))
    y = _dot(_sel(h, n, wires, k[1]), _sel(v, n, wires, k[0]))
    return x.imag + y.imag if name == "RX" else y.real - x.real


def _zero(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1
    return psi


def _forward(n, ops):
    psi = _zero(n)
    for g, w, inv, p in ops:
        _apply(psi, n, g, w, p, inv)
    return psi


def _adjoint(psi, hs, n, ops):
    """[observable][parameter] gradients, from the final state and the observables' states (both overwritten)."""
    out = []
    for g, w, inv, p in reversed(ops):
        if p:
            out.append(torch.stack([_generator(h, psi, n, g, w) for h in hs]))
        for v in [psi] + hs:
            _apply(v, n, g, w, p, not inv)
    return torch.stack(out[::-1], dim=1)


def _word(psi, n, wires, letters):
    out = psi.clone()
    for w, l in zip(wires, letters):
        a, b = _sel(out, n, (w,), (0,)), _sel(out, n, (w,), (1,))
        if l == "Z":
            b.neg_()
        else:
            x = a.clone()
            a.copy_(b if l == "X" else b * -1j)
            b.copy_(x if l == "X" else x * 1j)
    return out


def _observe(psi, n, words):
    out = torch.zeros_like(psi)
    for c, w, l in words:
        out.add_(_word(psi, n, w, l), alpha=c)
    return out


def _z(psi, n):
    p = psi.abs().square()
    return [float(_sel(p, n, (w,), (0,)).sum() - _sel(p, n, (w,), (1,)).sum()) for w in range(n)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        if case["circuits"] * case["max_qubits"] * (case["max_layers"] + 5) > 100_000:
            return None
        values, grads = [], []
        for n, ops, words in _batch(case, seed):
            psi = _forward(n, ops)
            h = _observe(psi, n, words)
            values.append(_dot(psi, h).real)
            grads.append(_adjoint(psi, [h], n, ops)[0])
        return {"values": torch.stack(values), "jacobian": torch.cat(grads)}
    n = case["qubits"]
    if kind == "hamiltonian":
        psi = _random_state(n, seed, 0.7)
        if case["dtype"] == "c64":
            psi = psi.to(torch.complex64).to(torch.complex128)
        return np.float64(sum(c * float(_dot(psi, _word(psi, n, w, l)).real) for c, w, l in _words(case, seed)))
    if kind == "gates":
        psi = _random_state(n, seed)
        if case["dtype"] == "c64":
            psi = psi.to(torch.complex64).to(torch.complex128)
        for g, w, p, u in _gate_calls(case, seed):
            _apply(psi, n, g, w, p, False, u)
        return torch.view_as_real(psi)
    ops = _circuit(case, seed)
    if kind == "gradient" and case["dtype"] == "c64":  # the parameters that the call is given
        ops = [(g, w, i, [float(np.float32(x)) for x in p]) for g, w, i, p in ops]
    psi = _forward(n, ops)
    if kind == "circuit":
        return {"state": torch.view_as_real(psi), "z": np.array(_z(psi, n))}
    if kind == "gradient":
        h = _observe(psi, n, _words(case, seed))
        value = _dot(psi, h).real.reshape(1)
        return {"value": value, "gradient": _adjoint(psi, [h], n, ops)[0]}
    if case["qubits"] * len(ops) * (1 << n) > 3e10:
        return None
    state = torch.view_as_real(psi.clone())
    hs = [_word(psi, n, [w], "Z") for w in range(n)]
    return {"state": state, "jacobian": _adjoint(psi, hs, n, ops)}
