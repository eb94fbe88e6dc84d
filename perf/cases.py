"""Performance cases of the simulate path: circuits, channels, gradients and readouts of the sizes
the repository's configurations, tests and benchmark use, each through the package's public calls.

A case is a dict of plain values; its "kind" says which use it stands for:

  run      one small circuit per call from |0...0>, full probabilities and shots in one round trip
           (a variational or teaching loop over circuits of at most 12 qubits; launches and host
           work are the time)
  sv       complex128 state vector: reinit, evolve, then the readouts of a simulate call
  sv64     complex64 state vector: the same, read out as single-precision expectation values
  dm       density matrix with noise after every gate, in either noise rule: the diagonal and
           expectation values on up to four qubits
  grad     energy and full gradient of a variational ansatz by the adjoint method (complex128
           arrays; complex64 through the torch autograd function with a float32 parameter vector)
  batch    many uneven circuits in one call, Pauli expectation values per circuit (and shots on
           complex128 states)
  readout  results of a state that is already there: Pauli and tensor-product expectation values,
           a marginal, shots

Shots are returned from complex128 states only: they are whole numbers, drawn by comparing against a
running sum, and a single-precision state's last bits move the boundaries themselves.
"""
import math

import numpy as np
import torch

import __graft_entry__ as _entry

_bs = None


def _package():
    global _bs
    if _bs is None:
        _bs = _entry.load_package()
    return _bs


def listed():
    return [
        # the smallest call a user repeats: a GHZ circuit with its probabilities and 1000 shots
        {"name": "run_ghz10", "kind": "run", "circuit": "ghz", "n": 10, "layers": 1, "shots": 1000},
        # one evaluation of a 12-qubit hardware-efficient ansatz
        {"name": "run_ansatz12", "kind": "run", "circuit": "ansatz", "n": 12, "layers": 4, "shots": 1000},
        # ordinary state vectors: 17 qubits with the whole probability vector, 21 with shots
        {"name": "sv17_ansatz", "kind": "sv", "circuit": "ansatz", "n": 17, "layers": 8, "shots": 1000},
        {"name": "sv21_mix", "kind": "sv", "circuit": "mix", "n": 21, "layers": 30, "shots": 1000},
        # the dense random circuit (Haar SU(2) and CZ, then strides 1, 8, 16) on a large state
        {"name": "sv28_dense", "kind": "sv", "circuit": "dense", "n": 28, "layers": 8, "shots": 10000},
        # a large single-precision state under a random mix of gates
        {"name": "sv25_c64_mix", "kind": "sv64", "circuit": "mix", "n": 25, "layers": 30, "shots": 0},
        # noisy density matrices: the reference's noise rule, and the full channel
        {"name": "dm13_reference", "kind": "dm", "mode": "reference", "n": 13, "layers": 3},
        {"name": "dm12_physical", "kind": "dm", "mode": "physical", "n": 12, "layers": 4},
        # training steps: energy and all gradients
        {"name": "grad20", "kind": "grad", "precision": "c128", "n": 20, "layers": 5, "terms": 24},
        {"name": "grad22_c64", "kind": "grad", "precision": "c64", "n": 22, "layers": 6, "terms": 48},
        # many uneven circuits at once, in the benchmark's gate mix
        {"name": "batch48_c64", "kind": "batch", "precision": "c64", "circuits": 48, "lo": 12, "hi": 22, "layers": 40, "shots": 0},
        # readouts of a large state
        {"name": "readout26", "kind": "readout", "n": 26, "terms": 12, "shots": 100000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "sv", "sv64", "dm", "grad", "batch", "readout"])
    if kind == "run":
        return {"kind": kind, "circuit": rng.choice(["ghz", "ansatz", "mix"]), "n": rng.randint(3, 12),
                "layers": rng.randint(1, 6), "shots": _log_int(rng, 50, 3000)}
    if kind == "sv":
        circuit = rng.choice(["ansatz", "mix", "dense"])
        n = rng.randint(13, 27)
        return {"kind": kind, "circuit": circuit, "n": n, "layers": rng.randint(8, 30) if circuit == "mix" else rng.randint(2, 8),
                "shots": _log_int(rng, 100, 20000)}
    if kind == "sv64":
        circuit = rng.choice(["ansatz", "mix", "dense"])
        return {"kind": kind, "circuit": circuit, "n": rng.randint(13, 26),
                "layers": rng.randint(8, 30) if circuit == "mix" else rng.randint(2, 8), "shots": 0}
    if kind == "dm":
        return {"kind": kind, "mode": rng.choice(["reference", "physical"]), "n": rng.randint(3, 12), "layers": rng.randint(1, 4)}
    if kind == "grad":
        return {"kind": kind, "precision": rng.choice(["c128", "c64"]), "n": rng.randint(5, 21), "layers": rng.randint(1, 6),
                "terms": _log_int(rng, 4, 48)}
    if kind == "batch":
        lo = rng.randint(4, 14)
        precision = rng.choice(["c64", "c128"])
        return {"kind": kind, "precision": precision, "circuits": _log_int(rng, 4, 40), "lo": lo,
                "hi": rng.randint(lo + 1, 21), "layers": rng.randint(10, 40), "shots": _log_int(rng, 50, 1000) if precision == "c128" else 0}
    return {"kind": kind, "n": rng.randint(13, 26), "terms": _log_int(rng, 2, 16), "shots": _log_int(rng, 100, 100000)}


# ------------------------------------------------------------------ circuits as plain lists
# (name, qubits, parameter): "u" carries a 2x2 matrix, rotations an angle, channels a probability.


def _haar(rng):
    a = rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2))
    q, r = np.linalg.qr(a)
    q = q * (np.diag(r) / np.abs(np.diag(r)))
    return q / np.sqrt(np.linalg.det(q))


def _ghz(rng, n):
    return [("h", (0,), None)] + [("cnot", (0, k), None) for k in range(1, n)] + [("rz", (n - 1,), float(rng.uniform(-np.pi, np.pi)))] + \
        [("ry", (0,), float(rng.uniform(-np.pi, np.pi)))]


def _ansatz(rng, n, layers):
    ops = []
    for _ in range(layers):
        for q in range(n):
            ops.append(("ry", (q,), float(rng.uniform(-np.pi, np.pi))))
            ops.append(("rz", (q,), float(rng.uniform(-np.pi, np.pi))))
        for q in range(n if n > 2 else n - 1):
            ops.append(("cnot", (q, (q + 1) % n), None))
    return ops


def _dense(rng, n, layers):
    """Half of the layers with CZ on an alternating brick, half with CZ at strides 1, 8, 16."""
    ops = []
    for layer in range(layers):
        ops += [("u", (q,), _haar(rng)) for q in range(n)]
        if layer < (layers + 1) // 2:
            ops += [("cz", (q, q + 1), None) for q in range(layer % 2, n - 1, 2)]
        else:
            s, used = (1, 8, 16)[layer % 3], set()
            for q in range(n):
                r = (q + s) % n
                if q != r and q not in used and r not in used:
                    used.update((q, r))
                    ops.append(("cz", (q, r), None))
    return ops


def _mix(rng, n, layers):
    """ceil(n/2) gates a layer from {H, Rx, Ry, Rz, CNOT, CZ, Swap, CCNot} on random qubits, after
    one Ry on every qubit."""
    ops = [("ry", (q,), float(rng.uniform(-np.pi, np.pi))) for q in range(n)]
    for _ in range(layers * ((n + 1) // 2)):
        r = int(rng.integers(8))
        q = [int(x) for x in rng.choice(n, 3, replace=False)]
        name = ("h", "rx", "ry", "rz", "cnot", "cz", "swap", "ccnot")[r]
        k = (1, 1, 1, 1, 2, 2, 2, 3)[r]
        ops.append((name, tuple(q[:k]), float(rng.uniform(-np.pi, np.pi)) if r in (1, 2, 3) else None))
    return ops


def _noisy(rng, n, layers):
    ops = []
    for _ in range(layers):
        for q in range(n):
            ops.append((("rx", "ry", "rz")[rng.integers(3)], (q,), float(rng.uniform(0, 2 * np.pi))))
            ops += [("depolarizing", (q,), 1e-3), ("damping", (q,), 5e-3)]
        for q in range(n - 1):
            ops += [("cnot", (q, q + 1), None), ("depolarizing2", (q, q + 1), 1e-2), ("damping", (q,), 5e-3), ("damping", (q + 1,), 5e-3)]
    return ops


def _variational(rng, n, layers):
    ops = []
    for _ in range(layers):
        for q in range(n):
            ops.append(("ry", (q,), float(rng.uniform(-np.pi, np.pi))))
            ops.append(("rz", (q,), float(rng.uniform(-np.pi, np.pi))))
        for q in range(n):
            ops.append(("zz", (q, (q + 1) % n), float(rng.uniform(-np.pi, np.pi))))
    return ops


def _paulis(rng, n, terms):
    out = []
    for _ in range(terms):
        qs = rng.choice(n, int(rng.integers(1, min(4, n) + 1)), replace=False)
        out.append({int(q): "XYZ"[rng.integers(3)] for q in qs})
    return out


def _dm_terms(qubits):
    """X on all of the qubits, Z on the first, Z on the first two."""
    return [{q: "X" for q in qubits}, {qubits[0]: "Z"}, {q: "Z" for q in qubits[:2]}]


def _circuit(rng, case):
    c = case["circuit"]
    if c == "ghz":
        return _ghz(rng, case["n"])
    return {"ansatz": _ansatz, "dense": _dense, "mix": _mix}[c](rng, case["n"], case["layers"])


def _plan(case, seed):
    """Everything random of a case, as plain data."""
    rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, 20])
    kind = case["kind"]
    p = {}
    if kind in ("run", "sv", "sv64"):
        p["ops"] = _circuit(rng, case)
        p["paulis"] = _paulis(rng, case["n"], 8)
        p["seed"] = int(rng.integers(1 << 30))
    elif kind == "dm":
        p["ops"] = _noisy(rng, case["n"], case["layers"])
        p["x"] = sorted(int(q) for q in rng.choice(case["n"], min(4, case["n"]), replace=False))
    elif kind == "grad":
        p["ops"] = _variational(rng, case["n"], case["layers"])
        p["h"] = [(float(rng.normal()), t) for t in _paulis(rng, case["n"], case["terms"])]
    elif kind == "batch":
        p["n"] = [case["lo"] + (case["hi"] - case["lo"]) * i // max(1, case["circuits"] - 1) for i in range(case["circuits"])]
        p["circuits"] = [_mix(rng, n, max(4, case["layers"] - int(rng.integers(case["layers"] // 2 + 1)))) for n in p["n"]]
        p["obs"] = [_paulis(rng, n, 8) for n in p["n"]]
        p["seed"] = int(rng.integers(1 << 30))
    else:
        p["ops"] = _dense(rng, case["n"], 2)
        p["paulis"] = _paulis(rng, case["n"], case["terms"])
        p["seed"] = int(rng.integers(1 << 30))
        p["marginal"] = sorted(int(q) for q in rng.choice(case["n"], 8, replace=False))
    return p


# ------------------------------------------------------------------ the framework's side


def _instruction(op):
    bs = _package()
    name, q, v = op
    if name == "u":
        g = bs.Unitary(v)
    elif name in ("rx", "ry", "rz", "zz"):
        g = {"rx": bs.Rx, "ry": bs.Ry, "rz": bs.Rz, "zz": bs.ZZ}[name](v)
    elif name == "depolarizing":
        g = bs.Depolarizing(v)
    elif name == "damping":
        g = bs.AmplitudeDamping(v)
    elif name == "depolarizing2":
        g = bs.TwoQubitDepolarizing(v)
    else:
        g = {"h": bs.H, "cnot": bs.CNot, "cz": bs.CZ, "swap": bs.Swap, "ccnot": bs.CCNot}[name]()
    return bs.Instruction(g, list(q))


def _observable(term):
    o = _package().observables
    qs = sorted(term)
    return o.TensorProduct([{"X": o.X, "Y": o.Y, "Z": o.Z}[term[q]]() for q in qs]), qs


def prepare(case, seed):
    bs = _package()
    p = _plan(case, seed)
    kind = case["kind"]
    s = {"case": dict(case)}
    if kind == "run":
        s["ops"] = [_instruction(o) for o in p["ops"]]
        s["seed"] = p["seed"]
        s["sim"] = bs.StateVectorSimulator(case["n"], case["shots"])
    elif kind in ("sv", "sv64"):
        s["ops"] = [_instruction(o) for o in p["ops"]]
        s["obs"] = [_observable(t) for t in p["paulis"]]
        s["seed"] = p["seed"]
        s["sim"] = bs.StateVectorSimulator(case["n"], case["shots"], precision="c64" if kind == "sv64" else "c128")
    elif kind == "dm":
        s["ops"] = [_instruction(o) for o in p["ops"]]
        s["obs"] = [_observable(t) for t in _dm_terms(p["x"])]
        s["sim"] = bs.DensityMatrixSimulator(case["n"], 0, noise_mode=case["mode"])
    elif kind == "grad":
        s["h"] = p["h"]
        s["sim"] = bs.StateVectorSimulator(case["n"], 0, precision=case["precision"])
        if case["precision"] == "c64":
            plain = [(name, q) for name, q, _ in p["ops"]]
            s["energy"] = bs.torch_energy(lambda th: [_instruction((name, q, float(v))) for (name, q), v in zip(plain, th)], p["h"], s["sim"])
            s["theta"] = torch.tensor([v for _, _, v in p["ops"]], dtype=torch.float32, requires_grad=True)
        else:
            s["ops"] = [_instruction(o) for o in p["ops"]]
    elif kind == "batch":
        s["circuits"] = [[_instruction(o) for o in c] for c in p["circuits"]]
        s["n"], s["obs"], s["seed"] = p["n"], p["obs"], p["seed"]
    else:
        s["sim"] = bs.StateVectorSimulator(case["n"], case["shots"])
        s["sim"].evolve([_instruction(o) for o in p["ops"]])
        s["obs"] = [_observable(t) for t in p["paulis"]]
        s["seed"], s["marginal"] = p["seed"], p["marginal"]
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "run":
        p, shots = s["sim"].run(s["ops"], case["shots"], seed=s["seed"])
        return {"probabilities": p, "shots": shots}
    if kind in ("sv", "sv64"):
        sim = s["sim"]
        sim.reinit(case["n"], case["shots"])
        sim.evolve(s["ops"])
        values = [sim.expectation(o, *q) for o, q in s["obs"]]
        if kind == "sv64":
            return {"expectations": np.array(values, dtype=np.float32)}
        out = {"expectations": np.array(values), "shots": sim.samples(s["seed"])}
        if case["n"] <= 20:
            out["probabilities"] = sim.probabilities()
        return out
    if kind == "dm":
        sim = s["sim"]
        sim.reinit(case["n"], 0)
        sim.evolve(s["ops"])
        return {"probabilities": sim.probabilities(), "expectations": np.array([sim.expectation(o, *q) for o, q in s["obs"]])}
    if kind == "grad":
        if case["precision"] == "c64":
            s["theta"].grad = None
            e = s["energy"](s["theta"])
            e.backward()
            return {"energy": e.detach(), "gradient": s["theta"].grad}
        e, g = _package().adjoint_gradient(s["sim"], s["ops"], s["h"])
        return {"energy": np.array([e]), "gradient": g}
    if kind == "batch":
        values, shots, _ = _package().batch_simulate(s["circuits"], s["n"], s["obs"], shots=case["shots"], seed=s["seed"], precision=case["precision"])
        if case["precision"] == "c64":
            return {"expectations": values.astype(np.float32)}
        return {"expectations": values, "shots": shots}
    sim = s["sim"]
    return {"expectations": np.array([sim.expectation(o, *q) for o, q in s["obs"]]),
            "marginal": sim.marginal_probabilities(s["marginal"]), "shots": sim.samples(s["seed"])}


# ------------------------------------------------------------------ what a pass cannot do without

_FLOPS_PER_AMPLITUDE = {"u": 14, "h": 4, "rx": 8, "ry": 6, "rz": 6, "zz": 6, "cnot": 0, "cz": 0.5, "swap": 0, "ccnot": 0}


def _gate_flops(ops, amplitudes):
    return float(amplitudes) * sum(_FLOPS_PER_AMPLITUDE.get(name, 0) for name, _, _ in ops)


def work(case):
    """Bytes: the state written once by the evolution and read once by the readouts, results written.
    Flops: the real operations of the gates as the circuit lists them, on every amplitude."""
    kind = case["kind"]
    p = _plan(case, 1)
    if kind == "batch":
        el = 8 if case["precision"] == "c64" else 16
        return {"bytes": float(sum(2 * el * 2 ** n for n in p["n"])) + 8.0 * case["shots"] * len(p["n"]) + 64.0 * len(p["n"]),
                "flops": float(sum(_gate_flops(c, 2 ** n) for c, n in zip(p["circuits"], p["n"])))}
    n = case["n"]
    if kind == "dm":
        # 4^n elements; gates act from both sides, each channel's superoperator on its targets
        flops = 2 * _gate_flops(p["ops"], 4 ** n)
        if case["mode"] == "physical":
            flops += 4.0 ** n * sum({"depolarizing": 4, "damping": 4, "depolarizing2": 8}.get(name, 0) for name, _, _ in p["ops"])
        return {"bytes": 16.0 * 4 ** n + 3 * 16.0 * 2 ** n, "flops": flops}
    if kind == "grad":
        el = 8 if case["precision"] == "c64" else 16
        # forward state, then both states of the reverse sweep; a gate and an inner product per parameter
        return {"bytes": 4.0 * el * 2 ** n + 8.0 * len(p["ops"]), "flops": 3 * _gate_flops(p["ops"], 2 ** n) + 4.0 * len(p["ops"]) * 2 ** n +
                8.0 * case["terms"] * 2 ** n}
    if kind == "readout":
        return {"bytes": 16.0 * 2 ** n + 8.0 * (case["shots"] + 256), "flops": 2.0 ** n * (4.0 * case["terms"] + 4)}
    el = 8 if kind == "sv64" else 16
    out = 8.0 * case["shots"] + (8.0 * 2 ** n if kind == "run" or (kind == "sv" and n <= 20) else 64)
    return {"bytes": 2.0 * el * 2 ** n + out, "flops": _gate_flops(p["ops"], 2 ** n)}


# ------------------------------------------------------------------ the same in 64 bits, without the package


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _matrix(name, v):
    if name == "u":
        return np.asarray(v, dtype=np.complex128)
    if name == "h":
        return np.array([[1, 1], [1, -1]], dtype=np.complex128) / math.sqrt(2)
    c, s = math.cos(v / 2), math.sin(v / 2)
    if name == "rx":
        return np.array([[c, -1j * s], [-1j * s, c]])
    if name == "ry":
        return np.array([[c, -s], [s, c]], dtype=np.complex128)
    return np.array([[c - 1j * s, 0], [0, c + 1j * s]])


def _dense_bit(x, m, bit):
    """A 2x2 matrix on index bit `bit` of the flat vector x, in place."""
    w = x.view(-1, 2, 1 << bit)
    a, b = w[:, 0].clone(), w[:, 1].clone()
    w[:, 0] = complex(m[0, 0]) * a + complex(m[0, 1]) * b
    w[:, 1] = complex(m[1, 0]) * a + complex(m[1, 1]) * b


def _bits_view(x, bits):
    """x viewed with one axis of length 2 per bit (descending) between the blocks in between."""
    shape, top = [], int(x.numel()).bit_length() - 1
    for b in bits:
        shape += [1 << (top - b - 1), 2]
        top = b
    return x.view(shape + [1 << top])


def _axis_index(bits, values):
    ix = []
    for b in bits:
        ix += [slice(None), values[b]]
    return tuple(ix)


def _apply(x, op, bit_of, conj=False):
    """One gate on the flat vector x; bit_of[q] is the index bit of qubit q."""
    name, q, v = op
    if name in ("u", "h", "rx", "ry", "rz"):
        m = _matrix(name, v)
        _dense_bit(x, np.conj(m) if conj else m, bit_of[q[0]])
        return
    bits = sorted((bit_of[t] for t in q), reverse=True)
    w = _bits_view(x, bits)
    b = [bit_of[t] for t in q]
    if name == "cz":
        w[_axis_index(bits, {b[0]: 1, b[1]: 1})] *= -1
    elif name == "zz":
        ph = complex(math.cos(v / 2), math.sin(v / 2) if conj else -math.sin(v / 2))
        for i in (0, 1):
            for j in (0, 1):
                w[_axis_index(bits, {b[0]: i, b[1]: j})] *= ph if i == j else ph.conjugate()
    else:
        if name == "swap":
            one, two = {b[0]: 0, b[1]: 1}, {b[0]: 1, b[1]: 0}
        else:
            c = {t: 1 for t in b[:-1]}
            one, two = {**c, b[-1]: 0}, {**c, b[-1]: 1}
        one, two = _axis_index(bits, one), _axis_index(bits, two)
        t = w[one].clone()
        w[one] = w[two]
        w[two] = t


def _state(ops, n):
    x = torch.zeros(1 << n, dtype=torch.complex128, device=_device())
    x[0] = 1
    for op in ops:
        _apply(x, op, [n - 1 - q for q in range(n)])
    return x


def _pauli_applied(x, term, n):
    y = x
    for q, c in term.items():
        w = y.view(-1, 2, 1 << (n - 1 - q))
        if c == "X":
            w = w.flip(1)
        elif c == "Y":
            w = w.flip(1) * torch.tensor([-1j, 1j], dtype=x.dtype, device=x.device).view(1, 2, 1)
        else:
            w = w * torch.tensor([1.0, -1.0], dtype=torch.float64, device=x.device).view(1, 2, 1)
        y = w.reshape(-1)
    return y


def _expect(x, term, n):
    return float(torch.vdot(x, _pauli_applied(x, term, n)).real)


def _exact_gradient(p, n):
    ops, h = p["ops"], p["h"]
    bit_of = [n - 1 - q for q in range(n)]
    psi = _state(ops, n)
    lam = torch.zeros_like(psi)
    for c, t in h:
        lam += c * _pauli_applied(psi, t, n)
    e = float(torch.vdot(psi, lam).real)
    g = np.zeros(len(ops))
    gen = {"ry": "Y", "rz": "Z", "zz": "Z"}
    for i in range(len(ops) - 1, -1, -1):
        name, q, v = ops[i]
        g[i] = float(torch.vdot(lam, _pauli_applied(psi, {t: gen[name] for t in q}, n)).imag)
        for x in (psi, lam):
            _apply(x, (name, q, -v), bit_of)
    return e, g


_PAULI = [np.eye(2), np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), np.diag([1.0, -1.0])]


def _kraus(name, v):
    if name == "depolarizing":
        return [math.sqrt(1 - v if i == 0 else v / 3) * m.astype(np.complex128) for i, m in enumerate(_PAULI)]
    if name == "damping":
        return [np.array([[1, 0], [0, math.sqrt(1 - v)]], dtype=np.complex128), np.array([[0, math.sqrt(v)], [0, 0]], dtype=np.complex128)]
    return [math.sqrt(1 - v if i + j == 0 else v / 15) * np.kron(a, b).astype(np.complex128) for i, a in enumerate(_PAULI) for j, b in enumerate(_PAULI)]


def _channel(S, op, n, mode):
    """The channel's superoperator on the target rows and columns of the stored matrix (which holds the
    transpose of rho): every block, or (the reference's rule) the blocks whose row and column share all
    other bits, updated as K B K^dagger."""
    name, q, v = op
    d = 1 << len(q)
    bits = [n - 1 - t for t in reversed(q)]      # matrix bit j <-> bits[j], first target most significant
    rest = torch.arange(1 << (n - len(q)), device=S.device)
    for b in sorted(bits):
        rest = ((rest >> b) << (b + 1)) | (rest & ((1 << b) - 1))
    idx = [rest + sum(((i >> j) & 1) << b for j, b in enumerate(bits)) for i in range(d)]
    ks = _kraus(name, v)
    M = S.view(1 << n, 1 << n)                   # M[column, row] of the stored matrix
    sup = sum(np.kron(k, np.conj(k)) if mode == "reference" else np.kron(np.conj(k), k) for k in ks)   # (row, column) pairs
    if mode == "reference":
        old = torch.stack([M[idx[j], idx[i]] for i in range(d) for j in range(d)])
        new = torch.as_tensor(sup, device=S.device) @ old
        for i in range(d):
            for j in range(d):
                M[idx[j], idx[i]] = new[i * d + j]
        return
    # all blocks: one column-index set at a time, kept small
    for r in torch.arange(rest.numel(), device=S.device).split(max(1, (1 << 24) // (d * d * rest.numel()) or 1)):
        old = torch.stack([M[idx[j][r]][:, idx[i]] for i in range(d) for j in range(d)])
        new = (torch.as_tensor(sup, device=S.device) @ old.reshape(d * d, -1)).view(old.shape)
        for i in range(d):
            for j in range(d):
                M[idx[j][r][:, None], idx[i][None, :]] = new[i * d + j]


def _exact_dm(p, n, mode):
    S = torch.zeros(1 << (2 * n), dtype=torch.complex128, device=_device())
    S[0] = 1
    for op in p["ops"]:
        if op[0] in ("depolarizing", "damping", "depolarizing2"):
            _channel(S, op, n, mode)
        else:
            _apply(S, op, [2 * n - 1 - q for q in range(n)])
            _apply(S, op, [n - 1 - q for q in range(n)], conj=True)
    M = S.view(1 << n, 1 << n)
    a = torch.arange(1 << n, device=S.device)
    prob, values = M[a, a].real, []
    for t in _dm_terms(p["x"]):
        if "X" in t.values():
            values.append(float(M[a ^ sum(1 << (n - 1 - q) for q in t), a].real.sum()))
        else:
            sign = torch.ones_like(prob)
            for q in t:
                sign = sign * (1 - 2 * ((a >> (n - 1 - q)) & 1))
            values.append(float((sign * prob).sum()))
    return prob, np.array(values)


def exact(case, seed):
    kind = case["kind"]
    p = _plan(case, seed)
    if kind == "dm":
        if case["mode"] == "physical" and case["n"] > 12 or case["n"] > 13:
            return None
        prob, ex = _exact_dm(p, case["n"], case["mode"])
        return {"probabilities": prob.cpu().numpy(), "expectations": ex}
    if kind == "grad":
        e, g = _exact_gradient(p, case["n"])
        if case["precision"] == "c64":
            # the parameters as the program holds them, in float32
            q = dict(p, ops=[(name, t, float(np.float32(v))) for name, t, v in p["ops"]])
            e, g = _exact_gradient(q, case["n"])
            return {"energy": np.float64(e), "gradient": g}
        return {"energy": np.array([e]), "gradient": g}
    if kind == "batch":
        values = np.zeros((len(p["n"]), 8))
        for i, (c, n) in enumerate(zip(p["circuits"], p["n"])):
            x = _state(c, n)
            values[i] = [_expect(x, t, n) for t in p["obs"][i]]
        return {"expectations": values} if case["precision"] == "c64" else {"expectations": values, "shots": None}
    n = case["n"]
    x = _state(p["ops"], n)
    if kind == "run":
        return {"probabilities": (x.real ** 2 + x.imag ** 2).cpu().numpy(), "shots": None}
    out = {"expectations": np.array([_expect(x, t, n) for t in p["paulis"]])}
    if kind == "sv64":
        return out
    out["shots"] = None
    if kind == "sv" and n <= 20:
        out["probabilities"] = (x.real ** 2 + x.imag ** 2).cpu().numpy()
    if kind == "readout":
        w = x.real ** 2 + x.imag ** 2
        for q in range(n - 1, -1, -1):           # qubit q is index bit n-1-q; summed bits go from the low end
            if q not in p["marginal"]:
                low = sum(1 for t in p["marginal"] if t > q)
                w = w.view(-1, 2, 1 << low).sum(1).reshape(-1)
        out["marginal"] = w.cpu().numpy()
    return out
