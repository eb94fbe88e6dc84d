"""Fused 5-qubit unitaries on the tcgen05 tensor cores (exact bf16 digit split):
parity with the FP64 oracle at 1e-12 relative, against the float-float path, and
on the edge cases of the per-column scaling (zero columns, wide dynamic range,
unnormalised states)."""
import os

import numpy as np
import pytest

import oracle
from conftest import bs, random_circuit, rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-12


class tc_mode:
    """BS_TC=0 keeps every gate on the float-float tile path; BS_TC_MIN_BITS lowers the state size
    from which fused tensor-core sweeps are used (22 vector bits by default) so that oracle-sized
    cases exercise them.  Both are read on every evolve."""

    def __init__(self, on):
        self.on = on

    def __enter__(self):
        self.old = {k: os.environ.get(k) for k in ("BS_TC", "BS_TC_MIN_BITS")}
        os.environ["BS_TC"] = "1" if self.on else "0"
        os.environ["BS_TC_MIN_BITS"] = "12"

    def __exit__(self, *a):
        for k, v in self.old.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v


def haar(rng, d=2):
    a = rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d))
    q, r = np.linalg.qr(a)
    return q * (np.diag(r) / np.abs(np.diag(r)))


def brick(n, layers, rng):
    ops = []
    for layer in range(layers):
        for q in range(n):
            ops.append(bs.Instruction(bs.Unitary(haar(rng)), [q]))
        for q in range(layer % 2, n - 1, 2):
            ops.append(bs.Instruction(bs.CZ() if layer % 3 else bs.CNot(), [q, q + 1]))
    return ops


@pytest.mark.parametrize("n", [12, 14, 17, 20])
def test_brick_layers_fuse_onto_tensor_cores(n):
    rng = np.random.default_rng(500 + n)
    ops = brick(n, 10, rng)
    ref = oracle.OracleSV(n).evolve(ops).psi
    with tc_mode(True):
        sim = bs.StateVectorSimulator(n, 0).evolve(ops)
        st = sim.last_stats()
        got = sim.state_vector
    assert st["tc_gates"] > 0
    assert rel_err(got, ref) < TOL
    with tc_mode(False):
        sim0 = bs.StateVectorSimulator(n, 0).evolve(ops)
        assert sim0.last_stats()["tc_gates"] == 0
        assert rel_err(sim0.state_vector, ref) < TOL


@pytest.mark.parametrize("n", [12, 13, 16])
@pytest.mark.parametrize("pows", [False, True])
def test_random_gate_families(n, pows):
    rng = np.random.default_rng(900 + 10 * n + pows)
    ops = random_circuit(n, 300, rng, pows=pows)
    ref = oracle.OracleSV(n).evolve(ops).psi
    with tc_mode(True):
        sim = bs.StateVectorSimulator(n, 0).evolve(ops)
        assert sim.last_stats()["tc_gates"] > 0
        assert rel_err(sim.state_vector, ref) < TOL


def test_zero_columns_from_basis_state():
    # gates on three qubits of |0...0>: almost every column of every tile is zero
    n = 14
    rng = np.random.default_rng(3)
    ops = []
    for _ in range(8):
        for q in (0, 5, 13):
            ops.append(bs.Instruction(bs.Unitary(haar(rng)), [q]))
        ops.append(bs.Instruction(bs.CNot(), [0, 5]))
        ops.append(bs.Instruction(bs.CZ(), [5, 13]))
    ref = oracle.OracleSV(n).evolve(ops).psi
    with tc_mode(True):
        sim = bs.StateVectorSimulator(n, 0).evolve(ops)
        assert rel_err(sim.state_vector, ref) < TOL


@pytest.mark.parametrize("scale", [1.0, 1e3, 1e-9])
def test_wide_dynamic_range_and_unnormalised_states(scale):
    n = 13
    rng = np.random.default_rng(11)
    mag = 10.0 ** rng.uniform(-18, 0, size=2 ** n)
    psi0 = mag * np.exp(2j * np.pi * rng.random(2 ** n))
    psi0 = scale * psi0 / np.linalg.norm(psi0)
    ops = brick(n, 6, rng)
    o = oracle.OracleSV(n)
    o.psi = psi0.copy()
    ref = o.evolve(ops).psi
    with tc_mode(True):
        sim = bs.StateVectorSimulator(n, 0)
        sim.state_vector = psi0
        sim.evolve(ops)
        assert sim.last_stats()["tc_gates"] > 0
        assert rel_err(sim.state_vector, ref) < TOL


def test_inverse_roundtrip_through_fused_gates():
    n = 15
    rng = np.random.default_rng(21)
    ops = brick(n, 8, rng)
    inv = [bs.Instruction(ix.operator.inv(), ix.target) for ix in reversed(ops)]
    with tc_mode(True):
        sim = bs.StateVectorSimulator(n, 0).evolve(ops + inv)
        psi = sim.state_vector
    e0 = np.zeros(2 ** n, complex)
    e0[0] = 1
    assert rel_err(psi, e0) < TOL


@pytest.mark.parametrize("n", [6, 7])
@pytest.mark.parametrize("mode", ["reference", "physical"])
def test_density_matrix_with_noise(n, mode):
    rng = np.random.default_rng(40 + n)
    ops = []
    for layer in range(6):
        for q in range(n):
            ops.append(bs.Instruction(bs.Unitary(haar(rng)), [q]))
            if rng.random() < 0.5:
                ops.append(bs.Instruction(bs.Depolarizing(0.01), [q]))
        for q in range(layer % 2, n - 1, 2):
            ops.append(bs.Instruction(bs.CNot(), [q, q + 1]))
            if rng.random() < 0.5:
                ops.append(bs.Instruction(bs.AmplitudeDamping(0.05), [q + 1]))
    ref = oracle.OracleDM(n, physical=(mode == "physical")).evolve(ops).matrix
    with tc_mode(True):
        sim = bs.DensityMatrixSimulator(n, 0, noise_mode=mode).evolve(ops)
        if mode == "physical":
            # channels are superoperator tile gates and fuse; in reference mode the reference-compatible
            # Kraus kernel runs between sweeps and leaves runs too short to be worth fusing
            assert sim.last_stats()["tc_gates"] > 0
        assert rel_err(sim.density_matrix, ref) < TOL


@pytest.mark.parametrize("n", [13, 15])
@pytest.mark.parametrize("low", [False, True])
def test_fused_products_of_every_gate_form(n, low):
    """Blocks of gates of all forms (dense on 1 to 4 targets, real and complex, singular and scaled; diagonal and
    monomial; controls on either value), with targets and controls inside the block and outside the tile."""
    rng = np.random.default_rng(77 + n)
    near = list(range(n - 5, n)) if low else list(range(5))   # 5 bits of one block
    far = [q for q in range(n) if q not in near]
    ops = [bs.Instruction(bs.Unitary(haar(rng)), [q]) for q in range(n)]
    for _ in range(12):
        p = [int(q) for q in rng.permutation(near)]
        f = [int(q) for q in rng.choice(far, 2, replace=False)]
        ops += [bs.Instruction(bs.Unitary(haar(rng, 4)), p[:2]), bs.Instruction(bs.Unitary(haar(rng, 8)), p[1:4]),
                bs.Instruction(bs.Unitary(haar(rng, 16)), p[:4]), bs.Instruction(bs.Ry(0.3), [p[4]]),
                bs.Instruction(bs.Control(bs.U(0.4, 0.2, -0.7), (0, 1)), [p[0], f[0], p[1]]),
                bs.Instruction(bs.Control(bs.PhaseShift(0.9), (1, 0)), [f[0], p[2], p[3]]),
                bs.Instruction(bs.ZZ(0.7), [p[0], f[1]]), bs.Instruction(bs.CPhaseShift(1.1), [f[1], p[1]]),
                bs.Instruction(bs.CSwap(), [p[2], p[3], p[4]]), bs.Instruction(bs.Control(bs.Y(), (0,)), [f[1], p[0]]),
                bs.Instruction(bs.ISwap(), [p[1], p[4]]),
                bs.Instruction(bs.Unitary(2.0 * haar(rng)), [p[2]]), bs.Instruction(bs.Unitary(0.5 * haar(rng)), [p[3]])]
    ref = oracle.OracleSV(n).evolve(ops).psi
    with tc_mode(True):
        sim = bs.StateVectorSimulator(n, 0).evolve(ops)
        assert sim.last_stats()["tc_gates"] > 0
        assert rel_err(sim.state_vector, ref) < TOL


@pytest.mark.parametrize("factor,ok", [(15.0, True), (17.0, False)])
def test_fused_matrix_entries_reach_4096(factor, ok):
    """Matrices up to 2^12 are applied (15^3 = 3375); above it (17^3 = 4913) the list is refused, whatever the bound
    from the gates' norms says (a gate between them has norm 4)."""
    n = 13
    s = np.array([[factor, 0], [0, 0.25]])
    g = np.array([[1.0, 0], [0, 4.0]])
    ops = [bs.Instruction(bs.Unitary(m), [2]) for m in (s, g, s, g, s)] + [bs.Instruction(bs.Ry(0.1), [q]) for q in (3, 4, 5)]
    with tc_mode(True):
        sim = bs.StateVectorSimulator(n, 0)
        if ok:
            sim.evolve(ops)
            assert sim.last_stats()["tc_gates"] > 0
            assert rel_err(sim.state_vector, oracle.OracleSV(n).evolve(ops).psi) < TOL
        else:
            with pytest.raises(Exception, match="out of range"):
                sim.evolve(ops)


@pytest.mark.parametrize("n", [18, 19, 21, 22, 23, 24, 25])
@pytest.mark.parametrize("ring", [False, True])
def test_rows_of_a_tile_by_size(n, ring):
    """Tiles take 5, 4 or 3 low bits by the vector's size and the plan's cost: the state against tiles of 2^11 with 5
    low bits on the float-float path (double-double sums of about 300 gates: 1e-12 relative)."""
    rng = np.random.default_rng(300 + n)
    ops = brick(n, 3, rng)
    for layer in range(3):
        for q in range(n):
            ops.append(bs.Instruction(bs.Ry(float(rng.uniform(-3, 3))), [q]))
            ops.append(bs.Instruction(bs.CNot() if ring else bs.CPhaseShift(0.4), [q, (q + (1 if ring else 7)) % n]))
    sim = bs.StateVectorSimulator(n, 0).evolve(ops)
    assert (sim.last_stats()["tc_gates"] > 0) == (n >= 20)   # 3 layers of generic matrices
    ref = bs.StateVectorSimulator(n, 0)
    bs.set_tuning(ref, tile_bits=11, tc=0)
    ref.evolve(ops)
    assert rel_err(sim.state_vector, ref.state_vector) < TOL


@pytest.mark.parametrize("n,kind,wide,layers,tc", [(19, "sv", 0, 3, False), (20, "sv", 0, 2, True), (20, "sv", 0, 1, False),
                                                   (16, "sv", 2, 0, False), (16, "sv", 3, 0, True), (15, "sv", 3, 0, False),
                                                   (20, "real", 0, 3, False), (8, "dm", 3, 0, True), (8, "dm", 2, 0, False)])
def test_lists_below_22_bits(n, kind, wide, layers, tc):
    """Which lists run on the tensor cores below 22 bits: generic one-qubit matrices from 20 bits, gates on 4 targets
    (and two-qubit channels) from 16, real rotations not; the states against the oracle."""
    rng = np.random.default_rng(60 + n)
    ops = [bs.Instruction(bs.H(), [q]) for q in range(n)]
    for _ in range(layers):
        ops += [bs.Instruction(bs.Ry(float(rng.uniform(-3, 3))) if kind == "real" else bs.Unitary(haar(rng)), [q]) for q in range(n)]
        ops += [bs.Instruction(bs.CZ(), [q, q + 1]) for q in range(n - 1)]
    for i in range(wide):
        q = [int(x) for x in rng.permutation(n)[:4]]
        ops.append(bs.Instruction(bs.TwoQubitDepolarizing(0.02), q[:2]) if kind == "dm" else bs.Instruction(bs.Unitary(haar(rng, 16)), q))
        ops.append(bs.Instruction(bs.CNot(), q[2:]))
    if kind == "dm":
        sim = bs.DensityMatrixSimulator(n, 0, noise_mode="physical").evolve(ops)
        got, ref = sim.density_matrix, oracle.OracleDM(n, physical=True).evolve(ops).matrix
    else:
        sim = bs.StateVectorSimulator(n, 0).evolve(ops)
        got, ref = sim.state_vector, oracle.OracleSV(n).evolve(ops).psi
    assert (sim.last_stats()["tc_gates"] > 0) == tc
    assert rel_err(got, ref) < TOL


@pytest.mark.parametrize("n,kind,tune", [(13, "sv", True), (16, "sv", False), (20, "sv", False), (22, "sv", False), (8, "dm", False)])
@pytest.mark.parametrize("same", [True, False])
def test_products_out_of_range_run_on_the_float_float_sweeps(n, kind, tune, same):
    """Lists that take the tensor cores by their size, gates or tuning and whose fused product has entries of 2^12 and
    more: matrices of norm 17 six times on one qubit, or twice on each of five.  The sweep that holds them runs
    float-float, the others stay fused; the state against the oracle."""
    rng = np.random.default_rng(800 + n)
    big = np.array([[17.0, 0.3], [0.2, 0.25]])
    ops = [bs.Instruction(bs.Unitary(haar(rng)), [q]) for q in range(n) for _ in range(1 + 2 * (n >= 20))]
    for layer in range(2):
        ops += [bs.Instruction(bs.CZ(), [q, q + 1]) for q in range(n - 1)]
        ops += [bs.Instruction(bs.Unitary(haar(rng)), [q]) for q in range(n)]
        for _ in range(2 if n < 20 and kind == "sv" else 0):
            ops.append(bs.Instruction(bs.Unitary(haar(rng, 16)), [int(q) for q in rng.permutation(n)[:4]]))
    if kind == "dm":
        ops += [bs.Instruction(bs.TwoQubitDepolarizing(0.02), [int(q) for q in rng.permutation(n)[:2]]) for _ in range(4)]
    ops += [bs.Instruction(bs.Unitary(big), [2])] * 6 if same else [bs.Instruction(bs.Unitary(big), [q]) for q in range(5)] * 2
    ops += [bs.Instruction(bs.Ry(0.1), [q]) for q in (3, 4, 5)]
    if kind == "dm":
        sim = bs.DensityMatrixSimulator(n, 0, noise_mode="physical").evolve(ops)
        got, ref = sim.density_matrix, oracle.OracleDM(n, physical=True).evolve(ops).matrix
    else:
        sim = bs.StateVectorSimulator(n, 0)
        if tune:
            bs.set_tuning(sim, tc_min_bits=12)
        got, ref = sim.evolve(ops).state_vector, oracle.OracleSV(n).evolve(ops).psi
    assert rel_err(got, ref) < TOL


@pytest.mark.parametrize("n,gates,tc", [(16, 6, False), (17, 12, False), (19, 24, False), (20, 12, True), (21, 3, False)])
def test_gates_on_three_targets_below_22_bits(n, gates, tc):
    """Lists of 3-target gates stay on the float-float sweeps below 20 bits, which are faster for them, and count as
    generic matrices from there (at least 40 units of a dense 1-qubit gate, 4 each); the states against the oracle."""
    rng = np.random.default_rng(90 + n)
    ops = [bs.Instruction(bs.H(), [q]) for q in range(n)]
    ops += [bs.Instruction(bs.Unitary(haar(rng, 8)), [int(x) for x in rng.permutation(n)[:3]]) for _ in range(gates)]
    sim = bs.StateVectorSimulator(n, 0).evolve(ops)
    assert (sim.last_stats()["tc_gates"] > 0) == tc
    assert rel_err(sim.state_vector, oracle.OracleSV(n).evolve(ops).psi) < TOL
