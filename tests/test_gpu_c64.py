"""complex64 states: FP32 gate arithmetic (error against the FP64 oracle is reported and
bounded), and FP64-accurate reductions on the stored complex64 values."""
import numpy as np
import pytest

import oracle
from conftest import bs, random_circuit, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 9, 14, 17])
def test_c64_random_circuits_within_fp32_error(n):
    rng = np.random.default_rng(500 + n)
    ops = random_circuit(n, 50, rng)
    sim = bs.StateVectorSimulator(n, 0, precision="c64").evolve(ops)
    ref = oracle.OracleSV(n).evolve(ops).psi
    err = rel_err(sim.state_vector, ref)
    # FP32 rounding per gate, accumulated over 50 gates
    assert err < 2e-5, err


def test_c64_dense_layers_and_fused_sweeps():
    n = 18
    rng = np.random.default_rng(9)
    ops = []
    for layer in range(8):
        for q in range(n):
            a = rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2))
            ops.append(bs.Instruction(bs.Unitary(np.linalg.qr(a)[0]), [q]))
        for q in range(layer % 2, n - 1, 2):
            ops.append(bs.Instruction(bs.CZ(), [q, q + 1]))
    sim = bs.StateVectorSimulator(n, 0, precision="c64").evolve(ops)
    err = rel_err(sim.state_vector, oracle.OracleSV(n).evolve(ops).psi)
    assert err < 2e-5, err


@pytest.mark.parametrize("mode", ["reference", "physical"])
def test_c64_noisy_density_matrix(mode):
    n = 5
    rng = np.random.default_rng(31)
    ops = []
    for ix in random_circuit(n, 25, rng):
        ops.append(ix)
        ops.append(bs.Instruction(bs.Depolarizing(0.05), [ix.target[0]]))
        ops.append(bs.Instruction(bs.AmplitudeDamping(0.02), [ix.target[-1]]))
    sim = bs.DensityMatrixSimulator(n, 0, noise_mode=mode, precision="c64").evolve(ops)
    ref = oracle.OracleDM(n, physical=(mode == "physical")).evolve(ops).matrix
    assert rel_err(sim.density_matrix, ref) < 2e-5


def test_c64_reductions_are_fp64_accurate_on_the_stored_values():
    n = 12
    rng = np.random.default_rng(4)
    ops = random_circuit(n, 40, rng)
    sim = bs.StateVectorSimulator(n, 0, precision="c64").evolve(ops)
    v = sim.state_vector                     # exact complex64 values, widened
    p = np.abs(v) ** 2
    assert rel_err(sim.probabilities(), p) < 1e-14
    for _ in range(6):
        x, z = int(rng.integers(0, 2 ** n)), int(rng.integers(0, 2 ** n))
        out = np.empty(1)
        sim._h.call("bs_expectation_pauli", 1, bs._abi.u64ptr(np.array([x], dtype=np.uint64)),
                    bs._abi.u64ptr(np.array([z], dtype=np.uint64)), bs._abi.dptr(np.ones(1)), bs._abi.dptr(out))
        assert abs(out[0] - oracle.expectation_pauli_sv(v.astype(np.complex128), n, x, z)) < 1e-13
    s = bs.StateVectorSimulator(n, 2000, precision="c64")
    s.state_vector = v
    u = rng.random(2000)
    got = s.samples_direct(u, wsum=float(np.sum(p)))
    assert np.sum(got != oracle.sample_direct(p, u, float(np.sum(p)))) <= 2


def test_c64_state_roundtrip_and_copy():
    v = (np.arange(256) + 1j * np.arange(256)[::-1]) / 3000.0
    s = bs.StateVectorSimulator(8, 0, precision="c64")
    s.state_vector = v
    assert np.allclose(s.state_vector, v.astype(np.complex64), rtol=0, atol=0)
    c = s.copy()
    assert np.array_equal(c.state_vector, s.state_vector)


def test_c64_runs_on_qubit_pairs_fold_into_two_bit_gates():
    """Complex64 sweeps fold runs of 1- and 2-qubit gates on the same two qubits (controls in the
    tile, or out of it) into dense 2-bit gates: same result as the oracle within FP32 error."""
    n = 16
    rng = np.random.default_rng(77)
    ops = []
    for _ in range(12):
        a, b = (int(x) for x in rng.choice(n, 2, replace=False))
        c = int(rng.integers(n))
        for ix in (bs.Instruction(bs.H(), [a]), bs.Instruction(bs.CNot(), [a, b]),
                   bs.Instruction(bs.Rz(float(rng.uniform(-3, 3))), [b]), bs.Instruction(bs.CZ(), [b, a]),
                   bs.Instruction(bs.Ry(float(rng.uniform(-3, 3))), [a]), bs.Instruction(bs.Swap(), [a, b]),
                   bs.Instruction(bs.Rx(float(rng.uniform(-3, 3))), [c])):
            ops.append(ix)
        if c not in (a, b):
            ops.append(bs.Instruction(bs.CCNot(), [c, a, b]))
    sim = bs.StateVectorSimulator(n, 0, precision="c64").evolve(ops)
    err = rel_err(sim.state_vector, oracle.OracleSV(n).evolve(ops).psi)
    assert err < 2e-5, err


def _block_circuit(n, gates, rng, kinds):
    """Gates of the register blocks' kinds on random qubits: one-target gates of every matrix class with
    any controls, swaps, diagonals on and off the block, and (kind "wide") gates that keep their pass."""
    ops, a = [], lambda: float(rng.uniform(-np.pi, np.pi))
    for _ in range(gates):
        q = [int(x) for x in rng.choice(n, min(n, 4), replace=False)]
        k = kinds[int(rng.integers(len(kinds)))]
        if k == "one":
            g = [bs.H(), bs.X(), bs.Y(), bs.Rx(a()), bs.Ry(a()), bs.Rz(a()), bs.S(), bs.U(a(), a(), a()), bs.V()][int(rng.integers(9))]
            ops.append(bs.Instruction(g, [q[0]]))
        elif k == "ctrl":
            g = [bs.X(), bs.Ry(a()), bs.U(a(), a(), a()), bs.Z()][int(rng.integers(4))]
            nc = int(rng.integers(1, 3))   # the oracle has kernels for up to two controls
            ops.append(bs.Instruction(bs.Control(g, tuple(int(b) for b in rng.integers(0, 2, nc))), q[:nc + 1]))
        elif k == "diag":
            g = [bs.CZ(), bs.ZZ(a()), bs.CPhaseShift(a()), bs.CPhaseShift01(a())][int(rng.integers(4))]
            ops.append(bs.Instruction(g, q[:2]))
        elif k == "swap":
            ops.append(bs.Instruction(bs.Swap(), q[:2]))
        else:
            g = [bs.XX(a()), bs.ISwap(), bs.FermionicSWAP(a())][int(rng.integers(3))]
            ops.append(bs.Instruction(g, q[:2]))
    return ops


@pytest.mark.parametrize("n,gates,kinds", [
    (12, 60, ("one", "ctrl", "diag", "swap")),       # one tile, every bit in it
    (13, 80, ("one", "ctrl", "diag", "swap")),       # one bit outside
    (17, 120, ("one", "ctrl", "diag", "swap")),
    (18, 90, ("one", "diag", "wide")),               # passes between blocks
    (16, 60, ("diag",)),                             # no moved bit at all
    (12, 400, ("one", "ctrl")),                      # more operations than are staged at a time
    (11, 60, ("one", "ctrl", "diag")),               # below a full tile: no blocks
])
def test_register_blocks_match_the_oracle(n, gates, kinds):
    rng = np.random.default_rng(7000 + n + gates)
    ops = [bs.Instruction(bs.H(), [q]) for q in range(n)] + _block_circuit(n, gates, rng, kinds)
    err = rel_err(bs.StateVectorSimulator(n, 0, precision="c64").evolve(ops).state_vector, oracle.OracleSV(n).evolve(ops).psi)
    # an FP32 rounding of the matrix and of the state per gate, each at most 2^-24 of the norm
    assert err < len(ops) * 2.0 ** -23, err


def test_register_blocks_on_a_density_matrix():
    n, rng = 7, np.random.default_rng(8)
    ops = [bs.Instruction(bs.H(), [q]) for q in range(n)] + _block_circuit(n, 40, rng, ("one", "ctrl", "diag", "swap"))
    err = rel_err(bs.DensityMatrixSimulator(n, 0, precision="c64").evolve(ops).density_matrix, oracle.OracleDM(n).evolve(ops).matrix)
    assert err < 2 * len(ops) * 2.0 ** -23, err


def test_c64_state_is_rounded_once_per_folded_run():
    """Gates that meet on a pair of qubits are multiplied out in FP64 and the state is rounded once for all of them.
    30 inputs of one-qubit matrices, CZ and one-qubit matrices again on six pairs: the mean error is that of six 4x4
    matrices applied in complex64 on the host (1.0e-7; a quarter more is allowed for the order of the sums).  A
    rounding per gate gives twice that."""
    n, err, model = 12, [], []
    cz = np.diag([1, 1, 1, -1.0])

    def pair(x, m, q):
        return np.einsum("abij,lijr->labr", m.reshape(2, 2, 2, 2), x.reshape(1 << q, 2, 2, -1)).reshape(-1)

    for seed in range(30):
        rng = np.random.default_rng(seed)
        u = [[np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))[0] for _ in range(n)] for _ in range(2)]
        exact = np.zeros(1 << n, dtype=np.complex128)
        exact[0] = 1
        low, ops = exact.astype(np.complex64), []
        for q in range(0, n, 2):
            m = np.kron(u[1][q], u[1][q + 1]) @ cz @ np.kron(u[0][q], u[0][q + 1])
            exact, low = pair(exact, m, q), pair(low, m.astype(np.complex64), q)
        for layer in range(2):
            ops += [bs.Instruction(bs.Unitary(u[layer][q]), [q]) for q in range(n)]
            if layer == 0:
                ops += [bs.Instruction(bs.CZ(), [q, q + 1]) for q in range(0, n, 2)]
        got = bs.StateVectorSimulator(n, 0, precision="c64").evolve(ops).state_vector
        err.append(np.linalg.norm(got - exact))
        model.append(np.linalg.norm(low - exact))
    assert np.mean(err) < 1.25 * np.mean(model), (np.mean(err), np.mean(model))
