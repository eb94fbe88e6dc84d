"""Adjoint gradients vs the parameter-shift rule (exact for these generators) and
central finite differences."""
import numpy as np
import pytest

from conftest import bs

pytestmark = pytest.mark.gpu
from importlib import import_module  # noqa: E402

adj = import_module("braketsimulator_gb300.adjoint")


def ansatz(n, layers, rng):
    ops = []
    for _ in range(layers):
        for q in range(n):
            ops.append(bs.Instruction(bs.Ry(float(rng.uniform(-np.pi, np.pi))), [q]))
            ops.append(bs.Instruction(bs.Rz(float(rng.uniform(-np.pi, np.pi))), [q]))
        for q in range(n):
            ops.append(bs.Instruction(bs.ZZ(float(rng.uniform(-np.pi, np.pi))), [q, (q + 1) % n]))
    return ops


def hamiltonian(n, terms, rng):
    h = []
    for _ in range(terms):
        w = int(rng.integers(1, min(4, n) + 1))
        qs = rng.choice(n, w, replace=False)
        h.append((float(rng.normal()), {int(q): "XYZ"[rng.integers(3)] for q in qs}))
    return h


@pytest.mark.parametrize("n,layers", [(2, 1), (4, 2), (7, 2), (12, 2)])
def test_adjoint_matches_parameter_shift(n, layers):
    rng = np.random.default_rng(n)
    ops = ansatz(n, layers, rng)
    h = hamiltonian(n, 8, rng)
    sim = bs.StateVectorSimulator(n, 0)
    e, g = adj.adjoint_gradient(sim, ops, h)
    e_ref = adj.energy(sim, ops, h)
    ps = adj.parameter_shift_gradient(sim, ops, h)
    assert abs(e - e_ref) < 1e-12
    assert np.max(np.abs(g - ps)) < 1e-10


def test_adjoint_other_generators_and_shared_parameters():
    rng = np.random.default_rng(4)
    n = 5
    ops = [bs.Instruction(bs.H(), [q]) for q in range(n)]
    ops += [bs.Instruction(bs.Rx(0.3), [0]), bs.Instruction(bs.XX(0.7), [1, 3]), bs.Instruction(bs.YY(-0.4), [2, 4]),
            bs.Instruction(bs.PhaseShift(1.1), [2]), bs.Instruction(bs.CNot(), [0, 4]), bs.Instruction(bs.Rx(0.3), [3])]
    h = hamiltonian(n, 6, rng)
    sim = bs.StateVectorSimulator(n, 0)
    e, g = adj.adjoint_gradient(sim, ops, h)
    ps = adj.parameter_shift_gradient(sim, ops, h)
    fd = adj.finite_difference_gradient(sim, ops, h)
    assert np.max(np.abs(g - ps)) < 1e-10
    assert np.max(np.abs(g - fd)) < 1e-6
    # shared parameter: both Rx gates use slot 0
    pidx = [-1] * n + [0, 1, 2, 3, -1, 0]
    e2, g2 = adj.adjoint_gradient(sim, ops, h, pidx)
    assert abs(g2[0] - (g[0] + g[4])) < 1e-12


@pytest.mark.parametrize("n", [6, 13])
def test_adjoint_complex64_state(n):
    """complex64 state, float-float arithmetic and FP64-grade inner products: the gradient differs
    from the complex128 one by the complex64 rounding of the stored states only."""
    rng = np.random.default_rng(60 + n)
    ops = ansatz(n, 3, rng)
    h = hamiltonian(n, 10, rng)
    e128, g128 = adj.adjoint_gradient(bs.StateVectorSimulator(n, 0), ops, h)
    e64, g64 = adj.adjoint_gradient(bs.StateVectorSimulator(n, 0, precision="c64"), ops, h)
    scale = max(1.0, sum(abs(c) for c, _ in h))
    assert abs(e64 - e128) < 2e-5 * scale
    assert np.max(np.abs(g64 - g128)) < 2e-5 * scale


@pytest.mark.parametrize("segments", [1, 2, 5, 40])
def test_adjoint_checkpoint_segments(segments):
    """Forward checkpoints (psi kept after each segment, restored on the way back) give the same
    gradients as pure uncomputation, for any segment count (including more segments than gates
    per segment allow)."""
    n = 9
    rng = np.random.default_rng(77)
    ops = ansatz(n, 3, rng)
    h = hamiltonian(n, 8, rng)
    ref = bs.StateVectorSimulator(n, 0)
    bs.set_tuning(ref, adj_segments=1)
    e1, g1 = adj.adjoint_gradient(ref, ops, h)
    sim = bs.StateVectorSimulator(n, 0)
    bs.set_tuning(sim, adj_segments=segments)
    e, g = adj.adjoint_gradient(sim, ops, h)
    assert abs(e - e1) < 1e-12
    assert np.max(np.abs(g - g1)) < 1e-12
    ps = adj.parameter_shift_gradient(sim, ops, h)
    assert np.max(np.abs(g - ps)) < 1e-10


def test_adjoint_checkpoints_bound_complex64_drift():
    """complex64: uncomputing psi through a deep circuit drifts; checkpoints reset it per segment."""
    n = 10
    rng = np.random.default_rng(90)
    ops = ansatz(n, 12, rng)
    h = hamiltonian(n, 10, rng)
    _, g128 = adj.adjoint_gradient(bs.StateVectorSimulator(n, 0), ops, h)
    errs = {}
    for seg in (1, 16):
        sim = bs.StateVectorSimulator(n, 0, precision="c64")
        bs.set_tuning(sim, adj_segments=seg)
        _, g64 = adj.adjoint_gradient(sim, ops, h)
        errs[seg] = float(np.max(np.abs(g64 - g128)))
    scale = max(1.0, sum(abs(c) for c, _ in h))
    assert errs[16] < 2e-5 * scale
    assert errs[16] <= errs[1] * 1.5


def test_rrule_and_torch_autograd():
    import torch
    n = 6
    rng = np.random.default_rng(12)
    h = hamiltonian(n, 6, rng)
    theta0 = rng.uniform(-np.pi, np.pi, size=3 * n)

    def build(th):
        ops = []
        for q in range(n):
            ops.append(bs.Instruction(bs.Ry(float(th[q])), [q]))
            ops.append(bs.Instruction(bs.Rz(float(th[n + q])), [q]))
        for q in range(n):
            ops.append(bs.Instruction(bs.ZZ(float(th[2 * n + q])), [q, (q + 1) % n]))
        return ops

    sim = bs.StateVectorSimulator(n, 0)
    e, pb = bs.energy_rrule(sim, build(theta0), h)
    ps = adj.parameter_shift_gradient(sim, build(theta0), h)
    assert np.max(np.abs(pb(2.0) - 2.0 * ps)) < 1e-10
    f = bs.torch_energy(build, h, sim)
    theta = torch.tensor(theta0, dtype=torch.float64, requires_grad=True)
    out = 3.0 * f(theta)
    out.backward()
    assert abs(out.item() - 3.0 * e) < 1e-12
    assert np.max(np.abs(theta.grad.numpy() - 3.0 * ps)) < 1e-10


def _all_forms(n, layers, rng):
    """Every item form of the backward sweep: X/Y rotations (gate and marker in one pass), diagonal
    rotations and phases, two-qubit generators, fixed dense / monomial / diagonal gates with controls,
    a diagonal gate on more bits than a folded table holds."""
    ops = [bs.Instruction(bs.H(), [q]) for q in range(n)]
    a = lambda: float(rng.uniform(-np.pi, np.pi))  # noqa: E731
    for layer in range(layers):
        for q in range(n):
            ops.append(bs.Instruction([bs.Rx, bs.Ry, bs.Rz][(q + layer) % 3](a()), [q]))
        for q in range(0, n - 1, 2):
            ops.append(bs.Instruction([bs.ZZ, bs.XX, bs.YY][(q // 2 + layer) % 3](a()), [q, q + 1]))
        for q in range(n):
            ops.append(bs.Instruction(bs.PhaseShift(a()), [q]) if q % 2 else bs.Instruction(bs.Rz(a()), [q]))
        if n > 1:
            ops.append(bs.Instruction(bs.CNot(), [layer % n, (layer + 1) % n]))
            ops.append(bs.Instruction(bs.CPhaseShift(0.3), [(layer + 1) % n, layer % n]))
            ops.append(bs.Instruction(bs.Control(bs.H(), (1,)), [n - 1, 0]))
        if n >= 10:
            ops.append(bs.Instruction(bs.Control(bs.Z(), tuple([1] * 9)), list(range(10))))
    return ops


@pytest.mark.parametrize("n,layers", [(1, 3), (3, 2), (9, 2), (10, 1), (12, 1), (13, 1), (15, 1)])
def test_backward_sweep_forms_match_parameter_shift(n, layers):
    rng = np.random.default_rng(900 + n)
    ops = _all_forms(n, layers, rng)
    # the fixed controlled phases are not parameters; every differentiable gate is
    h = hamiltonian(n, 6, rng)
    sim = bs.StateVectorSimulator(n, 0)
    e, g = adj.adjoint_gradient(sim, ops, h)
    ps = adj.parameter_shift_gradient(sim, ops, h)
    assert abs(e - adj.energy(sim, ops, h)) < 1e-12 * max(1.0, sum(abs(c) for c, _ in h))
    assert np.max(np.abs(g - ps)) < 1e-10
    e64, g64 = adj.adjoint_gradient(bs.StateVectorSimulator(n, 0, precision="c64"), ops, h)
    assert np.max(np.abs(g64 - ps)) < 2e-5 * max(1.0, sum(abs(c) for c, _ in h))


def test_more_rotations_in_a_sweep_than_the_sum_buffer_holds():
    n, rng = 12, np.random.default_rng(77)   # one tile: every gate in one sweep, 60 rotation sums
    ops = [bs.Instruction([bs.Rx, bs.Ry][layer % 2](float(rng.uniform(-3, 3))), [q]) for layer in range(5) for q in range(n)]
    h = hamiltonian(n, 5, rng)
    sim = bs.StateVectorSimulator(n, 0)
    bs.set_tuning(sim, adj_segments=1)
    _, g = adj.adjoint_gradient(sim, ops, h)
    assert np.max(np.abs(g - adj.parameter_shift_gradient(sim, ops, h))) < 1e-10


def test_diagonal_gate_that_is_not_unitary_keeps_its_place():
    """A diagonal matrix with entries off the unit circle does not leave conj(lambda) psi alone: the
    markers on its bits stay on their side of it, so the gradient equals the one with the same matrix
    given as a dense gate with a tiny off-diagonal entry."""
    rng = np.random.default_rng(5)
    h = hamiltonian(4, 5, rng)
    grads = []
    for eps in (0.0, 1e-300):
        m = np.array([[1.0, eps], [0.0, 0.7]], dtype=complex)
        ops = [bs.Instruction(bs.H(), [q]) for q in range(4)] + [bs.Instruction(bs.Rz(0.4), [0]), bs.Instruction(bs.Ry(0.3), [1])]
        ops += [bs.Instruction(bs.Unitary(m), [0]), bs.Instruction(bs.ZZ(0.9), [0, 2]), bs.Instruction(bs.Rx(-0.8), [0])]
        grads.append(adj.adjoint_gradient(bs.StateVectorSimulator(4, 0), ops, h)[1])
    assert np.max(np.abs(grads[0] - grads[1])) < 1e-12


def test_gradients_keep_at_most_4_gib_between_calls():
    """Checkpoints stay for a handle's next gradient, 4 GiB over all handles: ten simulators of 21 qubits (512 MiB of
    checkpoints each) leave no more than that behind beside their states, plans and scratch, and nothing once closed."""
    import gc
    import torch
    n, rng = 21, np.random.default_rng(4)
    ops = [bs.Instruction([bs.Rx, bs.Ry][(q + k) % 2](float(rng.uniform(-3, 3))), [q]) for k in range(12) for q in range(n)]
    h = hamiltonian(n, 3, rng)
    adj.adjoint_gradient(bs.StateVectorSimulator(n, 0), ops, h)   # the library's own set-up
    gc.collect()
    free0 = torch.cuda.mem_get_info()[0]
    sims = [bs.StateVectorSimulator(n, 0) for _ in range(10)]
    first = [adj.adjoint_gradient(s, ops, h) for s in sims]
    left = free0 - torch.cuda.mem_get_info()[0]
    assert left < (4 << 30) + 10 * (64 << 20), left >> 20
    again = [adj.adjoint_gradient(s, ops, h) for s in sims]
    for (e, g), (e2, g2) in zip(first, again):
        assert abs(e - e2) < 1e-12 and np.max(np.abs(g - g2)) < 1e-12
    del sims
    gc.collect()
    assert free0 - torch.cuda.mem_get_info()[0] < 64 << 20
