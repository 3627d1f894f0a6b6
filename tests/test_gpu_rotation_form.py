"""Specialised and generic passes on circuits whose one-qubit gates sit at the edges of their rotation form: exact
signs, flips and identities, near-flips (cosine below 2^-20), zero angles, projections and other
non-unitary matrices, runs of mixed gates, every tile size, and depolarizing channels at the ends of
their range."""
import math

import numpy as np
import pytest

from conftest import AMP_TOL, random_density_matrix, random_state, random_unitary
from qulacs_b200 import DensityMatrix, QuantumCircuit, QuantumState, gate as G

pytestmark = pytest.mark.gpu


def _one_qubit_gates(q, rng):
    tiny = 2.0 ** -24
    return [G.X(q), G.Y(q), G.Z(q), G.H(q), G.S(q), G.Tdag(q), G.sqrtX(q), G.sqrtYdag(q), G.RX(q, math.pi),
            G.RY(q, math.pi), G.RY(q, math.pi - tiny), G.RX(q, math.pi + tiny), G.RY(q, 0.0), G.RZ(q, 0.0),
            G.RX(q, 0.0), G.RZ(q, math.pi), G.RY(q, 5.0), G.RX(q, -4.0), G.U3(q, math.pi, 0.3, -1.0),
            G.U3(q, 0.0, 0.2, 0.1), G.U3(q, 1e-9, 2.0, 1.0), G.DenseMatrix(q, random_unitary(1, rng)),
            G.DenseMatrix(q, np.array([[1.1, 0.2j], [0.3, 0.8 - 0.1j]])),
            G.DenseMatrix(q, np.array([[0.0, 0.9], [-1.2j, 0.0]])),
            G.DenseMatrix(q, np.array([[0.0, 0.9], [1e-3, 0.0]])),
            G.DiagonalMatrix([q], [0.9j, -1.1])]


@pytest.mark.parametrize("n", [7, 11, 12, 14, 19])
@pytest.mark.parametrize("mode", ["staged", "staged_fused"])
@pytest.mark.parametrize("spec", [1, 0])
def test_edge_gates_against_oracle(port, n, mode, spec):
    rng = np.random.default_rng(70 + n)
    c = QuantumCircuit(n)
    c.set_specialized(spec)
    if mode == "staged_fused":
        c.set_fusion(1)
    want = random_state(n, rng)
    s = QuantumState(n)
    s.load(want)

    def add(g, controls=()):
        c.add_gate(g)
        if g.name == "CNOT":
            port.CNOT_gate(g.targets[0], g.targets[1], want)
        elif g.name == "CZ":
            port.CZ_gate(g.targets[0], g.targets[1], want)
        else:
            port.multi_qubit_dense_matrix_gate(g.targets, g.get_matrix(), want)

    pool = [g for _ in range(6) for g in _one_qubit_gates(0, rng)]
    for i in rng.permutation(len(pool)):
        g = pool[i].copy()
        g.targets = [int(rng.integers(n))]
        add(g)
        r = rng.random()
        a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
        if r < 0.25:
            add(G.CNOT(a, b))
        elif r < 0.5:
            add(G.CZ(a, b))
        elif r < 0.6:
            add(G.SWAP(a, b))
        elif r < 0.65:
            add(G.DenseMatrix([a, b], random_unitary(2, rng)))
    for q in (0, n - 1):
        add(G.P0(q))
    c.update_quantum_state(s, mode=mode)
    assert np.max(np.abs(s.get_vector() - want)) <= AMP_TOL * max(1.0, float(np.max(np.abs(want))))


@pytest.mark.parametrize("spec", [1, 0])
def test_long_runs_of_near_flips_keep_their_scale(port, spec):
    """200 near-flips on the qubits of one tile: the cosines deferred over a pass (2^-19 each) exceed the
    bound on a deferred scale, so the later ones must not be deferred."""
    n = 12
    rng = np.random.default_rng(8)
    c = QuantumCircuit(n)
    c.set_specialized(spec)
    want = random_state(n, rng)
    s = QuantumState(n)
    s.load(want)
    for i in range(200):
        g = G.RY(i % n, math.pi - 2.0 ** -18) if i % 2 else G.RX(i % n, math.pi - 2.0 ** -18)
        c.add_gate(g)
        port.multi_qubit_dense_matrix_gate(g.targets, g.get_matrix(), want)
        if i % n == n - 1:
            c.add_gate(G.CNOT(0, n - 1))
            port.CNOT_gate(0, n - 1, want)
    c.update_quantum_state(s)
    assert np.max(np.abs(s.get_vector() - want)) <= AMP_TOL


def test_channels_of_a_small_density_matrix(port):
    """5 qubits: the generic kernel's channel steps, channels merged past unitaries, against the oracle."""
    n = 5
    rng = np.random.default_rng(10)
    c = QuantumCircuit(n)
    rho = random_density_matrix(n, rng)
    d = DensityMatrix(n)
    d.load(rho)
    want = rho.copy()
    for _ in range(4):
        for q in range(n):
            g = G.RY(q, float(rng.uniform(0, 6)))
            c.add_gate(g)
            port.dm_single_qubit_dense_matrix_gate(q, g.get_matrix(), want)
            c.add_gate(G.DepolarizingNoise(q, 0.1))
            port.dm_depolarizing_noise(q, 0.1, want)
            u = random_unitary(1, rng)
            c.add_gate(G.DenseMatrix(q, u))
            port.dm_single_qubit_dense_matrix_gate(q, u, want)
        for a in range(n):
            b, p = (a + 2) % n, float(rng.choice([0.02, 15 / 16, 1.0]))
            c.add_gate(G.CZ(a, b) if a % 2 else G.CNOT(a, b))
            (port.dm_CZ_gate if a % 2 else port.dm_CNOT_gate)(a, b, want)
            c.add_gate(G.TwoQubitDepolarizingNoise(a, b, p))
            port.dm_two_qubit_depolarizing_noise(a, b, p, want)
    c.update_quantum_state(d, mode="staged")
    assert np.max(np.abs(d.get_matrix() - want)) <= AMP_TOL


@pytest.mark.parametrize("p1,p2", [(0.01, 0.02), (0.75, 15 / 16), (1.0, 1.0), (0.0, 0.9374)])
@pytest.mark.parametrize("mode", ["staged", "staged_fused"])
def test_channels_against_gate_by_gate(mode, p1, p2):
    """11 qubits: the smallest density matrix whose passes are specialised.  The channel kernels of the
    gate-by-gate mode are checked against the oracle in test_gpu_dm.py."""
    n = 11
    rng = np.random.default_rng(9)
    c = QuantumCircuit(n)
    for _ in range(3):
        for q in range(n):
            c.add_gate(G.RY(q, float(rng.uniform(0, 6))))
            c.add_gate(G.DepolarizingNoise(q, p1))
            c.add_gate(G.U3(q, *(float(x) for x in rng.uniform(0, 6, 3))))
            c.add_gate(G.DepolarizingNoise(q, 0.03))
        for _ in range(n):
            a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
            c.add_gate(G.CZ(a, b) if rng.random() < 0.5 else G.CNOT(a, b))
            c.add_gate(G.TwoQubitDepolarizingNoise(a, b, p2 if rng.random() < 0.2 else 0.01))
        c.add_gate(G.DenseMatrix(3, np.array([[1.0, 0.1], [0.0, 0.9]])))  # not unitary: channels stay before it
    if mode == "staged_fused":
        c.set_fusion(2)
    psi = QuantumState(n)
    psi.set_Haar_random_state(4)
    a, b = DensityMatrix(n), DensityMatrix(n)
    a.load(psi)
    b.load(psi)
    c.update_quantum_state(a, mode=mode)
    c.update_quantum_state(b, mode="gate_by_gate")
    assert np.max(np.abs(a.get_matrix() - b.get_matrix())) <= AMP_TOL


@pytest.mark.parametrize("n", [5, 11])
@pytest.mark.parametrize("mode", ["staged", "staged_fused"])
def test_channels_after_non_unitary_diagonals(n, mode):
    """Diagonals that are not unitary before channels, in the generic (5 qubits) and the specialised kernels (11)."""
    rng = np.random.default_rng(12)
    c = QuantumCircuit(n)
    for q in range(n):
        c.add_gate(G.RY(q, float(rng.uniform(0, 6))))
        c.add_gate(G.DiagonalMatrix([q], [1.0, 0.8] if q % 2 else [0.9j, -1.1]))
        c.add_gate(G.DepolarizingNoise(q, 0.3))
    for q in range(n - 1):
        c.add_gate(G.CNOT(q, q + 1))
        c.add_gate(G.DiagonalMatrix([q], [0.8, 1.2]))
        c.add_gate(G.TwoQubitDepolarizingNoise(q, q + 1, 0.1))
        c.add_gate(G.DepolarizingNoise(q, 0.1))
    if mode == "staged_fused":
        c.set_fusion(1)
    psi = QuantumState(n)
    psi.set_Haar_random_state(5)
    a, b = DensityMatrix(n), DensityMatrix(n)
    a.load(psi)
    b.load(psi)
    c.update_quantum_state(a, mode=mode)
    c.update_quantum_state(b, mode="gate_by_gate")
    want = b.get_matrix()
    assert np.max(np.abs(a.get_matrix() - want)) <= AMP_TOL * max(1.0, float(np.max(np.abs(want))))


@pytest.mark.parametrize("n", [2, 5, 11])
def test_hundreds_of_channels_in_one_pass(n):
    """Channels whose deferred scales exceed the bound of a pass run unscaled, in the generic and the specialised
    (11 qubits) kernels."""
    c = QuantumCircuit(n)
    for i in range(300):
        c.add_gate(G.DepolarizingNoise(0, 1.0))
        c.add_gate(G.RY(0, 0.1 * i))
        c.add_gate(G.CZ(0, 1))
        if i % 3 == 0:
            c.add_gate(G.TwoQubitDepolarizingNoise(0, 1, 0.9))
    psi = QuantumState(n)
    psi.set_Haar_random_state(6)
    a, b = DensityMatrix(n), DensityMatrix(n)
    a.load(psi)
    b.load(psi)
    c.update_quantum_state(a, mode="staged")
    c.update_quantum_state(b, mode="gate_by_gate")
    got = a.get_matrix()
    assert np.all(np.isfinite(got)) and np.max(np.abs(got - b.get_matrix())) <= AMP_TOL


def test_failed_fused_planning_leaves_no_schedule():
    """A block size whose kernels cannot be compiled (a NaN among parameters that are too many for a parameter
    block) fails the call; the next call must not find a half-built schedule."""
    n = 12
    rng = np.random.default_rng(2)
    c = QuantumCircuit(n)
    c.set_specialized(1)
    c.add_gate(G.DenseMatrix(0, np.full((2, 2), np.nan)))
    for layer in range(22):  # k = 2: 132 blocks with a 4 x 4 matrix each; k = 0, 1: one angle per gate
        for a in range(layer % 2, n, 2):
            b = (a + 1) % n
            for _ in range(3):
                c.add_gate(G.RY(a, float(rng.uniform(0.1, 0.5))))
                c.add_gate(G.RY(b, float(rng.uniform(0.1, 0.5))))
                c.add_gate(G.CNOT(a, b))
    s = QuantumState(n)
    for _ in range(2):
        with pytest.raises(RuntimeError, match="NVRTC compile failed"):
            c.update_quantum_state(s, mode="staged_fused")
        assert c.fusion_info()[0] == -1
    c.set_fusion(0)
    c.update_quantum_state(s, mode="staged_fused")
    assert c.fusion_info()[0] == 0


@pytest.mark.parametrize("n", [4, 7, 13, 19])
@pytest.mark.parametrize("spec", [1, 0])
def test_permutations_are_exact(n, spec):
    """CNOT, SWAP and X move amplitudes without arithmetic, tiny ones beside large ones included."""
    rng = np.random.default_rng(n)
    v = rng.normal(size=1 << n) * 10.0 ** rng.uniform(-18, 0, size=1 << n) + 0j
    idx = np.arange(1 << n)
    c = QuantumCircuit(n)
    if n >= 7:
        c.set_specialized(spec)
    for i in range(8 * n):
        a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
        if i % 4 < 2:
            c.add_gate(G.CNOT(a, b))
            idx = np.where((idx >> a) & 1, idx ^ (1 << b), idx)
        elif i % 4 == 2:
            c.add_gate(G.SWAP(a, b))
            x = ((idx >> a) ^ (idx >> b)) & 1
            idx = idx ^ (x << a) ^ (x << b)
        else:
            c.add_gate(G.X(a))
            idx = idx ^ (1 << a)
    want = np.empty_like(v)
    want[idx] = v
    s = QuantumState(n)
    s.load(v)
    c.update_quantum_state(s)
    assert np.array_equal(s.get_vector(), want)


@pytest.mark.parametrize("n", [8, 13, 16])
def test_block_size_of_small_states_counts_launches(n):
    """Blocks of three and more qubits run outside the passes, one launch each: on states that fit the L2 cache the
    autotuner must not take them for free."""
    from qulacs_b200 import workloads as W
    for gates in (W.layered_rotation_circuit(n, 10, 1), W.hea_circuit(n, 8, 1), W.u3_cz_circuit(n, 20, 1)):
        c = W.to_circuit(gates, n)
        c.update_quantum_state(QuantumState(n), mode="staged_fused")
        assert 0 <= c.fusion_info()[0] <= 2
