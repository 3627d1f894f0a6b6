"""The staged planner without a GPU: random circuits through the passes, phases and programs of the staged modes,
replayed on the host (qs_debug_staged_replay), against plain gate-by-gate application with the oracle."""
import ctypes as C

import numpy as np
import pytest

from conftest import random_density_matrix, random_state, random_unitary
from qulacs_b200 import QuantumCircuit
from qulacs_b200 import gate as G
from qulacs_b200._lib import call

TOL = 1e-13  # a few hundred gates of rounding (2e-16 each) on normalised states


def replay(circ, state, k=0, spec=True, tile_bits=12, dm=False):
    out = np.ascontiguousarray(state, dtype=np.complex128).copy()
    call("qs_debug_staged_replay", circ._h, int(dm), k, int(spec), tile_bits, out.ctypes.data_as(C.c_void_p),
         1 << circ.qubit_count)
    return out


def apply_vector(port, gates, v):
    """Each gate as a dense matrix over its qubits (controls expanded)."""
    c = QuantumCircuit(int(np.log2(v.size)))
    for g in gates:
        c.add_gate(g)
    flat = c.fuse(0)
    for i in range(len(flat)):
        qubits, m = flat[i]
        port.multi_qubit_dense_matrix_gate(qubits, m, v)
    return c


def apply_matrix(port, gates, rho):
    n = int(np.log2(rho.shape[0]))
    c = QuantumCircuit(n)
    for g in gates:
        c.add_gate(g)
    for g in gates:
        t = g.get_target_index_list()
        if g.kind == "DEPOLARIZING":
            if len(t) == 1:
                port.dm_depolarizing_noise(t[0], float(g.params[0]), rho)
            else:
                port.dm_two_qubit_depolarizing_noise(t[0], t[1], float(g.params[0]), rho)
            continue
        one = QuantumCircuit(n)
        one.add_gate(g)
        qubits, m = one.fuse(0)[0]
        port.dm_multi_qubit_dense_matrix_gate(qubits, m, rho)
    return c


def random_gate(n, rng, unitary=True, channels=False):
    q = int(rng.integers(n))
    a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
    ang = float(rng.uniform(0, 6.3))
    r = rng.random()
    if channels and r < 0.3:
        p = float(rng.choice([0.02, 0.3, 0.75, 1.0]))
        return G.DepolarizingNoise(q, p) if rng.random() < 0.6 else G.TwoQubitDepolarizingNoise(a, b, p)
    if not unitary and rng.random() < 0.25:
        return [G.DiagonalMatrix([q], [1.0, 0.8]), G.DiagonalMatrix([q], [0.9j, -1.1]), G.P0(q),
                G.DenseMatrix(q, np.array([[1.1, 0.2j], [0.3, 0.8 - 0.1j]])),
                G.DenseMatrix(q, np.array([[0.0, 0.9], [-1.2j, 0.0]]))][int(rng.integers(5))]
    kinds = [lambda: G.RX(q, ang), lambda: G.RY(q, ang), lambda: G.RZ(q, ang), lambda: G.H(q), lambda: G.X(q),
             lambda: G.Y(q), lambda: G.Z(q), lambda: G.S(q), lambda: G.T(q), lambda: G.sqrtX(q),
             lambda: G.U3(q, ang, 0.3, -ang), lambda: G.DenseMatrix(q, random_unitary(1, rng)),
             lambda: G.CNOT(a, b), lambda: G.CNOT(a, b), lambda: G.CZ(a, b), lambda: G.SWAP(a, b),
             lambda: G.DenseMatrix([a, b], random_unitary(2, rng)), lambda: G.PauliRotation([a, b], [1, 2], ang),
             lambda: controlled(a, b, rng)]
    return kinds[int(rng.integers(len(kinds)))]()


def controlled(a, b, rng):
    g = G.DenseMatrix(a, random_unitary(1, rng))
    g.add_control_qubit(b, int(rng.integers(2)))
    return g


@pytest.mark.parametrize("spec", [True, False])
@pytest.mark.parametrize("k,tile_bits", [(0, 12), (0, 5), (1, 12), (2, 11)])
def test_random_state_circuits(port, spec, k, tile_bits):
    rng = np.random.default_rng(100 * k + tile_bits)
    for trial in range(12):
        n = 4 + trial % 4
        v = random_state(n, rng)
        want = v.copy()
        c = apply_vector(port, [random_gate(n, rng, unitary=trial % 2 == 0) for _ in range(60)], want)
        got = replay(c, v, k, spec, tile_bits)
        assert np.max(np.abs(got - want)) <= TOL * max(1.0, float(np.max(np.abs(want))))


def edge_gate(q, rng):
    """One-qubit gates at the edges of the rotation form: flips, signs, near-flips, zero angles, non-unitary."""
    tiny = 2.0 ** -24
    pool = [G.X(q), G.Y(q), G.Z(q), G.H(q), G.S(q), G.RX(q, np.pi), G.RY(q, np.pi), G.RY(q, np.pi - tiny),
            G.RX(q, np.pi + tiny), G.RY(q, 0.0), G.RZ(q, np.pi), G.U3(q, np.pi, 0.3, -1.0), G.U3(q, 1e-9, 2.0, 1.0),
            G.DenseMatrix(q, np.array([[1.1, 0.2j], [0.3, 0.8 - 0.1j]])), G.DiagonalMatrix([q], [0.9j, -1.1]),
            G.DenseMatrix(q, np.array([[0.0, 0.9], [-1.2j, 0.0]])), G.DenseMatrix(q, np.array([[0.0, 0.9], [1e-3, 0.0]]))]
    return pool[int(rng.integers(len(pool)))]


@pytest.mark.parametrize("spec", [True, False])
def test_edge_gates_between_relabellings(port, spec):
    rng = np.random.default_rng(1)
    for trial in range(400):
        n = 4
        gates = []
        for _ in range(trial % 25 + 1):
            a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
            gates.append(edge_gate(int(rng.integers(n)), rng))
            gates += [[G.CNOT(a, b)], [G.CZ(a, b)], [G.SWAP(a, b)], []][int(rng.choice(4, p=[0.35, 0.25, 0.1, 0.3]))]
        v = random_state(n, rng)
        want = v.copy()
        c = apply_vector(port, gates, want)
        assert np.max(np.abs(replay(c, v, spec=spec) - want)) <= TOL * max(1.0, float(np.max(np.abs(want))))


@pytest.mark.parametrize("spec", [True, False])
@pytest.mark.parametrize("k,tile_bits", [(0, 12), (0, 5), (2, 11)])
def test_random_noisy_matrix_circuits(port, spec, k, tile_bits):
    rng = np.random.default_rng(200 * k + tile_bits)
    for trial in range(8):
        n = 2 + trial % 3
        rho = random_density_matrix(n, rng)
        want = rho.copy()
        c = apply_matrix(port, [random_gate(n, rng, channels=True) for _ in range(60)], want)
        assert np.max(np.abs(replay(c, rho, k, spec, tile_bits, dm=True) - want)) <= TOL


@pytest.mark.parametrize("spec", [True, False])
@pytest.mark.parametrize("d", [[1.0, 0.8], [0.9j, -1.1], [0.6, 0.6], [1.0, 1.0 + 2.0 ** -30]])
def test_channels_after_non_unitary_diagonals(port, d, spec):
    """A depolarizing channel commutes with unitary diagonals only: one whose entries are not of modulus 1 is
    applied before the channel that follows it."""
    gates = [G.RY(0, 1.0), G.DiagonalMatrix([0], d), G.DepolarizingNoise(0, 0.3), G.RY(1, 0.4), G.RZ(0, 0.5),
             G.DiagonalMatrix([1], d), G.H(1), G.RX(1, 0.3), G.DiagonalMatrix([1], d), G.DepolarizingNoise(1, 0.1),
             G.TwoQubitDepolarizingNoise(0, 1, 0.2)]
    rng = np.random.default_rng(3)
    rho = random_density_matrix(2, rng)
    want = rho.copy()
    c = apply_matrix(port, gates, want)
    assert np.max(np.abs(replay(c, rho, spec=spec, dm=True) - want)) <= TOL


@pytest.mark.parametrize("spec", [True, False])
def test_random_noisy_matrix_circuits_with_non_unitary_gates(port, spec):
    rng = np.random.default_rng(17)
    for trial in range(60):
        n = 2 + trial % 3
        rho = random_density_matrix(n, rng)
        want = rho.copy()
        c = apply_matrix(port, [random_gate(n, rng, unitary=False, channels=True) for _ in range(30)], want)
        got = replay(c, rho, trial % 3, spec, dm=True)
        assert np.max(np.abs(got - want)) <= TOL * max(1.0, float(np.max(np.abs(want))))


@pytest.mark.parametrize("spec", [True, False])
@pytest.mark.parametrize("p,two", [(0.5, False), (1.0, False), (0.1, True), (0.9, True), (1.0, True), (15 / 16, True)])
def test_thousands_of_channels_in_one_pass(port, p, two, spec):
    """The scales that channels defer over a pass are bounded: 2000 of them on one tile."""
    gates = []
    for i in range(1000):
        gates.append(G.TwoQubitDepolarizingNoise(0, 1, p) if two else G.DepolarizingNoise(i % 2, p))
        gates.append(G.U3(i % 2, 0.7, 0.1 * (i % 50), 0.4))
        gates.append(G.CZ(0, 1) if i % 3 else G.TwoQubitDepolarizingNoise(1, 0, p))
    rng = np.random.default_rng(3)
    rho = random_density_matrix(2, rng)
    want = rho.copy()
    c = apply_matrix(port, gates, want)
    got = replay(c, rho, spec=spec, dm=True)
    assert np.all(np.isfinite(got)) and np.max(np.abs(got - want)) <= 10 * TOL


@pytest.mark.parametrize("spec", [True, False])
def test_long_products_of_non_unitary_diagonals_in_one_pass(port, spec):
    """Non-unitary diagonals that shrink the state by 2^-650 over a pass, beside rotations that defer 2^400: the
    result keeps its precision."""
    n = 4
    gates = []
    for i in range(750):
        gates += [G.DiagonalMatrix([i % n], [0.55, 0.52]), G.RY(i % n, 2.5), G.CNOT(i % n, (i + 1) % n)]
    rng = np.random.default_rng(4)
    v = random_state(n, rng)
    want = v.copy()
    c = apply_vector(port, gates, want)
    got = replay(c, v, spec=spec)
    assert 0 < np.max(np.abs(want)) < 1e-180
    assert np.max(np.abs(got - want)) <= 10 * TOL * float(np.max(np.abs(want)))


@pytest.mark.parametrize("spec", [True, False])
@pytest.mark.parametrize("k", [0, 2])
def test_permutations_are_exact(spec, k):
    """CNOT, SWAP and X move amplitudes without arithmetic: a tiny amplitude beside a large one stays as it is,
    between rotations on other qubits too."""
    n = 7
    rng = np.random.default_rng(6)
    v = rng.normal(size=1 << n) * 10.0 ** rng.uniform(-18, 0, size=1 << n) + 0j
    idx = np.arange(1 << n)
    c = QuantumCircuit(n)
    for _ in range(60):
        a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
        r = rng.random()
        if r < 0.6:
            c.add_gate(G.CNOT(a, b))
            idx = np.where((idx >> a) & 1, idx ^ (1 << b), idx)
        elif r < 0.8:
            c.add_gate(G.SWAP(a, b))
            x = ((idx >> a) ^ (idx >> b)) & 1
            idx = idx ^ (x << a) ^ (x << b)
        else:
            c.add_gate(G.X(a))
            idx = idx ^ (1 << a)
    want = np.empty_like(v)
    want[idx] = v
    assert np.array_equal(replay(c, v, k, spec), want)


@pytest.mark.parametrize("spec", [True, False])
@pytest.mark.parametrize("kind", ["scaled", "column", "skewed", "real", "diagonal"])
def test_matrices_near_unitary_are_applied_as_given(port, kind, spec):
    """A deviation from unitarity of 5e-14 is in the matrix that a caller gave: 200 of them show as 1e-11."""
    n, eps = 4, 5e-14
    rng = np.random.default_rng(9)
    u = random_unitary(1, rng)
    if kind == "real":
        c, s = np.cos(0.7), np.sin(0.7)
        u = np.array([[c, s], [-s * (1 + eps), c * (1 + eps)]])
    elif kind == "diagonal":
        u = np.diag([1.0, (1 + eps) * np.exp(0.3j)])
    else:
        u = u @ {"scaled": np.eye(2) * (1 + eps), "column": np.diag([1.0, 1 + 2 * eps]),
                 "skewed": np.array([[1.0, 2 * eps], [0.0, 1.0]])}[kind]
    gates = []
    for i in range(200):
        gates += [G.DenseMatrix(i % n, u), G.CNOT(i % n, (i + 1) % n)]
    v = random_state(n, rng)
    want = v.copy()
    c = apply_vector(port, gates, want)
    assert np.max(np.abs(replay(c, v, spec=spec) - want)) <= 5 * TOL
    rho = random_density_matrix(2, rng)
    gates = []
    for i in range(100):
        gates += [G.DenseMatrix(i % 2, u), G.DepolarizingNoise(i % 2, 0.01), G.RY(i % 2, 0.1)]
    want = rho.copy()
    c = apply_matrix(port, gates, want)
    assert np.max(np.abs(replay(c, rho, spec=spec, dm=True) - want)) <= 5 * TOL
