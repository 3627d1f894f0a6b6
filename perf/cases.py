"""Timed cases: what a program built on this package has it do, through the package's public classes.

Kinds of work (a case's "kind"):
  circuit   reset the state, apply a parametrised circuit to it and, with "terms" > 0, read the energy --
            the inner loop of a variational program or of a random-circuit run.  "precision" is the
            state's: c128, or c64 for the reduced-precision path
  energy    <H> of a random Hamiltonian on a given state
  dense     multi-qubit dense gates (kmin..kmax targets, one gate of each size) on a given state
  noisy     a density matrix through a circuit with depolarizing noise after every gate
  batch     many small circuits of uneven sizes, each with its own Hamiltonian, in one call
  sampling  shots from a given state

Circuits: "layered" (RX, RY, RZ on every qubit, then a CNOT ladder), "hea" (RY, RZ on every qubit, then a
CZ ring), "u3cz" (U3 on every qubit, then CZ on a random matching).
"""
import math

import numpy as np
import torch

import qulacs_b200 as Q
from qulacs_b200.batch import BatchRunner

CUDA = "cuda"


def listed():
    return [
        # one step of a variational loop on a small molecule: all latency
        dict(name="vqe_10q", kind="circuit", ansatz="hea", n=10, depth=4, mode="staged", precision="c128", terms=30, weight=4),
        # the small random-circuit workload: 16 qubits, ten layers, 64 Pauli strings, default mode
        dict(name="layered_16q", kind="circuit", ansatz="layered", n=16, depth=10, mode="staged", precision="c128", terms=64, weight=4),
        # the plain method (one kernel per gate) on a state that fits the L2 cache, an odd qubit count
        dict(name="plain_21q", kind="circuit", ansatz="layered", n=21, depth=4, mode="gate_by_gate", precision="c128", terms=0, weight=0),
        # the large random-circuit workload: a 16 GiB state, fused execution
        dict(name="layered_30q", kind="circuit", ansatz="layered", n=30, depth=10, mode="staged_fused", precision="c128", terms=0, weight=0),
        # energy of a many-term Hamiltonian on a state much larger than L2
        dict(name="energy_28q", kind="energy", n=28, precision="c128", terms=256, weight=6),
        # reduced precision: a mid-size variational step, and the large U3 + CZ circuit
        dict(name="u3cz_23q_c64", kind="circuit", ansatz="u3cz", n=23, depth=20, mode="staged", precision="c64", terms=64, weight=4),
        dict(name="u3cz_30q_c64", kind="circuit", ansatz="u3cz", n=30, depth=20, mode="staged", precision="c64", terms=0, weight=0),
        # user-given multi-qubit unitaries, 3 to 6 targets at random positions
        dict(name="dense_25q", kind="dense", n=25, kmin=3, kmax=6),
        # noisy simulation on a density matrix (256 MiB)
        dict(name="noisy_12q", kind="noisy", n=12, depth=8, mode="staged_fused", p=0.001),
        # throughput: uneven small circuits with a Hamiltonian each, both precisions
        dict(name="batch_c128", kind="batch", circuits=64, nmin=10, nmax=20, depth_max=16, terms=200, weight=4, precision="c128"),
        dict(name="batch_c64", kind="batch", circuits=64, nmin=10, nmax=20, depth_max=16, terms=200, weight=4, precision="c64"),
        # shots from a 1 GiB state
        dict(name="sampling_26q", kind="sampling", n=26, shots=1024),
    ]


def draw(rng):
    kind = rng.choice(["circuit", "circuit", "circuit", "energy", "dense", "noisy", "batch", "sampling"])
    if kind == "circuit":
        c64 = rng.random() < 0.5
        mode = "staged" if c64 else rng.choice(["staged", "staged_fused", "gate_by_gate"])
        return dict(kind=kind, ansatz=rng.choice(["layered", "hea", "u3cz"]), n=rng.randint(4, 28),
                    depth=rng.randint(1, 20 if c64 else 10), mode=mode, precision="c64" if c64 else "c128",
                    terms=rng.choice([0, rng.randint(1, 128)]), weight=rng.randint(1, 6))
    if kind == "energy":
        return dict(kind=kind, n=rng.randint(4, 28), precision=rng.choice(["c128", "c64"]),
                    terms=int(round(2 ** rng.uniform(0, 8))), weight=rng.randint(1, 6))
    if kind == "dense":
        kmin = rng.randint(1, 6)
        return dict(kind=kind, n=rng.randint(8, 24), kmin=kmin, kmax=min(8, kmin + rng.randint(0, 3)))
    if kind == "noisy":
        return dict(kind=kind, n=rng.randint(2, 12), depth=rng.randint(1, 8),
                    mode=rng.choice(["staged", "staged_fused", "gate_by_gate"]), p=10 ** rng.uniform(-4, -1))
    if kind == "batch":
        nmin = rng.randint(4, 16)
        return dict(kind=kind, circuits=rng.randint(2, 64), nmin=nmin, nmax=min(20, nmin + rng.randint(0, 10)),
                    depth_max=rng.randint(4, 16), terms=rng.randint(1, 200), weight=rng.randint(1, 4),
                    precision=rng.choice(["c128", "c64"]))
    return dict(kind=kind, n=rng.randint(4, 28), shots=int(round(2 ** rng.uniform(0, 12))))


# ---- inputs, from the seed alone -------------------------------------------------------------------


def _gates(ansatz, n, depth, rng):
    """[("layer", [each qubit's [(kind, *angles)]]) | ("CNOT" | "CZ", a, b)] in program order."""
    out = []
    for _ in range(depth):
        if ansatz == "layered":
            out.append(("layer", [[(k, rng.uniform(0, 2 * math.pi)) for k in ("RX", "RY", "RZ")] for _ in range(n)]))
            out += [("CNOT", q, q + 1) for q in range(n - 1)]
        elif ansatz == "hea":
            out.append(("layer", [[(k, rng.uniform(0, 2 * math.pi)) for k in ("RY", "RZ")] for _ in range(n)]))
            out += [("CZ", q, (q + 1) % n) for q in range(n) if not (n == 2 and q == 1)]
        else:
            out.append(("layer", [[("U3", *rng.uniform(0, 2 * math.pi, 3))] for _ in range(n)]))
            perm = rng.permutation(n)
            out += [("CZ", int(perm[i]), int(perm[i + 1])) for i in range(0, n - 1, 2)]
    return out


def _terms(n, count, weight, rng):
    """(coefficient, qubits, Pauli ids 1..3) of `count` random strings."""
    out = []
    for _ in range(count):
        w = int(rng.integers(1, min(weight, n) + 1))
        qs = [int(q) for q in rng.choice(n, size=w, replace=False)]
        out.append((float(rng.normal()), qs, [int(p) for p in rng.integers(1, 4, size=w)]))
    return out


def _unitary(k, rng):
    m = 1 << k
    q, r = np.linalg.qr(rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def _dense_gates(case, seed):
    rng = np.random.default_rng([seed, 3])
    ks = range(case["kmin"], min(case["kmax"], case["n"]) + 1)
    return [([int(q) for q in rng.choice(case["n"], size=k, replace=False)], _unitary(k, rng)) for k in ks]


def _batch_jobs(case, seed):
    rng = np.random.default_rng([seed, 4])
    out = []
    for _ in range(case["circuits"]):
        n, depth = int(rng.integers(case["nmin"], case["nmax"] + 1)), int(rng.integers(4, case["depth_max"] + 1))
        out.append((n, depth, _gates("hea", n, depth, rng), _terms(n, case["terms"], case["weight"], rng)))
    return out


def _random_state(n, seed, dtype):
    """Normalised complex Gaussian amplitudes."""
    g = torch.Generator(device=CUDA).manual_seed(int(seed) * 7 + 1)
    v = torch.empty(1 << n, dtype=torch.complex64 if dtype == "c64" else torch.complex128, device=CUDA)
    torch.view_as_real(v).normal_(generator=g)
    return v.div_(torch.linalg.vector_norm(v))


# ---- a program's objects -----------------------------------------------------------------------------


class _Buffer:
    """A state's device memory for torch; the tensor made from it keeps it, and so the state, alive."""

    def __init__(self, state, shape, typestr):
        self.state = state
        self.__cuda_array_interface__ = dict(data=(state.data_ptr(), False), shape=shape, typestr=typestr, version=3)


def _tensor(state, c64=False, matrix=False):
    """The state's own device buffer as a tensor."""
    shape = (state.dim, state.dim) if matrix else (state.dim,)
    return torch.as_tensor(_Buffer(state, shape, "<c8" if c64 else "<c16"), device=CUDA)


def _circuit(gates, n, noise=None):
    c = Q.QuantumCircuit(n)
    add = c.add_gate if noise is None else (lambda g: c.add_noise_gate(g, "Depolarizing", noise))
    for g in gates:
        if g[0] == "layer":
            for q, ops in enumerate(g[1]):
                for kind, *a in ops:
                    add(getattr(Q.gate, kind)(q, *a))
        else:
            add(getattr(Q.gate, g[0])(g[1], g[2]))
    return c


def _observable(terms, n):
    obs = Q.Observable(n)
    for coef, qs, ids in terms:
        obs.add_operator(Q.PauliOperator(" ".join("%s %d" % ("IXYZ"[p], q) for q, p in zip(qs, ids)), coef))
    return obs


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "circuit":
        n, c64 = case["n"], case["precision"] == "c64"
        rng = np.random.default_rng([seed, 1])
        s["circuit"] = _circuit(_gates(case["ansatz"], n, case["depth"], rng), n)
        s["obs"] = _observable(_terms(n, case["terms"], case["weight"], rng), n) if case["terms"] else None
        s["state"] = Q.QuantumStateC64(n) if c64 else Q.QuantumState(n)
        s["out"] = _tensor(s["state"], c64)
    elif kind == "energy":
        n, c64 = case["n"], case["precision"] == "c64"
        s["obs"] = _observable(_terms(n, case["terms"], case["weight"], np.random.default_rng([seed, 2])), n)
        s["state"] = Q.QuantumStateC64(n) if c64 else Q.QuantumState(n)
        _tensor(s["state"], c64).copy_(_random_state(n, seed, case["precision"]))
    elif kind == "dense":
        n = case["n"]
        s["circuit"] = Q.QuantumCircuit(n)
        for qs, m in _dense_gates(case, seed):
            s["circuit"].add_dense_matrix_gate(qs, m)
        s["state"] = Q.QuantumState(n)
        s["out"] = _tensor(s["state"])
        s["out"].copy_(_random_state(n, seed, "c128"))
    elif kind == "noisy":
        n = case["n"]
        s["circuit"] = _circuit(_gates("hea", n, case["depth"], np.random.default_rng([seed, 1])), n, case["p"])
        s["state"] = Q.DensityMatrix(n)
        s["out"] = _tensor(s["state"], matrix=True)
    elif kind == "batch":
        s["runner"] = BatchRunner(32 << 30, precision=case["precision"])
        s["jobs"] = [(_circuit(gates, n), _observable(terms, n)) for n, _, gates, terms in _batch_jobs(case, seed)]
    else:
        s["state"] = Q.QuantumState(case["n"])
        _tensor(s["state"]).copy_(_random_state(case["n"], seed, "c128"))
        s["seed"] = seed
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "circuit":
        s["state"].set_zero_state()
        s["circuit"].update_quantum_state(s["state"], mode=case["mode"])
        if s["obs"] is None:
            return {"state": s["out"]}
        return {"state": s["out"], "energy": s["obs"].get_expectation_value(s["state"])}
    if kind == "energy":
        return {"energy": s["obs"].get_expectation_value(s["state"])}
    if kind == "dense":
        s["circuit"].update_quantum_state(s["state"])
        return {"state": s["out"]}
    if kind == "noisy":
        s["state"].set_zero_state()
        s["circuit"].update_quantum_state(s["state"], mode=case["mode"])
        return {"matrix": s["out"]}
    if kind == "batch":
        return {"energies": s["runner"].run(s["jobs"])}
    return {"indices": np.asarray(s["state"].sampling(case["shots"], s["seed"]), dtype=np.int64)}


# ---- what a pass cannot do without -------------------------------------------------------------------


def _rotations(ansatz, n, depth):
    """Rotations of a circuit that no identity merges: each is psi += i t P psi, 4 flop per amplitude."""
    return n * depth * (3 if ansatz == "layered" else 2)


def work(case):
    kind = case["kind"]
    if kind == "circuit":
        n, amp = case["n"], 8 if case["precision"] == "c64" else 16
        return {"bytes": amp * 2.0 ** n, "flops": (4.0 * _rotations(case["ansatz"], n, case["depth"]) + 2.0 * case["terms"]) * 2.0 ** n}
    if kind == "energy":
        return {"bytes": (8 if case["precision"] == "c64" else 16) * 2.0 ** case["n"], "flops": 2.0 * case["terms"] * 2.0 ** case["n"]}
    if kind == "dense":
        ks = range(case["kmin"], min(case["kmax"], case["n"]) + 1)
        return {"bytes": 32 * 2.0 ** case["n"], "flops": sum(8.0 * 2 ** k for k in ks) * 2.0 ** case["n"]}
    if kind == "noisy":
        n = case["n"]
        return {"bytes": 16 * 4.0 ** n, "flops": 4.0 * 2 * _rotations("hea", n, case["depth"]) * 4.0 ** n}
    if kind == "batch":  # the middle of the ranges
        n, depth = (case["nmin"] + case["nmax"]) / 2, (4 + case["depth_max"]) / 2
        amps = case["circuits"] * (2.0 ** (case["nmax"] + 1) - 2.0 ** case["nmin"]) / (case["nmax"] - case["nmin"] + 1)
        return {"bytes": (8 if case["precision"] == "c64" else 16) * amps, "flops": (8.0 * n * depth + 2.0 * case["terms"]) * amps}
    return {"bytes": 16 * 2.0 ** case["n"], "flops": 3 * 2.0 ** case["n"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "sampling":  # draws at a boundary of two cumulative sums
        return {"rel": 0.0, "differ": 0.004}
    reads_energy = kind == "energy" or case.get("terms", 0) > 0
    if case.get("precision") == "c64":
        if kind == "circuit":  # products of operands with 16 bits or more; energies of scrambled states cancel
            return {"rel": 1e-2, "max": 0.03} if reads_energy else {"rel": 3e-4, "max": 0.005}
        return {"rel": 1e-6, "max": 1e-5}  # 24-bit amplitudes, 53-bit sums
    # 53 bits through up to a thousand gates; energies of scrambled states cancel
    return {"rel": 1e-11, "max": 1e-9} if reads_energy else {"rel": 2e-13, "max": 1e-11}


# ---- the same results in plain 64-bit torch ----------------------------------------------------------


def _matrix(kind, *a):
    if kind == "U3":
        t, p, l = a
        c, s = math.cos(t / 2), math.sin(t / 2)
        return np.array([[c, -np.exp(1j * l) * s], [np.exp(1j * p) * s, np.exp(1j * (p + l)) * c]])
    c, s = math.cos(a[0] / 2), math.sin(a[0] / 2)
    return {"RX": np.array([[c, 1j * s], [1j * s, c]]), "RY": np.array([[c, s], [-s, c]], dtype=complex),
            "RZ": np.array([[c + 1j * s, 0], [0, c - 1j * s]])}[kind]


def _layer(v, mats, first=0):
    """mats[j] on bit first + j, four bits at a time."""
    for lo in range(0, len(mats), 4):
        m = np.ones((1, 1))
        for u in mats[lo:lo + 4]:
            m = np.kron(u, m)
        t = torch.from_numpy(np.ascontiguousarray(m)).to(CUDA)
        right = 1 << (first + lo)
        if right == 1:
            v = (v.view(-1, m.shape[0]) @ t.T).reshape(-1)
        else:
            v = torch.matmul(t, v.view(-1, m.shape[0], right)).reshape(-1)
    return v


def _pair(v, a, b):
    """View with the bits a and b as axes (…, a, …, b, …) in descending order, and whether a comes first."""
    hi, lo = max(a, b), min(a, b)
    return v.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo), a == hi


def _two(v, kind, a, b):
    w, first = _pair(v, a, b)
    if kind == "CZ":
        w[:, 1, :, 1].mul_(-1)
        return
    x, y = (w[:, 1, :, 0], w[:, 1, :, 1]) if first else (w[:, 0, :, 1], w[:, 1, :, 1])
    t = x.clone()
    x.copy_(y)
    y.copy_(t)


def _evolve(gates, n):
    v = torch.zeros(1 << n, dtype=torch.complex128, device=CUDA)
    v[0] = 1
    for g in gates:
        if g[0] == "layer":
            mats = []
            for ops in g[1]:
                m = np.eye(2)
                for kind, *a in ops:
                    m = _matrix(kind, *a) @ m
                mats.append(m)
            v = _layer(v, mats)
        else:
            _two(v, *g)
    return v


def _energy(v, terms, n):
    v = v.to(torch.complex128)
    size = min(1 << 24, 1 << n)
    base = torch.arange(size, device=CUDA)
    total = 0.0
    for coef, qs, ids in terms:
        x = sum(1 << q for q, p in zip(qs, ids) if p in (1, 2))
        z = sum(1 << q for q, p in zip(qs, ids) if p in (2, 3))
        val = torch.zeros((), dtype=torch.complex128, device=CUDA)
        for at in range(0, 1 << n, size):
            j = (base + at) ^ x
            par = j & z
            for sh in (16, 8, 4, 2, 1):
                par = par ^ (par >> sh)
            val += (v[at:at + size].conj() * v[j] * (1 - 2 * (par & 1))).sum()
        total += coef * (1j ** sum(p == 2 for p in ids) * complex(val)).real
    return total


def _trace_out(v, bits, total):
    """I / 2^k on `bits` times the trace over them, for a density matrix as a vector (column bits first)."""
    t = v.view([2] * total)
    for q in bits:
        a, b = total - 1 - q, total - 1 - (q + total // 2)
        diag = (t.select(a, 0).select(b if b < a else b - 1, 0) + t.select(a, 1).select(b if b < a else b - 1, 1)) / 2
        out = torch.zeros_like(t)
        for i in (0, 1):
            out.select(a, i).select(b if b < a else b - 1, i).copy_(diag)
        t = out
    return t.reshape(-1)


def _noisy(gates, n, p):
    v = torch.zeros(1 << (2 * n), dtype=torch.complex128, device=CUDA)
    v[0] = 1
    eye = np.eye(2)
    for g in gates:
        if g[0] == "layer":
            for q, ops in enumerate(g[1]):
                for kind, *a in ops:
                    m = _matrix(kind, *a)
                    v = torch.matmul(torch.from_numpy(m.conj()).to(CUDA), v.view(-1, 2, 1 << q)).reshape(-1)
                    v = torch.matmul(torch.from_numpy(m).to(CUDA), v.view(-1, 2, 1 << (q + n))).reshape(-1)
                    v = (1 - 4 * p / 3) * v + 4 * p / 3 * _trace_out(v, [q], 2 * n)
        else:
            _two(v, *g)
            _two(v, g[0], g[1] + n, g[2] + n)
            v = (1 - 16 * p / 15) * v + 16 * p / 15 * _trace_out(v, [g[1], g[2]], 2 * n)
    return v.view(1 << n, 1 << n)


def exact(case, seed):
    kind = case["kind"]
    if kind == "circuit":
        n = case["n"]
        rng = np.random.default_rng([seed, 1])
        gates = _gates(case["ansatz"], n, case["depth"], rng)
        terms = _terms(n, case["terms"], case["weight"], rng)
        v = _evolve(gates, n)
        return {"state": v, "energy": _energy(v, terms, n)} if terms else {"state": v}
    if kind == "energy":
        n = case["n"]
        terms = _terms(n, case["terms"], case["weight"], np.random.default_rng([seed, 2]))
        return {"energy": _energy(_random_state(n, seed, case["precision"]), terms, n)}
    if kind == "dense":
        n = case["n"]
        v = _random_state(n, seed, "c128")
        for qs, m in _dense_gates(case, seed):
            k = len(qs)
            axes = [n - 1 - q for q in reversed(qs)]  # the matrix index's bit j is qs[j]
            t = v.view([2] * n).movedim(axes, list(range(k))).reshape(1 << k, -1)
            t = (torch.from_numpy(m).to(CUDA) @ t).view([2] * n)
            v = t.movedim(list(range(k)), axes).reshape(-1)
        return {"state": v}
    if kind == "noisy":
        return {"matrix": _noisy(_gates("hea", case["n"], case["depth"], np.random.default_rng([seed, 1])), case["n"], case["p"])}
    if kind == "batch":
        return {"energies": np.array([_energy(_evolve(gates, n), terms, n) for n, _, gates, terms in _batch_jobs(case, seed)])}
    return None  # whole numbers only
