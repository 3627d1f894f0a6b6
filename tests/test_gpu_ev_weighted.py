"""sum_k c_k <P_k> from the weighted passes (no per-term values) against the oracle: every kind of
term evaluation (Z-only, bit flips within a thread's registers, partner amplitudes from shared memory,
per-thread selected rows, one value each), complex coefficients, complex128 and complex64 states."""
import numpy as np
import pytest

from conftest import EV_TOL, random_state
from qulacs_b200 import Observable, PauliOperator, QuantumState, QuantumStateC64
from qulacs_b200 import workloads as W
from qulacs_b200.observable import expectation_specialized_info, set_expectation_specialized

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["generic", "generated"])
def kernels(request):
    """Every test runs with the generic pass kernel and with per-pass kernels generated at first use."""
    set_expectation_specialized(0 if request.param == "generic" else 2)
    yield request.param
    set_expectation_specialized(1)


def observable(n, terms, coefs):
    obs = Observable(n)
    for c, (_, tl, ids) in zip(coefs, terms):
        obs.add_operator(PauliOperator(coef=c, targets=tl, pauli_ids=ids))
    return obs


def oracle_sum(port, a, terms, coefs):
    return sum(c * port.expectation_value(tl, ids, a) for c, (_, tl, ids) in zip(coefs, terms))


@pytest.mark.parametrize("n", [11, 12, 15, 19])
def test_weighted_matches_oracle_every_kind(port, n, kernels):
    rng = np.random.default_rng(9100 + n)
    a = random_state(n, rng)
    s = QuantumState(n)
    s.load(a)
    terms = W.random_pauli_terms(n, 150, 1, 6, seed=9200 + n)
    terms += [(0.0, [q], [1]) for q in range(4)]  # bit flips on qubits 0..3 alone
    terms += [(0.0, [int(q) for q in rng.choice(n, 3, replace=False)], [3, 3, 3]) for _ in range(10)]  # Z-only
    coefs = rng.normal(size=len(terms)) + 1j * rng.normal(size=len(terms))
    obs = observable(n, terms, coefs)
    plan = obs.weighted_plan()
    assert plan["passes"] >= 1
    for kind in ("z_only", "in_registers", "shared_partner", "selected_rows"):
        assert plan[kind] > 0, (kind, plan)
    launches0 = expectation_specialized_info()[0]
    got = obs.get_expectation_value_complex(s)
    launched = expectation_specialized_info()[0] - launches0
    assert (launched == plan["passes"]) if kernels == "generated" else (launched == 0)
    want = oracle_sum(port, a, terms, coefs)
    tol = EV_TOL * float(np.sum(np.abs(coefs)))
    assert abs(got - want) <= tol, (got, want)
    assert abs(obs.get_expectation_value(s) - want.real) <= tol
    # the per-term path gives the same sum
    vals = obs.term_values(s)
    assert abs(got - complex(np.sum(coefs * vals))) <= tol


def test_weighted_one_value_each_paths(port, kernels):
    """Below the tile size, with fewer than four bit-flip strings, and with strings that share no span:
    every term is evaluated alone and weighted on the host."""
    rng = np.random.default_rng(9300)
    for n, terms in [(8, W.random_pauli_terms(8, 30, 1, 4, seed=9301)),
                     (14, [(1.0, [0], [1]), (0.5, [3, 9], [2, 2]), (0.2, [1, 2], [3, 3])]),
                     (26, [(1.0, [q, q + 13], [1, 2]) for q in range(4, 13)])]:
        a = random_state(n, rng)
        s = QuantumState(n)
        s.load(a)
        coefs = rng.normal(size=len(terms))
        obs = observable(n, terms, coefs)
        want = oracle_sum(port, a, terms, coefs)
        assert abs(obs.get_expectation_value(s) - want.real) <= EV_TOL * float(np.sum(np.abs(coefs)))


def test_weighted_c64(port, kernels):
    n = 16
    rng = np.random.default_rng(9400)
    a = random_state(n, rng)
    s = QuantumStateC64(n)
    ref = QuantumState(n)
    ref.load(a)
    s.load(ref)
    a64 = s.get_vector().astype(np.complex128)  # the rounded amplitudes the kernel reads
    terms = W.random_pauli_terms(n, 120, 1, 6, seed=9401)
    coefs = rng.normal(size=len(terms))
    obs = observable(n, terms, coefs)
    want = oracle_sum(port, a64, terms, coefs)
    assert abs(obs.get_expectation_value(s) - want.real) <= EV_TOL * float(np.sum(np.abs(coefs)))


def test_weighted_repeatable(kernels):
    """The same call twice gives the same bits (fixed per-thread order, per-CTA partials folded in order)."""
    n = 18
    rng = np.random.default_rng(9500)
    s = QuantumState(n)
    s.load(random_state(n, rng))
    terms = W.random_pauli_terms(n, 200, 1, 6, seed=9501)
    obs = observable(n, terms, rng.normal(size=len(terms)))
    assert obs.get_expectation_value(s) == obs.get_expectation_value(s)


def test_generated_and_generic_agree_and_coefficients_reuse_kernels(port):
    """The generated kernels and the generic kernel give the same sum to rounding; new coefficients for
    the same strings reuse the generated kernels (no compile)."""
    n = 21
    rng = np.random.default_rng(9600)
    a = random_state(n, rng)
    s = QuantumState(n)
    s.load(a)
    terms = W.random_pauli_terms(n, 160, 1, 6, seed=9601)
    obs1 = observable(n, terms, rng.normal(size=len(terms)))
    set_expectation_specialized(0)
    generic = obs1.get_expectation_value(s)
    set_expectation_specialized(2)
    try:
        gen = obs1.get_expectation_value(s)
        assert abs(gen - generic) <= 1e-12
        coefs2 = rng.normal(size=len(terms))
        obs2 = observable(n, terms, coefs2)
        l0 = expectation_specialized_info()[0]
        e2 = obs2.get_expectation_value(s)
        assert expectation_specialized_info()[0] > l0
        want = oracle_sum(port, a, terms, coefs2).real
        assert abs(e2 - want) <= EV_TOL * float(np.sum(np.abs(coefs2)))
    finally:
        set_expectation_specialized(1)


def test_default_mode_generates_on_second_use():
    """Default policy: the first evaluation of a term list on >= 20 qubits runs the generic kernel, the
    second generates the pass kernels and runs them."""
    n = 20
    rng = np.random.default_rng(9700)
    s = QuantumState(n)
    s.load(random_state(n, rng))
    terms = W.random_pauli_terms(n, 64, 1, 5, seed=9701)
    obs = observable(n, terms, rng.normal(size=len(terms)))
    set_expectation_specialized(1)
    l0 = expectation_specialized_info()[0]
    e1 = obs.get_expectation_value(s)
    assert expectation_specialized_info()[0] == l0
    e2 = obs.get_expectation_value(s)
    assert expectation_specialized_info()[0] > l0
    assert abs(e1 - e2) <= 1e-12


def test_weighted_identity_repeated_and_zero_terms(port, kernels):
    """An identity term (coef x norm), the same string twice, a zero coefficient and a Y-only string:
    the weighted sum equals the oracle's."""
    n = 13
    rng = np.random.default_rng(9800)
    a = random_state(n, rng)
    s = QuantumState(n)
    s.load(a)
    terms = W.random_pauli_terms(n, 40, 1, 5, seed=9801)
    terms += [(0.0, [], []), terms[3], terms[7], (0.0, [2, 9], [2, 2]), (0.0, [0], [2])]
    coefs = rng.normal(size=len(terms))
    coefs[5] = 0.0
    obs = observable(n, terms, coefs)
    want = oracle_sum(port, a, terms, coefs).real
    assert abs(obs.get_expectation_value(s) - want) <= EV_TOL * float(np.sum(np.abs(coefs)))


@pytest.mark.parametrize("c64", [False, True])
@pytest.mark.parametrize("n,terms", [(1, 2), (2, 3), (5, 17), (10, 40), (11, 3), (17, 3)])
def test_small_state_strings_in_one_launch(port, n, terms, c64):
    """States below the pass evaluator (or with too few strings for it): every string of the call in one
    launch, Z-only strings 16 to a job, against the oracle."""
    rng = np.random.default_rng(300 + n)
    v = random_state(n, rng)
    if c64:
        v = v.astype(np.complex64).astype(np.complex128)
    s = QuantumStateC64(n) if c64 else QuantumState(n)
    s.load(v)
    ts = W.random_pauli_terms(n, terms, 1, min(4, n), seed=n)
    ts += [(0.5, [q], [3]) for q in range(n)]
    obs = W.to_observable(ts, n)
    want = np.array([port.expectation_value(tl, ids, v) for _, tl, ids in ts])
    assert np.max(np.abs(obs.term_values(s) - want)) <= EV_TOL
    assert abs(obs.get_expectation_value(s) - float(np.dot([t[0] for t in ts], want))) <= EV_TOL * len(ts)


@pytest.mark.parametrize("n", [1, 5, 12, 14])
@pytest.mark.parametrize("c64", [False, True])
def test_empty_sum_is_zero(lib, n, c64):
    """No terms at all, through the C entry points: 0, at every size."""
    import ctypes as C
    s = QuantumStateC64(n) if c64 else QuantumState(n)
    fn = lib.qs_expectation_value_pauli_weighted_c64 if c64 else lib.qs_expectation_value_pauli_weighted
    x, y, cf, out = (np.zeros(1, dtype=t) for t in (np.uint64, np.uint32, np.complex128, np.complex128))
    out[0] = 7.0
    p = [a.ctypes.data_as(C.c_void_p) for a in (x, y, cf, out)]
    assert fn(p[0], p[0], p[1], p[2], 0, s.data_ptr(), s.dim, None, p[3]) == 0
    assert out[0] == 0


@pytest.mark.parametrize("c64", [False, True])
@pytest.mark.parametrize("n", [1, 8, 12, 14, 17])
@pytest.mark.parametrize("flips,z_only", [(1, 0), (2, 0), (0, 1), (0, 16), (0, 17), (1, 1), (3, 5)])
def test_small_states_at_the_edges_of_one_launch(port, n, flips, z_only, c64):
    """Lists on both sides of the rule that sends a small state's strings out as one launch."""
    rng = np.random.default_rng(17 * n + flips + 3 * z_only)
    v = random_state(n, rng)
    if c64:
        v = v.astype(np.complex64).astype(np.complex128)
    s = QuantumStateC64(n) if c64 else QuantumState(n)
    s.load(v)
    ts = [(float(rng.normal()), [int(rng.integers(n))], [1 + i % 2]) for i in range(flips)]
    ts += [(float(rng.normal()), [int(rng.integers(n))], [3]) for _ in range(z_only)]
    obs = W.to_observable(ts, n)
    want = np.array([port.expectation_value(tl, ids, v) for _, tl, ids in ts])
    assert np.max(np.abs(obs.term_values(s) - want)) <= EV_TOL
    assert abs(obs.get_expectation_value(s) - float(np.dot([t[0] for t in ts], want))) <= EV_TOL * len(ts)


@pytest.mark.parametrize("c64", [False, True])
@pytest.mark.parametrize("n", [10, 11, 12])
@pytest.mark.parametrize("flips", [3, 4, 8, 9])
def test_few_strings_by_passes_or_in_one_launch(port, n, flips, c64):
    """Both sides of the rule that keeps 4 to 8 bit-flip strings at 11 and 12 qubits in passes, with Z-only ones."""
    rng = np.random.default_rng(31 * n + flips)
    v = random_state(n, rng)
    if c64:
        v = v.astype(np.complex64).astype(np.complex128)
    s = QuantumStateC64(n) if c64 else QuantumState(n)
    s.load(v)
    ts = []
    for i in range(flips):
        a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
        ts.append((float(rng.normal()), [a, b], [1 + i % 2, 1 + i % 3]))
    ts += [(0.5, [q], [3]) for q in range(2)]
    want = sum(t[0] * port.expectation_value(t[1], t[2], v) for t in ts)
    assert abs(W.to_observable(ts, n).get_expectation_value(s) - want) <= EV_TOL * len(ts)
