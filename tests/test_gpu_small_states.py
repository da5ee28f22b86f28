"""The per-gate engine on small states (one launch, the state in shared memory) and Pauli-sum
observables, against the oracle."""
import numpy as np
import pytest

from svsim_b200 import circuits, gates as G
from svsim_b200.gates import PAULI_DTYPE
from test_plan import mixed_circuit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count", [(1, 5), (2, 31), (5, 32), (6, 33), (7, 64), (9, 65), (10, 200), (11, 97), (12, 150)])
def test_small_states_are_the_reference_bit_for_bit(oracle, n, count):
    """Circuits of every op that fits n qubits, with op counts around the 32 staged at a time,
    from a random state; a second circuit uploaded over the first."""
    from svsim_b200 import _native as nat
    rng = np.random.default_rng(n)
    src = mixed_circuit(12, 4, seed=n)
    rows = []
    for g in src:
        k = G.N_QUBITS[G.OP_NAMES[int(g["op"])]]
        if k <= n:
            q = rng.permutation(n)[:k]
            g = g.copy()
            g["qb"] = tuple(int(x) for x in q) + (0,) * (5 - k)
            rows.append(g)
    g = np.array(rows[:count], dtype=src.dtype)
    st = rng.standard_normal((2, 1 << n))
    h = nat.Handle(n, 0, nat.SVB_FP64)
    h.set_engine(nat.ENGINE_PER_GATE)
    h.set_state(st[0], st[1])
    want = (st[0], st[1])
    for part in (g, g[::-1].copy()):
        h.set_circuit(part)
        h.run()
        want = oracle.run(n, part, state=want)
    re, im = h.get_state()
    assert np.array_equal(re, want[0]) and np.array_equal(im, want[1])


def random_terms(n, count, rng):
    t = np.zeros(count, dtype=PAULI_DTYPE)
    for k in range(count):
        kind = k % 4                         # Z strings, X strings, Y strings, any
        x = 0 if kind == 0 else int(rng.integers(1, 1 << n))
        z = int(rng.integers(0, 1 << n)) if kind in (0, 3) else (x if kind == 2 else 0)
        t[k] = (float(rng.normal()), x, z)
    return t


@pytest.mark.parametrize("n,count", [(1, 1), (1, 4), (2, 5), (5, 9), (7, 16), (10, 40), (13, 33), (18, 12)])
def test_pauli_sums(oracle, n, count):
    """Z, X, Y and mixed strings on states from two amplitudes to many blocks, by
    svb_expectation, in a batch and in the adjoint's energy.  Each term is a sum of 2^n products
    of a unit-norm state: 1e-14 a term of coefficient 1."""
    from svsim_b200 import _native as nat
    rng = np.random.default_rng(n + count)
    g = circuits.random_matching_circuit(n, 3, seed=n)
    t = random_terms(n, count, rng)
    re, im = oracle.run(n, g)
    want = oracle.expectation(n, re, im, t)
    bound = 1e-14 * float(np.sum(np.abs(t["coef"])))
    h = nat.Handle(n, 0, nat.SVB_FP64)
    h.set_circuit(g)
    h.run()
    assert abs(h.expectation(t) - want) <= bound
    b = nat.CircuitBatch([(n, g), (max(n - 1, 1), g[:0])], [t, None], tile_bits=10)
    e = b.run()
    assert abs(e[0] - want) <= bound and e[1] == 0.0
    binding = np.zeros(len(g), dtype=G.PARAM_DTYPE)
    binding["idx"] = -1
    ea, _ = h.adjoint(g, binding, 0, t)
    assert abs(ea - want) <= bound


@pytest.mark.parametrize("n", [1, 5, 13])
def test_pauli_sums_of_amplitudes_whose_squares_overflow(n):
    """X and Y strings multiply two different amplitudes: 1e200 and 1e-190 give a number where
    |1e200|^2 is none."""
    from svsim_b200 import _native as nat
    h = nat.Handle(n, 0, nat.SVB_FP64)
    re, im = np.full(1 << n, 1e-190), np.full(1 << n, 2e-190)
    re[0] = 1e200
    h.set_state(re, im)
    t = np.zeros(2, dtype=PAULI_DTYPE)
    t[0], t[1] = (0.5, 1, 0), (0.25, 1, 1)
    # <X_0> and <Y_0> of the pair (0, 1): 2 * 1e200 * 1e-190 and 2 * 1e200 * 2e-190
    assert abs(h.expectation(t) - (0.5 * 2e10 + 0.25 * 4e10)) <= 1e-4


def test_a_small_circuit_captured_into_the_callers_graph(oracle):
    """A run captured straight after its upload, replayed twice."""
    import torch
    from svsim_b200 import _native as nat
    n = 8
    g = circuits.random_matching_circuit(n, 6, seed=3)
    h = nat.Handle(n, 0, nat.SVB_FP64)
    h.set_engine(nat.ENGINE_PER_GATE)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    h.set_circuit(g)
    with torch.cuda.graph(graph, stream=side):
        h.run(side.cuda_stream)
    with torch.cuda.stream(side):
        graph.replay()
        graph.replay()
    side.synchronize()
    re, im = h.get_state()
    want = oracle.run(n, np.concatenate([g, g]))
    assert np.array_equal(re, want[0]) and np.array_equal(im, want[1])


@pytest.mark.parametrize("n,count", [(7, 4), (8, 3), (8, 4), (8, 300), (16, 5), (17, 3), (17, 4), (18, 4), (19, 3), (19, 4),
                                     (20, 9)])
@pytest.mark.parametrize("precision", [0, 1])
def test_pauli_sums_on_both_sides_of_the_lines_between_their_forms(oracle, n, count, precision):
    """One amplitude at a time and four at a time, by svb_expectation (19 qubits and 4 terms), in
    the adjoint (17) and in a batch, whose circuits then differ in their form (8): the oracle's
    sum, to 1e-14 a term of coefficient 1 (FP32: the state's rounding)."""
    from svsim_b200 import _native as nat
    rng = np.random.default_rng(n * 100 + count)
    g = circuits.random_matching_circuit(n, 3, seed=n)
    t = random_terms(n, count, rng)
    re, im = oracle.run(n, g)
    want = oracle.expectation(n, re, im, t)
    bound = (1e-14 if precision == 0 else 2e-6) * float(np.sum(np.abs(t["coef"])))
    h = nat.Handle(n, 0, precision)
    h.set_circuit(g)
    h.run()
    assert abs(h.expectation(t) - want) <= bound
    small = circuits.random_matching_circuit(3, 2, seed=1)
    ts = random_terms(3, 5, rng)
    b = nat.CircuitBatch([(n, g), (3, small), (2, small[:0])], [t, ts, None], precision=precision)
    e = b.run()
    assert abs(e[0] - want) <= bound and e[2] == 0.0
    assert abs(e[1] - oracle.expectation(3, *oracle.run(3, small), ts)) <= (1e-13 if precision == 0 else 1e-5)
    if precision == 0:
        binding = np.zeros(len(g), dtype=G.PARAM_DTYPE)
        binding["idx"] = -1
        ea, _ = h.adjoint(g, binding, 0, t)
        assert abs(ea - want) <= bound


def test_a_captured_run_keeps_its_circuit(oracle):
    """A graph that holds a run replays that circuit after the handle has others (of as many
    gates, so that any of the lists is one that the launch can read)."""
    import torch
    from svsim_b200 import _native as nat
    n = 8
    a, b, c = (circuits.random_matching_circuit(n, 6, seed=s) for s in range(3))
    h = nat.Handle(n, 0, nat.SVB_FP64)
    h.set_engine(nat.ENGINE_PER_GATE)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    h.set_circuit(a)
    with torch.cuda.graph(graph, stream=side):
        h.run(side.cuda_stream)
    for g in (b, c):
        h.set_circuit(g)
        h.run(side.cuda_stream)
    with torch.cuda.stream(side):
        graph.replay()
    h.run(side.cuda_stream)
    side.synchronize()
    re, im = h.get_state()
    want = oracle.run(n, np.concatenate([b, c, a, c]))
    assert np.array_equal(re, want[0]) and np.array_equal(im, want[1])
