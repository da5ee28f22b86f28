"""The butterfly form of the pair (FP64) and fused (FP32) engines on the GPU, against the
per-gate engine, which is the reference CPU's arithmetic bit for bit."""
import numpy as np
import pytest

from svsim_b200 import circuits, gates as G
from test_plan import phase_circuit, shared_register

pytestmark = pytest.mark.gpu


def qft(n, seed):
    rng = np.random.default_rng(seed)
    gl = [G.U3(*rng.uniform(0, 6, 3), q) for q in range(n)]
    for i in range(n - 1, -1, -1):
        gl.append(G.H(i))
        gl += [G.CU1(np.pi / (1 << (i - j)), j, i) for j in range(i - 1, -1, -1)]
    return G.to_array(gl + [G.SWAP(q, n - 1 - q) for q in range(n // 2)])


def swaps(n):
    """Only label changes: passes without a redistribution, whose stores permute the tile."""
    return G.to_array([G.SWAP(q, n - 1 - q) for q in range(n // 2)] + [G.CZ(0, n - 1)])


@pytest.mark.parametrize("n,precision,make", [
    (12, 0, phase_circuit), (13, 1, qft), (17, 0, phase_circuit), (20, 0, qft), (20, 1, qft), (23, 0, qft), (24, 1, qft),
    (14, 0, lambda n, s: swaps(n)), (24, 0, lambda n, s: swaps(n)), (23, 1, lambda n, s: swaps(n)),
    (25, 0, lambda n, s: circuits.random_matching_circuit(n, 3, seed=s))])
def test_matches_the_per_gate_engine(n, precision, make):
    """From a random state, one tile to many tiles per CTA, run twice (the second time as a
    replayed graph), the second on a stream of its own: 2-norm error within one rounding a
    gate in quadrature, times 8."""
    import torch
    from svsim_b200 import _native as nat
    g = make(n, n)
    h = nat.Handle(n, 0, precision)
    h.set_engine(nat.ENGINE_BUTTERFLY)
    ref = nat.Handle(n, 0, nat.SVB_FP64)
    ref.set_engine(nat.ENGINE_PER_GATE)
    h.set_circuit(g)
    info = h.plan_info()
    assert info.engine == (nat.ENGINE_FUSED if precision else nat.ENGINE_PAIRS) and info.n_blocks == 0
    ref.set_circuit(g)
    if n <= 20:
        rng = np.random.default_rng(n)
        st = rng.standard_normal((2, 1 << n))
        st /= np.sqrt((st ** 2).sum())
        h.set_state(st[0], st[1])
        ref.set_state(st[0], st[1])
    stream = torch.cuda.Stream()
    for s in (0, stream.cuda_stream):
        h.run(s)
        h.sync()
        ref.run()
        ref.sync()
    eps = 1.2e-7 if precision else 2.2e-16
    bound = 8 * eps * np.sqrt(2 * max(len(g), 100))
    a = torch.as_tensor(Dev(h), device="cuda").double()
    b = torch.as_tensor(Dev(ref), device="cuda")
    assert float(torch.linalg.vector_norm(a - b)) <= bound * float(torch.linalg.vector_norm(b))


class Dev:
    """A handle's amplitudes as torch sees them, no copy."""

    def __init__(self, h):
        ptr, prec = h.device_ptr()
        self.h = h
        self.__cuda_array_interface__ = {"shape": (2 << h.n,), "typestr": "<f8" if prec == 0 else "<f4", "version": 3,
                                         "data": (ptr, False)}


def test_routes(oracle):
    """Which circuits go where: phase-rich ones to butterflies, random U3 + CX below 25 qubits
    and FP32 circuits with a fusion width to the tensor cores, SRN to the staged engine."""
    from svsim_b200 import _native as nat
    h = nat.Handle(16, 0, nat.SVB_FP64)
    h.set_circuit(circuits.random_matching_circuit(16, 4, seed=1))
    assert h.plan_info().n_blocks > 0
    h.set_circuit(qft(16, 1))
    assert h.plan_info().n_blocks == 0 and h.plan_info().engine == nat.ENGINE_PAIRS
    f = nat.Handle(16, 0, nat.SVB_FP32)
    f.set_circuit(qft(16, 1))
    assert f.plan_info().n_blocks == 0 and f.plan_info().engine == nat.ENGINE_FUSED
    f.set_engine(nat.ENGINE_FUSED, 0, 4)
    f.set_circuit(qft(16, 1))
    assert f.plan_info().n_blocks > 0
    h.set_circuit(G.to_array(G.from_array(qft(16, 1)) + [G.SRN(0)]))
    assert h.plan_info().engine == nat.ENGINE_STAGED
    # a new circuit while the last one may still run reuses the plan buffer
    h.set_circuit(qft(16, 2))
    h.reset()
    h.run()
    h.set_circuit(qft(16, 3))
    h.run()
    re, im = h.get_state()
    want = oracle.run(16, np.concatenate([qft(16, 2), qft(16, 3)]))
    assert np.max(np.abs(re - want[0])) < 1e-13 and np.max(np.abs(im - want[1])) < 1e-13


@pytest.mark.parametrize("n,t,y", [(13, 5, 2), (14, 9, 4), (16, 5, 2)])
def test_packed_control_onto_a_shared_register(oracle, n, t, y):
    """FP32, as the default dispatch runs it: a CX from qubit 0 onto a qubit whose register
    another one depends on.  The circuits move and negate amplitudes: FP32 rounding of the
    state only."""
    from svsim_b200 import _native as nat
    g = shared_register(n, t, y, 8)
    st = np.random.default_rng(n).standard_normal((2, 1 << n))
    st /= np.sqrt((st ** 2).sum())
    h = nat.Handle(n, 0, nat.SVB_FP32)
    h.set_circuit(g)
    assert h.plan_info().n_blocks == 0
    h.set_state(st[0], st[1])
    h.run()
    re, im = h.get_state()
    want = oracle.run(n, g, state=(st[0], st[1]))
    assert np.sqrt(np.sum((re - want[0]) ** 2 + (im - want[1]) ** 2)) <= 1.2e-7


def test_either_form_can_be_named(oracle):
    """The tensor-core engines by name run blocks where the default runs butterflies, and
    butterflies by name run where the default runs blocks; both give the same state."""
    from svsim_b200 import _native as nat
    from svsim_b200._native import SvbError
    random_circuit = circuits.random_matching_circuit(16, 4, seed=1)
    for prec, blocks, tol in ((nat.SVB_FP64, nat.ENGINE_PAIRS, 1e-13), (nat.SVB_FP32, nat.ENGINE_FUSED, 2e-6)):
        for g in (qft(16, 1), random_circuit):
            want = oracle.run(16, g)
            for engine in (nat.ENGINE_AUTO, blocks, nat.ENGINE_BUTTERFLY):
                h = nat.Handle(16, 0, prec)
                h.set_engine(engine)
                h.set_circuit(g)
                butterflies = engine == nat.ENGINE_BUTTERFLY or (engine == nat.ENGINE_AUTO and g is not random_circuit)
                assert (h.plan_info().n_blocks == 0) == butterflies and h.plan_info().engine == blocks
                h.run()
                re, im = h.get_state()
                assert np.max(np.abs(re - want[0])) < tol and np.max(np.abs(im - want[1])) < tol
    big = nat.Handle(25, 0, nat.SVB_FP64)
    big.set_engine(nat.ENGINE_PAIRS)
    big.set_circuit(circuits.random_matching_circuit(25, 2, seed=1))
    assert big.plan_info().n_blocks > 0
    for n, prec, gl in ((11, nat.SVB_FP64, [G.H(0)]), (12, nat.SVB_FP32, [G.H(0)]), (14, nat.SVB_FP64, [G.SRN(0)]),
                        (14, nat.SVB_FP64, [G.R(0.5, 0)])):
        h = nat.Handle(n, 0, prec)
        h.set_engine(nat.ENGINE_BUTTERFLY)
        with pytest.raises(SvbError):
            h.set_circuit(G.to_array(gl))


@pytest.mark.parametrize("precision", [0, 1])
def test_autotune_times_both_forms(precision):
    """The autotuner has both forms among its candidates, and its choice is a name that
    set_engine takes and that gives the plan AUTO then has."""
    from svsim_b200 import _native as nat
    n = 17                               # a structure that no other test leaves to AUTO
    g = qft(n, 1)
    h = nat.Handle(n, 0, precision)
    r = h.autotune(g)
    # per gate, three tile sizes, and the pair engine or the fused engine at four widths, and butterflies
    assert r.candidates == (6 if precision == 0 else 9)
    tuned = h.plan_info().n_blocks
    f = nat.Handle(n, 0, precision)
    f.set_engine(r.engine, r.tile_bits, r.fusion_width)
    f.set_circuit(g)
    assert f.plan_info().n_blocks == tuned and f.plan_info().engine == h.plan_info().engine


@pytest.mark.parametrize("engine,precision,n", [("BUTTERFLY", 0, 15), ("BUTTERFLY", 1, 15), ("PAIRS", 0, 14), ("FUSED", 1, 14),
                                                ("STAGED", 0, 14), ("PER_GATE", 0, 8)])
def test_a_run_on_a_side_stream_straight_after_the_upload(oracle, engine, precision, n):
    """set_circuit returns with the plan on the device: a run on a stream that does not wait for
    the default one, with circuits of different length in turn (a reused plan buffer would hold
    the earlier one's)."""
    import torch
    from svsim_b200 import _native as nat
    stream = torch.cuda.Stream()
    h = nat.Handle(n, 0, precision)
    h.set_engine(getattr(nat, "ENGINE_" + engine))
    want = None
    for i in range(12):
        g = circuits.random_matching_circuit(n, 2 + 5 * (i % 3), seed=i)
        want = oracle.run(n, g, state=want)
        h.set_circuit(g)
        h.run(stream.cuda_stream)
    stream.synchronize()
    re, im = h.get_state()
    tol = 1e-5 if precision else 1e-12
    assert np.max(np.abs(re - want[0])) < tol and np.max(np.abs(im - want[1])) < tol


@pytest.mark.parametrize("engine,n", [("PER_GATE", 8), ("BUTTERFLY", 16)])
def test_an_upload_does_not_wait_for_another_handle(engine, n):
    """set_circuit waits for its own handle's runs where it reuses their buffer: not for another
    handle's, here about half a second of them queued on a stream of their own."""
    import torch
    from svsim_b200 import _native as nat
    busy = nat.Handle(28, 0, nat.SVB_FP64)
    busy.set_circuit(circuits.random_matching_circuit(28, 20, seed=1))
    h = nat.Handle(n, 0, nat.SVB_FP64)
    h.set_engine(getattr(nat, "ENGINE_" + engine))
    own, side = torch.cuda.Stream(), torch.cuda.Stream()
    g = [circuits.random_matching_circuit(n, 3, seed=s) for s in range(2)]
    for b, depth in ((busy, 3), (h, 8)):     # what the first run loads, and a buffer for all
        b.set_circuit(circuits.random_matching_circuit(b.n, depth, seed=2))
        b.run(own.cuda_stream)
        b.sync()
    for _ in range(40):
        busy.run(side.cuda_stream)
    done = torch.cuda.Event()
    done.record(side)
    for i in range(4):
        h.set_circuit(g[i % 2])
        h.run(own.cuda_stream)
    h.set_circuit(g[0])
    assert not done.query()
    torch.cuda.synchronize()
