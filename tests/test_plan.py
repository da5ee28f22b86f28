"""Host logic of the staged engine: plans executed on the CPU by tests/native's emulator
(the tile kernel's own index helpers) must reproduce the oracle."""
import ctypes
import math

import numpy as np
import pytest

from conftest import cx_dense_circuit, fidelity
from svsim_b200 import circuits, gates as G

_dp = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def emu():
    import build_emulator
    lib = ctypes.CDLL(build_emulator.build())
    return lib


def run_emu(lib, n, gates, M, precision=0, state=None):
    if state is None:
        re = np.zeros(1 << n)
        im = np.zeros(1 << n)
        re[0] = 1.0
    else:
        re, im = state[0].copy(), state[1].copy()
    np_, ns = ctypes.c_uint64(), ctypes.c_uint64()
    rc = lib.emu_staged_run(n, gates.ctypes.data, ctypes.c_size_t(len(gates)), M, precision,
                            re.ctypes.data_as(_dp), im.ctypes.data_as(_dp), ctypes.byref(np_),
                            ctypes.byref(ns))
    assert rc == 0, f"emulator rc {rc}"
    return re, im, np_.value


def mixed_circuit(n, reps, seed):
    rng = np.random.default_rng(seed)
    gl = G.from_array(circuits.random_matching_circuit(n, 1, seed=seed))
    for _ in range(reps):
        for name in G.OP_NAMES:
            qs = [int(x) for x in rng.permutation(n)[:G.N_QUBITS[name]]]
            npar = {"U3": 3, "U2": 2, "CU3": 3}.get(name, 1 if name in (
                "U1", "RX", "RY", "RZ", "CRX", "CRY", "CRZ", "CU1", "RXX", "RZZ", "RYY", "R") else 0)
            gl.append(G.FACTORIES[name](*([rng.uniform(-math.pi, math.pi) for _ in range(npar)] + qs)))
    return G.to_array(gl)


@pytest.mark.parametrize("n,M", [(10, 10), (12, 10), (12, 11), (12, 12), (13, 12), (15, 12)])
def test_staged_plan_random_matching_fp64(emu, oracle, n, M):
    g = circuits.random_matching_circuit(n, 10, seed=n * 31 + M)
    re, im, passes = run_emu(emu, n, g, M)
    ore, oim = oracle.run(n, g)
    assert np.max(np.abs(re - ore)) < 1e-13 and np.max(np.abs(im - oim)) < 1e-13
    assert passes < len(g)


@pytest.mark.parametrize("M", [10, 11, 12])
def test_staged_plan_every_op_fp64(emu, oracle, M):
    """All 38 ops, including the non-unitary SRN and R, interleaved at random."""
    n = 12
    g = mixed_circuit(n, 4, seed=M)
    re, im, _ = run_emu(emu, n, g, M)
    ore, oim = oracle.run(n, g)
    assert np.max(np.abs(re - ore)) < 1e-12 and np.max(np.abs(im - oim)) < 1e-12


@pytest.mark.parametrize("M", [11, 12, 13])
def test_staged_plan_every_op_fp32(emu, oracle, M):
    n = 13
    g = mixed_circuit(n, 3, seed=100 + M)
    re, im, _ = run_emu(emu, n, g, M, precision=1)
    ore, oim = oracle.run(n, g)
    assert 1 - fidelity(re + 1j * im, ore + 1j * oim) < 1e-6


def test_staged_plan_from_arbitrary_state(emu, oracle):
    n = 11
    rng = np.random.default_rng(5)
    st = (rng.standard_normal(1 << n), rng.standard_normal(1 << n))
    g = mixed_circuit(n, 2, seed=9)
    re, im, _ = run_emu(emu, n, g, 11, state=st)
    ore, oim = oracle.run(n, g, state=st)
    assert np.max(np.abs(re - ore)) < 1e-11 and np.max(np.abs(im - oim)) < 1e-11


def test_srn_is_ordered_against_complex_gates(emu, oracle):
    """SRN (svsim_nvgpu_sin.cuh:894-907) is only real-linear: moving it past a complex
    gate on another qubit changes the result, so the plan must not reorder it."""
    g = G.to_array([G.H(2), G.SRN(0), G.W(5), G.U2(-0.68, 0.36, 2)])
    re, im, _ = run_emu(emu, 12, g, 12)
    ore, oim = oracle.run(12, g)
    assert np.max(np.abs(re - ore)) < 1e-14 and np.max(np.abs(im - oim)) < 1e-14


def test_plan_pass_counts_headline_circuit(emu):
    """The n=30 depth-40 circuit (1,800 gates) needs far fewer passes than sweeps."""
    g = circuits.random_matching_circuit(30, 40)
    a, b, c, d = (ctypes.c_uint64() for _ in range(4))
    rc = emu.emu_plan_stats(30, g.ctypes.data, ctypes.c_size_t(len(g)), 12, 0, ctypes.byref(a),
                            ctypes.byref(b), ctypes.byref(c), ctypes.byref(d))
    assert rc == 0
    assert d.value == 1800
    assert a.value <= 80          # passes (each one read + one write of the state)


def run_fused_emu(lib, n, gates, k):
    re = np.zeros(1 << n)
    im = np.zeros(1 << n)
    re[0] = 1.0
    a, b = ctypes.c_uint64(), ctypes.c_uint64()
    rc = lib.emu_fused_run(n, gates.ctypes.data, ctypes.c_size_t(len(gates)), k,
                           re.ctypes.data_as(_dp), im.ctypes.data_as(_dp), ctypes.byref(a),
                           ctypes.byref(b))
    return rc, re, im, a.value, b.value


@pytest.mark.parametrize("n,k", [(12, 5), (13, 4), (14, 3), (15, 5)])
def test_fused_plan_random_matching(emu, oracle, n, k):
    """Fusion into k-qubit blocks, operand layouts and index tables of the tensor-core
    engine, executed on the CPU (MMA in FP64): only the FP32 rounding of the gates remains."""
    g = circuits.random_matching_circuit(n, 6, seed=n * 7 + k)
    rc, re, im, passes, blocks = run_fused_emu(emu, n, g, k)
    assert rc == 0
    ore, oim = oracle.run(n, g)
    assert 1 - fidelity(re + 1j * im, ore + 1j * oim) < 1e-12
    assert np.max(np.abs(re - ore)) < 1e-7 and blocks < len(g)


def test_fused_plan_every_op_but_srn(emu, oracle):
    n = 12
    g = mixed_circuit(n, 3, seed=21)
    g = g[g["op"] != G.OP["SRN"]]
    rc, re, im, _, _ = run_fused_emu(emu, n, g, 4)
    assert rc == 0
    ore, oim = oracle.run(n, g)
    assert 1 - fidelity(re + 1j * im, ore + 1j * oim) < 1e-12


def test_fused_plan_rejects_srn(emu):
    g = G.to_array([G.H(0), G.SRN(3)])
    rc, *_ = run_fused_emu(emu, 12, g, 4)
    assert rc == -3


def run_fused6_emu(lib, n, gates):
    re = np.zeros(1 << n)
    im = np.zeros(1 << n)
    re[0] = 1.0
    a = ctypes.c_uint64()
    rc = lib.emu_fused6_run(n, gates.ctypes.data, ctypes.c_size_t(len(gates)), re.ctypes.data_as(_dp),
                            im.ctypes.data_as(_dp), ctypes.byref(a))
    return rc, re, im, a.value


@pytest.mark.parametrize("n,depth", [(12, 6), (13, 5), (15, 4), (16, 3)])
def test_fused6_plan_random_matching(emu, oracle, n, depth):
    """Fusion width 6: greedy 6-qubit blocks (one per pass), the B-operand plane offsets,
    the canonical K-major reads of the MMA and the output offsets, executed on the CPU
    (MMA in FP64): only the TF32 hi + lo rounding of the gate remains."""
    g = circuits.random_matching_circuit(n, depth, seed=n * 11 + depth)
    rc, re, im, passes = run_fused6_emu(emu, n, g)
    assert rc == 0
    ore, oim = oracle.run(n, g)
    assert 1 - fidelity(re + 1j * im, ore + 1j * oim) < 1e-12
    assert np.max(np.abs(re - ore)) < 1e-7 and passes < len(g)


def test_fused6_plan_every_op_but_srn(emu, oracle):
    n = 13
    g = mixed_circuit(n, 3, seed=33)
    g = g[g["op"] != G.OP["SRN"]]
    rc, re, im, _ = run_fused6_emu(emu, n, g)
    assert rc == 0
    ore, oim = oracle.run(n, g)
    assert 1 - fidelity(re + 1j * im, ore + 1j * oim) < 1e-12


def test_fused6_plan_low_qubit_targets(emu, oracle):
    """Blocks whose targets include qubits 0 and 1 (both targets: the 2-way-conflict
    layout), only qubit 0, or neither, and blocks padded to 6 targets."""
    gl = []
    for q in range(12):
        gl.append(G.U3(0.3 + 0.1 * q, 0.2 * q, -0.4, q))
    gl += [G.CX(0, 1), G.CX(1, 5), G.CX(0, 7), G.U3(0.5, 0.1, 0.2, 0), G.CX(2, 3), G.CX(9, 11),
           G.CX(4, 13), G.H(12), G.CX(12, 0), G.RZ(0.7, 1), G.CX(10, 2)]
    g = G.to_array(gl)
    rc, re, im, _ = run_fused6_emu(emu, 14, g)
    assert rc == 0
    ore, oim = oracle.run(14, g)
    assert 1 - fidelity(re + 1j * im, ore + 1j * oim) < 1e-12


def test_fused6_plan_headline_circuit_blocks(emu):
    """n = 30, depth 40: 1,800 gates in at most 150 six-qubit blocks (passes), and at
    most 190 five-qubit blocks in 70 passes."""
    g = circuits.random_matching_circuit(30, 40, seed=2024)
    a, b = ctypes.c_uint64(), ctypes.c_uint64()
    rc = emu.emu_fused_stats(30, g.ctypes.data, ctypes.c_size_t(len(g)), 6, ctypes.byref(a), ctypes.byref(b))
    assert rc == 0
    assert a.value == b.value and a.value <= 150
    rc = emu.emu_fused_stats(30, g.ctypes.data, ctypes.c_size_t(len(g)), 5, ctypes.byref(a), ctypes.byref(b))
    assert rc == 0 and a.value <= 70 and b.value <= 190


def run_pairs_emu(lib, n, gates):
    re = np.zeros(1 << n)
    im = np.zeros(1 << n)
    st = np.zeros(4, dtype=np.uint64)
    vp = ctypes.c_void_p
    rc = lib.emu_pairs_run(ctypes.c_uint32(n), vp(gates.ctypes.data), ctypes.c_size_t(len(gates)),
                           vp(re.ctypes.data), vp(im.ctypes.data), vp(st.ctypes.data))
    return rc, re, im, st


@pytest.mark.parametrize("n,depth", [(12, 6), (13, 8), (16, 10), (17, 6)])
def test_pair_plan_random_matching(emu, oracle, n, depth):
    """Pair-engine plan (two-qubit blocks, lane/register exchanges, relayouts, tile-
    selected variants) run thread by thread with the kernel's data movement and MMA
    fragment rules, against the oracle."""
    g = circuits.random_matching_circuit(n, depth, seed=n + depth)
    rc, re, im, st = run_pairs_emu(emu, n, g)
    assert rc == 0, rc
    ore, oim = oracle.run(n, g)
    assert np.max(np.abs((re + 1j * im) - (ore + 1j * oim))) < 1e-13
    assert st[1] <= len(g)                  # no more blocks than gates


def test_pair_plan_every_op_but_srn_and_qaoa(emu, oracle):
    for n, g in [(15, mixed_circuit(15, 3, seed=31)),
                 (14, circuits.qaoa_instances(1, n_min=14, n_max=14, seed=5)[0].circuit()),
                 (16, circuits.brickwork_circuit(16, 20))]:
        g = g[g["op"] != G.OP["SRN"]]
        rc, re, im, _ = run_pairs_emu(emu, n, g)
        assert rc == 0, rc
        ore, oim = oracle.run(n, g)
        assert np.max(np.abs((re + 1j * im) - (ore + 1j * oim))) < 1e-13


def test_pair_plan_rejects_srn_and_small_states(emu):
    g = G.to_array([G.H(0), G.SRN(1)])
    assert run_pairs_emu(emu, 12, g)[0] == -6
    assert run_pairs_emu(emu, 11, G.to_array([G.H(0)]))[0] == -6


def test_pair_plan_shared_memory_staging(emu):
    """Every pass's ops and layouts, and its gate fragments where they fit, are copied
    into shared memory beside the 64 KiB tile: the largest copy stays within two CTAs per
    SM, the n=30 headline circuit stages every pass, and the CX-dense n=12 circuit (run on
    the GPU by test_pair_engine_pass_with_gates_beyond_shared_memory) has passes whose
    gates stay in global memory."""
    def stats(n, depth):
        g = circuits.random_matching_circuit(n, depth, seed=1)
        st = np.zeros(8, dtype=np.uint64)
        rc = emu.emu_pairs_stats(ctypes.c_uint32(n), ctypes.c_void_p(g.ctypes.data), ctypes.c_size_t(len(g)),
                                 ctypes.c_void_p(st.ctypes.data))
        assert rc == 0
        return st
    tile = 16 << 12
    for n, depth in ((12, 60), (20, 40), (30, 40)):
        st = stats(n, depth)
        assert tile + int(st[5]) <= 112 * 1024
    assert stats(30, 40)[4] == 0
    g = cx_dense_circuit()
    st = np.zeros(8, dtype=np.uint64)
    assert emu.emu_pairs_stats(ctypes.c_uint32(12), ctypes.c_void_p(g.ctypes.data), ctypes.c_size_t(len(g)),
                               ctypes.c_void_p(st.ctypes.data)) == 0
    assert st[4] >= 1 and tile + int(st[5]) <= 112 * 1024


def test_pair_plan_cx_dense_vs_oracle(emu, oracle):
    """The CX-dense circuit (passes whose gates stay in global memory) through the pair
    plan emulator."""
    g = cx_dense_circuit()
    rc, re, im, _ = run_pairs_emu(emu, 12, g)
    assert rc == 0, rc
    ore, oim = oracle.run(12, g)
    assert np.max(np.abs((re + 1j * im) - (ore + 1j * oim))) < 1e-13


# ---- every plan on a random input state -------------------------------------------------
# From |0..0>, an op that only multiplies amplitudes with some qubit at 1 (a phase on a
# non-local qubit, a tile-selected variant) is invisible until the state spreads; a plan that
# drops one passes every test that starts there.  These run each planner on circuits heavy
# in diagonal ops, from a random normalised state, against the oracle applied to that state.

def random_state(n, seed):
    rng = np.random.default_rng(seed)
    s = rng.normal(size=(2, 1 << n))
    s /= np.sqrt((s ** 2).sum())
    return s[0].copy(), s[1].copy()


def diagonal_heavy_circuit(n, m, seed):
    rng = np.random.default_rng(seed)
    gl = []
    for _ in range(m):
        r = rng.random()
        q = int(rng.integers(n))
        q2 = int(rng.integers(n - 1))
        q2 += q2 >= q
        if r < 0.3:
            gl.append(G.RZ(rng.uniform(-3, 3), q))
        elif r < 0.4:
            gl.append(G.T(q))
        elif r < 0.5:
            gl.append(G.U1(rng.uniform(-3, 3), q))
        elif r < 0.65:
            gl.append(G.CX(q, q2))
        elif r < 0.75:
            gl.append(G.CZ(q, q2))
        elif r < 0.85:
            gl.append(G.RY(rng.uniform(-3, 3), q))
        else:
            gl.append(G.U3(*rng.uniform(-3, 3, 3), q))
    return G.to_array(gl)


def ansatz_segment(n, lo, hi):
    """Ops lo..hi of the hardware-efficient ansatz: a segment that opens with a run of RZ
    (the adjoint's forward checkpoints cut the circuit like this)."""
    pc = circuits.hardware_efficient_ansatz(n=n, layers=2, seed=7)
    return np.ascontiguousarray(pc.evaluated(pc.params)[lo:hi])


STATE_CASES = [(n, diagonal_heavy_circuit(n, m, seed)) for n, m, seed in
               ((12, 60, 1), (13, 40, 2), (14, 80, 3), (15, 50, 4), (17, 90, 5))]
# n = 18, a pass of 12 local qubits: the segment's first RZ on 5 or more non-local qubits
# fill the tile phase twice over before any block
STATE_CASES += [(18, ansatz_segment(18, 22, 46)), (18, ansatz_segment(18, 58, 82))]


@pytest.mark.parametrize("case", range(len(STATE_CASES)))
def test_pair_plan_on_random_state(emu, oracle, case):
    n, g = STATE_CASES[case]
    re, im = random_state(n, case)
    ore, oim = oracle.run(n, g, state=(re, im))
    st = np.zeros(4, dtype=np.uint64)
    vp = ctypes.c_void_p
    rc = emu.emu_pairs_run_from(ctypes.c_uint32(n), vp(g.ctypes.data), ctypes.c_size_t(len(g)),
                                vp(re.ctypes.data), vp(im.ctypes.data), vp(st.ctypes.data))
    assert rc == 0
    assert np.max(np.abs((re + 1j * im) - (ore + 1j * oim))) < 1e-13


@pytest.mark.parametrize("case", range(len(STATE_CASES)))
def test_staged_plan_on_random_state(emu, oracle, case):
    n, g = STATE_CASES[case]
    st = random_state(n, case)
    ore, oim = oracle.run(n, g, state=st)
    for M in (10, 12):
        re, im, _ = run_emu(emu, n, g, M, state=st)
        assert np.max(np.abs((re + 1j * im) - (ore + 1j * oim))) < 1e-13, M


@pytest.mark.parametrize("case", range(len(STATE_CASES)))
def test_fused_plans_on_random_state(emu, oracle, case):
    n, g = STATE_CASES[case]
    st = random_state(n, case)
    ore, oim = oracle.run(n, g, state=st)
    for k in (3, 4, 5, 6):
        re, im = st[0].copy(), st[1].copy()
        if k < 6:
            a, b = ctypes.c_uint64(), ctypes.c_uint64()
            rc = emu.emu_fused_run(n, g.ctypes.data, ctypes.c_size_t(len(g)), k, re.ctypes.data_as(_dp),
                                   im.ctypes.data_as(_dp), ctypes.byref(a), ctypes.byref(b))
        else:
            a = ctypes.c_uint64()
            rc = emu.emu_fused6_run(n, g.ctypes.data, ctypes.c_size_t(len(g)), re.ctypes.data_as(_dp),
                                    im.ctypes.data_as(_dp), ctypes.byref(a))
        assert rc == 0, k
        assert 1 - fidelity(re + 1j * im, ore + 1j * oim) < 1e-12, k


def plan_cost(st):
    """The pair planner's cost model, in block units: blocks + 0.49 exchanges + 0.36 lane
    permutations + 2.05 relayouts + 0.6 passes."""
    return int(st[1]) + 0.49 * int(st[2]) + 0.36 * int(st[6]) + 2.05 * int(st[3]) + 0.6 * int(st[0])


@pytest.mark.parametrize("n,depth,seed", [(14, 12, 1), (18, 20, 2), (20, 40, 2024), (24, 40, 2024), (30, 40, 2024)])
def test_pair_plan_keeps_the_cheaper_pass_cut(emu, n, depth, seed):
    """plan_pairs plans the program-order and the seeded pass cut and keeps the cheaper by
    the cost model: never above the program-order plan; at n = 30 the seeded one (48
    passes against 50)."""
    g = circuits.random_matching_circuit(n, depth, seed=seed)
    both, one = np.zeros(8, dtype=np.uint64), np.zeros(8, dtype=np.uint64)
    vp = ctypes.c_void_p
    assert emu.emu_pairs_stats(ctypes.c_uint32(n), vp(g.ctypes.data), ctypes.c_size_t(len(g)), vp(both.ctypes.data)) == 0
    assert emu.emu_pairs_stats_one_cut(ctypes.c_uint32(n), vp(g.ctypes.data), ctypes.c_size_t(len(g)),
                                       vp(one.ctypes.data)) == 0
    assert plan_cost(both) <= plan_cost(one) + 1e-9
    if n == 30:
        assert int(one[0]) == 50 and int(both[0]) == 48 and plan_cost(both) < plan_cost(one)


def phase_circuit(n, seed, reps=2):
    """Controlled phases, CZ, RZZ and SWAPs between layers of every kind of one-qubit gate:
    the sequences the butterfly planner shortens, whole and interrupted."""
    rng = np.random.default_rng(seed)
    gl = G.from_array(circuits.random_matching_circuit(n, 1, seed=seed))
    for _ in range(reps):
        for a in range(n):
            gl.append(G.H(a))
            for b in rng.choice(n, size=min(4, n), replace=False):
                if int(b) == a:
                    continue
                t = float(rng.uniform(-3, 3))
                gl.append([lambda: G.CU1(t, a, int(b)), lambda: G.CZ(a, int(b)), lambda: G.RZZ(t, a, int(b)),
                           lambda: G.SWAP(a, int(b)), lambda: G.CX(a, int(b)), lambda: G.CRZ(t, a, int(b)),
                           lambda: G.RXX(t, a, int(b))][int(rng.integers(7))]())
            gl.append([G.X, G.T, G.Y, G.SDG][a % 4](int(rng.integers(n))))
    return G.to_array(gl)


def run_bfly(lib, n, gates, precision, seed=3):
    rng = np.random.default_rng(seed)
    st = rng.standard_normal((2, 1 << n))
    st /= np.sqrt((st ** 2).sum())
    re, im = st[0].copy(), st[1].copy()
    stats = (ctypes.c_uint64 * 8)()
    rc = lib.emu_bfly_run(n, gates.ctypes.data, ctypes.c_size_t(len(gates)), precision, 1, re.ctypes.data_as(_dp),
                          im.ctypes.data_as(_dp), stats)
    return rc, (re, im), st, list(stats)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,kind", [(12, "matching"), (13, "matching"), (16, "matching"), (13, "phases"), (15, "phases"),
                                    (13, "every"), (14, "every"), (14, "ansatz"), (15, "long")])
def test_butterfly_plan_from_random_states(emu, oracle, n, kind, precision):
    """The butterfly engine's plans, run thread by thread with the kernel's own arithmetic,
    from a random state: every op it takes (all but SRN and R), one tile and many, passes with
    and without redistributions, and circuits long enough to be cut at a pass's limits.  FP64
    within 8 ulps of a unit-norm state per hundred gates, FP32 within its own rounding."""
    if precision == 1 and n < 13:
        pytest.skip("an FP32 tile has 13 qubits")
    if kind == "matching":
        g = circuits.random_matching_circuit(n, 8, seed=n)
    elif kind == "phases":
        g = phase_circuit(n, seed=n)
    elif kind == "ansatz":
        g = circuits.hardware_efficient_ansatz(n, 4).gates
    elif kind == "long":
        g = np.concatenate([phase_circuit(n, seed=s, reps=6) for s in range(3)])
    else:
        g = mixed_circuit(n, 2, seed=n)
        g = g[(g["op"] != G.OP["SRN"]) & (g["op"] != G.OP["R"])]
    rc, got, st, stats = run_bfly(emu, n, g, precision)
    assert rc == 0 and stats[0] >= 1
    want = oracle.run(n, g, state=(st[0], st[1]))
    err = np.sqrt(np.sum((got[0] - want[0]) ** 2 + (got[1] - want[1]) ** 2))
    # 2-norm error: one rounding (eps / 2 of the norm at most) a gate, in quadrature, times 8
    eps = 2.2e-16 if precision == 0 else 1.2e-7
    assert err <= 8 * eps * np.sqrt(max(len(g), 100)), err


def test_butterfly_plan_rejects_what_it_cannot_split(emu):
    """SRN is not complex-linear, R not unitary: both stay on the other engines, as do states
    smaller than a tile."""
    for n, gl, precision in ((13, [G.SRN(1)], 0), (13, [G.R(0.5, 1)], 0), (11, [G.H(0)], 0), (12, [G.H(0)], 1)):
        assert run_bfly(emu, n, G.to_array(gl), precision)[0] == -5


@pytest.mark.parametrize("theta", [0.0, np.pi, 2 * np.pi, np.pi - 1e-9, 1e-9])
@pytest.mark.parametrize("precision", [0, 1])
def test_butterfly_plan_at_degenerate_angles(emu, oracle, theta, precision):
    """Gates whose split has a zero or vanishing diagonal (p = cos(theta / 2)): the scaled form."""
    n = 13
    gl = []
    for q in range(n):
        gl += [G.U3(theta, 0.3 * q, 1.1, q), G.CX(q, (q + 1) % n), G.RX(theta, (q + 3) % n), G.CX((q + 3) % n, q)]
    g = G.to_array(gl)
    rc, got, st, _ = run_bfly(emu, n, g, precision)
    want = oracle.run(n, g, state=(st[0], st[1]))
    err = np.sqrt(np.sum((got[0] - want[0]) ** 2 + (got[1] - want[1]) ** 2))
    assert rc == 0 and err <= 8 * (2.2e-16 if precision == 0 else 1.2e-7) * 10


def shared_register(n, t, y, phases):
    """CX(t -> y), after which y depends on t's register where y sits on a thread bit, then a CX
    from qubit 0, which FP32 packs two to a unit, onto t."""
    gl = [G.CX(t, y), G.CX(0, t)]
    return G.to_array(gl + [G.CZ(q, (q + 3) % n) for q in range(phases)])


@pytest.mark.parametrize("phases", [0, 8])
@pytest.mark.parametrize("n,t,y", [(13, 5, 2), (14, 9, 4), (16, 5, 2)])
def test_butterfly_plan_packed_control_onto_a_shared_register(emu, oracle, n, t, y, phases):
    """A packed control's CX waits for the next stage where another row shares the target's
    register: a row beside the packed one that differs between the halves of a unit has no
    address.  FP32 rounding only (the circuits move amplitudes and negate them)."""
    g = shared_register(n, t, y, phases)
    rc, got, st, _ = run_bfly(emu, n, g, 1)
    want = oracle.run(n, g, state=(st[0], st[1]))
    err = np.sqrt(np.sum((got[0] - want[0]) ** 2 + (got[1] - want[1]) ** 2))
    assert rc == 0 and err <= 1.2e-7


def short_circuit(n, rng):
    """A few gates of every kind the planner treats differently, on qubit 0 more than on others."""
    weights = ([4, 4, 0, 0, 0, 0, 0], [3, 1, 3, 2, 0, 0, 1], [4, 1, 1, 2, 2, 1, 1], [3, 0, 0, 1, 3, 1, 1])
    w = np.array(weights[int(rng.integers(4))], dtype=float)
    q = [0, 0] + list(range(n))
    gl = []
    for _ in range(int(2 ** rng.uniform(1, 6))):
        a = int(rng.choice(q))
        b = int(rng.choice([x for x in q if x != a]))
        t = float(rng.uniform(-3, 3))
        gl.append([lambda: G.CX(a, b), lambda: G.CZ(a, b), lambda: G.SWAP(a, b), lambda: G.H(a),
                   lambda: G.U3(*rng.uniform(0, 6, 3), a), lambda: G.CU1(t, a, b),
                   lambda: G.RX(t, a)][int(rng.choice(7, p=w / w.sum()))]())
    return G.to_array(gl)


@pytest.mark.parametrize("precision", [0, 1])
def test_butterfly_plan_on_random_short_circuits(emu, oracle, precision):
    """300 seeded circuits of a precision: few gates, so that what one stage leaves to the next
    differs from circuit to circuit."""
    eps = 2.2e-16 if precision == 0 else 1.2e-7
    for seed in range(300):
        rng = np.random.default_rng(seed)
        n = int(rng.integers(12, 15)) + precision
        g = short_circuit(n, rng)
        rc, got, st, _ = run_bfly(emu, n, g, precision, seed)
        want = oracle.run(n, g, state=(st[0], st[1]))
        err = np.sqrt(np.sum((got[0] - want[0]) ** 2 + (got[1] - want[1]) ** 2))
        assert rc == 0 and err <= 8 * eps * np.sqrt(100), (seed, rc, err)


def test_butterfly_plan_of_a_circuit_with_many_cuts(emu):
    """More than 32,767 passes: a period adds its own passes and gates and nothing else, so no
    cut takes a later one for the last that touches a qubit (which would apply what is pending,
    a phase a qubit)."""
    n = 13
    one = G.to_array([G.U3(0.3 + q, 0.2, 0.1, q) for q in range(n)] + [G.CX(q, (q + 1) % n) for q in range(n)])
    stats = {}
    for reps in (100, 200, 31000):
        g = np.tile(one, reps)
        st = (ctypes.c_uint64 * 8)()
        assert emu.emu_bfly_run(n, ctypes.c_void_p(g.ctypes.data), ctypes.c_size_t(len(g)), 0, 0, None, None, st) == 0
        stats[reps] = np.array([int(x) for x in st])
    period = stats[200] - stats[100]
    assert stats[31000][0] > 32767
    assert np.array_equal((stats[31000] - stats[100])[:4] * 100, period[:4] * 30900), stats


@pytest.mark.parametrize("precision,factor", [(1, 1.0), (1, 1e16), (1, 1e20), (1, 2e35), (0, 1e16), (0, 1e240), (0, 1e290)])
def test_butterfly_plan_keeps_large_amplitudes_finite(emu, oracle, precision, factor):
    """Gates with p = cos(theta / 2) = 0.02, which grow what is left unscaled most, between
    phases, on amplitudes up to `factor`: the same state to rounding, up to the range that
    bfly.h states."""
    n = 13
    gl = []
    for q in list(range(n)) * 2:
        gl += [G.U3(3.1, 0.2 * q, 0.1, q), G.CZ(q, (q + 1) % n), G.CZ(q, (q + 3) % n)]
    g = G.to_array(gl)
    st = np.random.default_rng(3).standard_normal((2, 1 << n))
    st /= np.sqrt(np.max(st[0] ** 2 + st[1] ** 2))
    re, im = st[0] * factor, st[1] * factor
    stats = (ctypes.c_uint64 * 8)()
    rc = emu.emu_bfly_run(n, ctypes.c_void_p(g.ctypes.data), ctypes.c_size_t(len(g)), precision, 1,
                          re.ctypes.data_as(_dp), im.ctypes.data_as(_dp), stats)
    want = oracle.run(n, g, state=(st[0], st[1]))
    err = np.sqrt(np.sum((re / factor - want[0]) ** 2 + (im / factor - want[1]) ** 2))
    norm = np.sqrt(np.sum(st ** 2))
    assert rc == 0 and err <= 8 * (2.2e-16 if precision == 0 else 1.2e-7) * np.sqrt(len(g) + 26) * norm


def fourier(n):
    gl = [G.U3(0.3 + 0.1 * q, 0.2, 0.1, q) for q in range(n)]
    for i in range(n - 1, -1, -1):
        gl += [G.H(i)] + [G.CU1(np.pi / (1 << (i - j)), j, i) for j in range(i - 1, -1, -1)]
    return G.to_array(gl + [G.SWAP(q, n - 1 - q) for q in range(n // 2)])


@pytest.mark.parametrize("make,n,depth,precision,form", [
    # butterflies / blocks measured: 1.32, 1.1, 0.94, 0.95, 0.94; 1.38, 1.18, 1.05; 0.56, 0.37, 0.35
    ("matching", 25, 2, 0, 0), ("matching", 28, 4, 0, 0), ("matching", 28, 30, 0, 1), ("matching", 30, 30, 0, 1),
    ("matching", 30, 40, 0, 1), ("brickwork", 25, 2, 0, 0), ("brickwork", 28, 4, 0, 0), ("brickwork", 26, 10, 0, 0),
    ("fourier", 16, 1, 0, 1), ("fourier", 24, 1, 0, 1), ("fourier", 25, 1, 0, 1), ("matching", 24, 25, 0, 0),
    ("fourier", 16, 1, 1, 1), ("matching", 24, 25, 1, 0)])
def test_default_form_is_the_faster_one(emu, make, n, depth, precision, form):
    """AUTO's choice between blocks and butterflies, for circuits whose two times lie apart:
    shallow random and brickwork circuits stay on blocks also from 25 qubits on."""
    g = {"matching": lambda: circuits.random_matching_circuit(n, depth, seed=1),
         "brickwork": lambda: circuits.brickwork_circuit(n, depth, seed=1), "fourier": lambda: fourier(n)}[make]()
    assert emu.emu_bfly_choice(ctypes.c_uint32(n), ctypes.c_void_p(g.ctypes.data), ctypes.c_size_t(len(g)),
                               precision) == form
