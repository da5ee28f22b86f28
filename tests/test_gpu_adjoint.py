"""Adjoint gradients (svb_adjoint) against central finite differences and the
parameter-shift rule, both evaluated with the plain FP64 path on the GPU, and the
energy against the oracle's state."""
import math

import numpy as np
import pytest

from svsim_b200 import circuits, gates as G

pytestmark = pytest.mark.gpu


def energy_plain(h, circuit, params, terms):
    h.reset()
    h.set_circuit(circuit.evaluated(params))
    h.run()
    return h.expectation(terms)


@pytest.fixture(scope="module")
def small_ansatz():
    return circuits.hardware_efficient_ansatz(n=10, layers=3, seed=3)


def test_energy_matches_oracle(oracle, small_ansatz):
    from svsim_b200 import _native as nat
    pc = small_ansatz
    terms = circuits.zz_x_hamiltonian(pc.n)
    h = nat.Handle(pc.n, 0, nat.SVB_FP64)
    e, _ = h.adjoint(pc.gates, pc.binding, len(pc.params), terms)
    re, im = oracle.run(pc.n, pc.gates)
    assert abs(e - oracle.expectation(pc.n, re, im, terms)) <= 1e-12
    # the handle holds psi(p) afterwards
    re2, im2 = h.get_state()
    assert np.max(np.abs(re2 - re)) <= 1e-12 and np.max(np.abs(im2 - im)) <= 1e-12


def test_gradient_vs_finite_differences_and_shift(small_ansatz):
    from svsim_b200 import _native as nat
    pc = small_ansatz
    terms = circuits.zz_x_hamiltonian(pc.n)
    h = nat.Handle(pc.n, 0, nat.SVB_FP64)
    _, g = h.adjoint(pc.gates, pc.binding, len(pc.params), terms)
    hp = nat.Handle(pc.n, 0, nat.SVB_FP64)
    step = 1e-6
    idx = np.random.default_rng(0).choice(len(pc.params), size=20, replace=False)
    for p in idx:
        pp = pc.params.copy()
        pp[p] += step
        ep = energy_plain(hp, pc, pp, terms)
        pp[p] -= 2 * step
        em = energy_plain(hp, pc, pp, terms)
        fd = (ep - em) / (2 * step)
        assert abs(fd - g[p]) <= 1e-7, (p, fd, g[p])
        # RY and RZ(=U1) are generated by Pauli/2: exact two-point shift of pi/2
        pp = pc.params.copy()
        pp[p] += math.pi / 2
        ep = energy_plain(hp, pc, pp, terms)
        pp[p] -= math.pi
        em = energy_plain(hp, pc, pp, terms)
        assert abs((ep - em) / 2 - g[p]) <= 1e-10


def test_composite_gates_differentiate(oracle):
    """Angles that enter through composites (CRZ, CU1, CU3, RXX, RZZ, RYY, CRX, CRY, U2)."""
    from svsim_b200 import _native as nat
    n = 6
    rng = np.random.default_rng(4)
    specs = [("CRZ", 1, 2), ("CU1", 1, 2), ("CU3", 3, 2), ("RXX", 1, 2), ("RZZ", 1, 2),
             ("RYY", 1, 2), ("CRX", 1, 2), ("CRY", 1, 2), ("U2", 2, 1), ("U3", 3, 1),
             ("RX", 1, 1), ("U1", 1, 1)]
    gl = list(G.from_array(circuits.random_matching_circuit(n, 1, seed=2)))
    binds = [(-1, -1, -1)] * len(gl)
    P = 0
    field_of = {"U3": (0, 1, 2), "CU3": (0, 1, 2), "U2": (1, 2), "U1": (2,), "CRX": (2,),
                "CRY": (2,), "CRZ": (2,), "CU1": (2,), "RXX": (0,), "RZZ": (0,), "RYY": (0,),
                "RX": (0,)}
    params = []
    for name, npar, nq in specs:
        qs = [int(x) for x in rng.permutation(n)[:nq]]
        vals = list(rng.uniform(-2, 2, npar))
        gl.append(G.FACTORIES[name](*(vals + qs)))
        b = [-1, -1, -1]
        for f, v in zip(field_of[name], vals):
            b[f] = P
            params.append(v)
            P += 1
        binds.append(tuple(b))
    gates = G.to_array(gl)
    bind = np.zeros(len(gl), dtype=G.PARAM_DTYPE)
    for i, b in enumerate(binds):
        bind[i]["idx"] = b
        bind[i]["coef"] = [1.0, 1.0, 1.0]
    pc = circuits.ParamCircuit(n, gates, bind, np.array(params))
    terms = circuits.zz_x_hamiltonian(n, 0.3)
    h = nat.Handle(n, 0, nat.SVB_FP64)
    _, g = h.adjoint(gates, bind, P, terms)
    hp = nat.Handle(n, 0, nat.SVB_FP64)
    for p in range(P):
        pp = pc.params.copy()
        pp[p] += 1e-6
        ep = energy_plain(hp, pc, pp, terms)
        pp[p] -= 2e-6
        em = energy_plain(hp, pc, pp, terms)
        assert abs((ep - em) / 2e-6 - g[p]) <= 1e-7, p


def test_non_unitary_rejected():
    from svsim_b200 import _native as nat
    h = nat.Handle(4, 0, nat.SVB_FP64)
    gates = G.to_array([G.H(0), G.SRN(1)])
    bind = np.zeros(2, dtype=G.PARAM_DTYPE)
    bind["idx"] = -1
    with pytest.raises(nat.SvbError) as e:
        h.adjoint(gates, bind, 0, circuits.zz_x_hamiltonian(4))
    assert e.value.status == nat.SVB_ERR_UNSUPPORTED


def test_torch_autograd(small_ansatz):
    import torch
    from svsim_b200 import _native as nat
    from svsim_b200.autograd import adjoint_energy
    pc = small_ansatz
    terms = circuits.zz_x_hamiltonian(pc.n)
    h = nat.Handle(pc.n, 0, nat.SVB_FP64)
    p = torch.tensor(pc.params, requires_grad=True)
    e = adjoint_energy(p, pc, terms, h)
    (3.0 * e).backward()
    _, g = nat.Handle(pc.n, 0, nat.SVB_FP64).adjoint(pc.gates, pc.binding, len(pc.params), terms)
    assert torch.allclose(p.grad, torch.from_numpy(3.0 * g), atol=1e-12)


def test_headline_ansatz_full_gradient():
    """n=20, 720 gates, 480 parameters: every component of the adjoint gradient against
    central finite differences (h = 1e-6, FP64, bar 1e-7) and the exact parameter-shift
    rule (RY and RZ = U1 are generated by Pauli/2), both on the plain FP64 path; two calls
    in a row (the second reuses the handle's scratch) give the same gradient."""
    from svsim_b200 import _native as nat
    pc = circuits.hardware_efficient_ansatz()
    terms = circuits.zz_x_hamiltonian(20)
    h = nat.Handle(20, 0, nat.SVB_FP64)
    e, g = h.adjoint(pc.gates, pc.binding, 480, terms)
    e2, g2 = h.adjoint(pc.gates, pc.binding, 480, terms)
    assert e == e2 and np.array_equal(g, g2)
    assert np.isfinite(e) and g.shape == (480,)
    hp = nat.Handle(20, 0, nat.SVB_FP64)
    assert abs(energy_plain(hp, pc, pc.params, terms) - e) <= 1e-12
    fd = np.empty(480)
    shift = np.empty(480)
    for p in range(480):
        pp = pc.params.copy()
        pp[p] += 1e-6
        ep = energy_plain(hp, pc, pp, terms)
        pp[p] -= 2e-6
        em = energy_plain(hp, pc, pp, terms)
        fd[p] = (ep - em) / 2e-6
        pp = pc.params.copy()
        pp[p] += math.pi / 2
        ep = energy_plain(hp, pc, pp, terms)
        pp[p] -= math.pi
        em = energy_plain(hp, pc, pp, terms)
        shift[p] = 0.5 * (ep - em)
    print(f"adjoint vs FD: max {np.max(np.abs(fd - g)):.3e}; vs parameter shift: "
          f"max {np.max(np.abs(shift - g)):.3e}")
    assert np.max(np.abs(fd - g)) <= 1e-7
    assert np.max(np.abs(shift - g)) <= 1e-10


@pytest.mark.parametrize("n,layers", [(14, 4), (20, 2)])
def test_energy_and_state_on_the_pair_engine_path(oracle, n, layers):
    """The forward segments run on the pair engine, split by checkpoints (224 and 120 ops):
    energy and the state left in the handle against the oracle, and the gradient against
    the per-gate path's finite differences.  At n = 20 a segment opens with RZ on 8 qubits
    that are not local in its first pass (their tile phases must all be applied)."""
    from svsim_b200 import _native as nat
    pc = circuits.hardware_efficient_ansatz(n=n, layers=layers, seed=5)
    terms = circuits.zz_x_hamiltonian(pc.n)
    h = nat.Handle(pc.n, 0, nat.SVB_FP64)
    e, g = h.adjoint(pc.gates, pc.binding, len(pc.params), terms)
    re, im = oracle.run(pc.n, pc.gates)
    assert abs(e - oracle.expectation(pc.n, re, im, terms)) <= 1e-12
    re2, im2 = h.get_state()
    assert np.max(np.abs(re2 - re)) <= 1e-12 and np.max(np.abs(im2 - im)) <= 1e-12
    hp = nat.Handle(pc.n, 0, nat.SVB_FP64)
    hp.set_engine(nat.ENGINE_PER_GATE, 0, 0)
    for p in range(0, len(pc.params), 7 if n <= 14 else 23):
        pp = pc.params.copy()
        pp[p] += 1e-6
        ep = energy_plain(hp, pc, pp, terms)
        pp[p] -= 2e-6
        em = energy_plain(hp, pc, pp, terms)
        assert abs((ep - em) / 2e-6 - g[p]) <= 1e-7, p


def test_sharded_parameter_points_single_rank(small_ansatz):
    """ShardedAdjoint's default evaluator on one GPU (no process group): a batch of
    parameter points gives each point's svb_adjoint energy and gradient, and the
    energy-only path (svb_run + svb_expectation) the same energies."""
    from svsim_b200 import _native as nat
    from svsim_b200.sharding import ShardedAdjoint
    pc = small_ansatz
    terms = circuits.zz_x_hamiltonian(pc.n)
    pts = np.random.default_rng(9).uniform(-np.pi, np.pi, size=(3, len(pc.params)))
    sa = ShardedAdjoint(pc, terms)
    e, g = sa.run(pts)
    e_only, none = sa.run(pts, gradients=False)
    sa.close()
    assert none is None
    h = nat.Handle(pc.n, 0, nat.SVB_FP64)
    for i, p in enumerate(pts):
        e_ref, g_ref = h.adjoint(pc.evaluated(p), pc.binding, len(p), terms)
        assert e[i] == e_ref and np.array_equal(g[i], g_ref)
        assert abs(e_only[i] - e_ref) <= 1e-12
        assert abs(energy_plain(h, pc, p, terms) - e_ref) <= 1e-12


@pytest.mark.parametrize("n", [9, 10, 11, 14])
def test_every_differentiated_kind(n):
    """U3, U2, U1, RX, RY, RZ and the composites that contain them, differentiated on low, high
    and (n > 10) non-local qubits, with fixed real, diagonal and complex gates in between:
    central differences of the plain path (step 1e-6: 1e-7)."""
    from svsim_b200 import _native as nat
    rng = np.random.default_rng(n)
    gl, idx, k = [], [], 0
    for layer in range(2):
        for q in range(n):
            kind = (q + 3 * layer) % 6
            a = rng.uniform(-3, 3, 3)
            g = [G.U3(*a, q), G.U2(a[0], a[1], q), G.U1(a[0], q), G.RX(a[0], q), G.RY(a[0], q), G.RZ(a[0], q)][kind]
            fields = [(0, 1, 2), (1, 2), (2,), (0,), (0,), (1,)][kind]
            gl.append(g)
            idx.append([(k + fields.index(f)) if f in fields else -1 for f in range(3)])
            k += len(fields)
        for q in range(0, n - 1, 2):
            t = float(rng.uniform(-3, 3))
            g = [G.CX(q, q + 1), G.RZZ(t, q, n - 1 - q if n - 1 - q != q else q + 1), G.CRY(t, q, q + 1), G.CU1(t, q + 1, q)][(q // 2) % 4]
            gl.append(g)
            f = {"RZZ": 0, "CRY": 2, "CU1": 2}.get(g.name)
            row = [-1, -1, -1]
            if f is not None:
                row[f] = k
                k += 1
            idx.append(row)
        for q in range(n):
            gl.append([G.H, G.T, G.X, G.S, G.Y, G.Z, G.W][(q + layer) % 7](q))
            idx.append([-1, -1, -1])
    gates = G.to_array(gl)
    binding = np.zeros(len(gates), dtype=G.PARAM_DTYPE)
    binding["idx"] = np.array(idx)
    binding["coef"] = 1.0
    params = np.zeros(k)
    for g, row in zip(gates, idx):
        for f, name in enumerate(("theta", "phi", "lam")):
            if row[f] >= 0:
                params[row[f]] = g[name]
    pc = circuits.ParamCircuit(n, gates, binding, params)
    terms = circuits.zz_x_hamiltonian(n)
    h = nat.Handle(n, 0, nat.SVB_FP64)
    _, grad = h.adjoint(gates, binding, k, terms)
    hp = nat.Handle(n, 0, nat.SVB_FP64)
    for p in range(k):
        e = []
        for s in (1e-6, -1e-6):
            pp = params.copy()
            pp[p] += s
            e.append(energy_plain(hp, pc, pp, terms))
        assert abs((e[0] - e[1]) / 2e-6 - grad[p]) <= 1e-7, (p, grad[p])
