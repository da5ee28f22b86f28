"""Timed workloads of the framework, through its public entry points.

Every case is one thing a program that uses svsim_b200 has it do: run a circuit (of a
handle's own plan, or uploaded anew) and sample it, differentiate a parametrised circuit,
evaluate a batch of QAOA instances or of parameter points, or evolve a density matrix.
`listed` names the sizes that are looked at each time; `draw` gives others of the same
ranges.  Circuits, ansaetze and QAOA instances are the seeded ones of svsim_b200.circuits.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sv-sim_b200"))

from svsim_b200 import _native as nat  # noqa: E402
from svsim_b200 import circuits  # noqa: E402
from svsim_b200.autograd import adjoint_energy  # noqa: E402
from svsim_b200.density import DensityMatrix, depolarizing  # noqa: E402
from svsim_b200.gates import GATE_DTYPE, OP  # noqa: E402

NOISE = 0.01          # depolarizing probability after every gate of the density cases
LARGEST = 30          # qubits of the largest FP64 state vector


def listed():
    return [
        # the reference's unit tests and first steps of a user: a register of a few qubits,
        # the whole program (upload, run, sample) every time, so launches and the host count
        dict(name="circuit_n6", kind="circuit", recipe="mixed", n=6, depth=4, fp32=False, upload=True, shots=1024),
        # brickwork circuit of 16 qubits and 20 layers with 1,024 shots: a state that fits L2
        dict(name="circuit_n16", kind="circuit", recipe="brickwork", n=16, depth=20, fp32=False, upload=False,
             shots=1024),
        # an ordinary whole program at an odd size: gates up, run, samples back
        dict(name="program_n23", kind="circuit", recipe="matching", n=23, depth=20, fp32=False, upload=True,
             shots=1024),
        # the headline circuit: 30 qubits (16 GiB), depth 40
        dict(name="circuit_n30", kind="circuit", recipe="matching", n=30, depth=40, fp32=False, upload=False, shots=0),
        # quantum Fourier transform of a random product state: H, controlled phases, swaps
        dict(name="qft_n25", kind="circuit", recipe="qft", n=25, depth=1, fp32=False, upload=False, shots=4096),
        # single precision, small enough for L2, new gates every call
        dict(name="program_n19_fp32", kind="circuit", recipe="matching", n=19, depth=20, fp32=True, upload=True,
             shots=0),
        # single precision, large (2 GiB), depth 40
        dict(name="circuit_n28_fp32", kind="circuit", recipe="matching", n=28, depth=40, fp32=True, upload=False,
             shots=0),
        # one step of a variational loop: energy and gradient of the 20-qubit, 480-parameter ansatz
        dict(name="adjoint_n20", kind="adjoint", n=20, layers=12),
        # batched QAOA, 4 layers, n ~ U{10..22}: energies and gradients, both precisions
        dict(name="qaoa_fp64", kind="qaoa", count=192, n_min=10, n_max=22, p=4, fp32=False),
        dict(name="qaoa_fp32", kind="qaoa", count=512, n_min=10, n_max=22, p=4, fp32=True),
        # 64 parameter points of the 20-qubit ansatz with their energies
        dict(name="points_n20", kind="points", count=64, n=20, layers=12),
        # noisy circuit of 13 qubits as a density matrix (26-qubit vector), depth 10
        dict(name="density_n13", kind="density", n=13, depth=10),
    ]


def draw(rng):
    kind = rng.choice(["circuit"] * 6 + ["adjoint", "qaoa", "points", "density"])
    if kind == "circuit":
        n = rng.randint(5, 28)
        return dict(kind=kind, recipe=rng.choice(["matching", "matching", "brickwork", "mixed", "qft"]), n=n,
                    depth=rng.randint(2, 30), fp32=rng.random() < 0.35, upload=rng.random() < 0.5,
                    shots=rng.choice([0, 0, 1, 1000, 4096]))
    if kind == "adjoint":
        return dict(kind=kind, n=rng.randint(6, 21), layers=rng.randint(2, 12))
    if kind == "qaoa":
        lo = rng.randint(5, 14)
        return dict(kind=kind, count=int(2 ** rng.uniform(3, 8)), n_min=lo, n_max=rng.randint(lo, 21),
                    p=rng.randint(1, 5), fp32=rng.random() < 0.5)
    if kind == "points":
        return dict(kind=kind, count=int(2 ** rng.uniform(2, 6)), n=rng.randint(6, 20), layers=rng.randint(2, 12))
    return dict(kind=kind, n=rng.randint(4, 13), depth=rng.randint(2, 12))


# ---- inputs ------------------------------------------------------------------------------

def _rows(rows):
    g = np.zeros(len(rows), dtype=GATE_DTYPE)
    for i, (op, qb, ang) in enumerate(rows):
        g[i] = (OP[op], tuple(qb) + (0,) * (5 - len(qb)), *ang)
    return g


def _u3_all(rng, n):
    return [("U3", (q,), tuple(rng.uniform(0, 2 * math.pi, 3))) for q in range(n)]


def _qft(n, rng):
    """U3 on every qubit (a random product state), then the textbook Fourier transform."""
    rows = _u3_all(rng, n)
    for i in range(n - 1, -1, -1):
        rows.append(("H", (i,), (0, 0, 0)))
        for j in range(i - 1, -1, -1):
            rows.append(("CU1", (j, i), (0, 0, math.pi / (1 << (i - j)))))
    rows += [("SWAP", (q, n - 1 - q), (0, 0, 0)) for q in range(n // 2)]
    return _rows(rows)


def _mixed(n, depth, rng):
    """Layers of the one- and two-qubit gates a general program uses."""
    rows = _u3_all(rng, n)
    for _ in range(depth):
        for q in range(n):
            op = ("H", "T", "RX", "RY", "RZ", "S", "X", "SDG", "U2")[rng.integers(9)]
            a = float(rng.uniform(-math.pi, math.pi))
            ang = {"RX": (a, 0, 0), "RY": (a, 0, 0), "RZ": (0, a, 0), "U2": (0, a, a / 2)}.get(op, (0, 0, 0))
            rows.append((op, (q,), ang))
        perm = [int(x) for x in rng.permutation(n)]
        for a, b in zip(perm[0::2], perm[1::2]):
            op = ("CX", "CX", "CZ", "CU1", "RZZ", "SWAP")[rng.integers(6)]
            t = float(rng.uniform(-math.pi, math.pi))
            rows.append((op, (a, b), {"CU1": (0, 0, t), "RZZ": (t, 0, 0)}.get(op, (0, 0, 0))))
    return _rows(rows)


def _gates(case, seed):
    n, rng = case["n"], np.random.default_rng(seed)
    if case["recipe"] == "brickwork":
        return circuits.brickwork_circuit(n, case["depth"], seed=seed)
    if case["recipe"] == "qft":
        return _qft(n, rng)
    if case["recipe"] == "mixed":
        return _mixed(n, case["depth"], rng)
    return circuits.random_matching_circuit(n, case["depth"], seed=seed)


def _uniforms(case, seed):
    return np.random.default_rng(seed + 1).random(case["shots"])


def _instances(case, seed):
    return circuits.qaoa_instances(case["count"], case["n_min"], case["n_max"], case["p"], seed=seed)


def _points(case, seed):
    """The ansatz, as the batch is built with it, and the `count` parameter vectors that are run."""
    a = circuits.hardware_efficient_ansatz(case["n"], case["layers"], seed=seed)
    rng = np.random.default_rng(seed + 1)
    return a, rng.uniform(-math.pi, math.pi, size=(case["count"], len(a.params)))


class _State:
    """The amplitudes of a handle as torch sees them: no copy, and the handle stays alive."""

    def __init__(self, handle):
        ptr, prec = handle.device_ptr()
        self.handle = handle
        self.__cuda_array_interface__ = {"shape": (1 << handle.n, 2), "version": 3, "data": (ptr, False),
                                         "typestr": "<f8" if prec == nat.SVB_FP64 else "<f4"}


def _view(handle):
    return torch.as_tensor(_State(handle), device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "circuit":
        h = nat.Handle(case["n"], 0, nat.SVB_FP32 if case["fp32"] else nat.SVB_FP64)
        g = _gates(case, seed)
        if not case["upload"]:
            h.set_circuit(g)
        return dict(case=case, h=h, gates=g, u=_uniforms(case, seed), out=_view(h))
    if kind == "adjoint":
        a = circuits.hardware_efficient_ansatz(case["n"], case["layers"], seed=seed)
        return dict(case=case, h=nat.Handle(case["n"], 0, nat.SVB_FP64), circuit=a,
                    terms=circuits.zz_x_hamiltonian(case["n"]),
                    params=torch.tensor(a.params, dtype=torch.float64, requires_grad=True))
    if kind == "qaoa":
        inst = _instances(case, seed)
        return dict(case=case, b=nat.QaoaBatch(inst, precision=nat.SVB_FP32 if case["fp32"] else nat.SVB_FP64),
                    gammas=np.stack([i.gammas for i in inst]), betas=np.stack([i.betas for i in inst]))
    if kind == "points":
        a, points = _points(case, seed)
        batch = [(case["n"], a.gates)] * case["count"]
        terms = [circuits.zz_x_hamiltonian(case["n"])] * case["count"]
        return dict(case=case, b=nat.CircuitBatch(batch, terms),
                    gates=np.concatenate([a.evaluated(p) for p in points]))
    dm = DensityMatrix(case["n"])
    dm.set_circuit(circuits.random_matching_circuit(case["n"], case["depth"], seed=seed), kraus=depolarizing(NOISE))
    return dict(case=case, dm=dm, out=_view(dm.handle))


def run(state):
    kind = state["case"]["kind"]
    if kind == "circuit":
        h = state["h"]
        if state["case"]["upload"]:
            h.set_circuit(state["gates"])
        h.reset()
        h.run()
        if not len(state["u"]):
            return {"state": state["out"]}
        samples, total = h.measure(state["u"])
        if state["case"]["fp32"]:
            # a sample is an index of a CDF that FP32 rounding moves by many entries: the
            # outcome itself is no number two correct implementations share
            return {"state": state["out"], "total": total}
        return {"state": state["out"], "samples": samples.astype(np.int64), "total": total}
    if kind == "adjoint":
        e = adjoint_energy(state["params"], state["circuit"], state["terms"], state["h"])
        (grad,) = torch.autograd.grad(e, state["params"])
        return {"energy": e.detach(), "grad": grad}
    if kind == "qaoa":
        e, g = state["b"].run(state["gammas"], state["betas"])
        return {"energies": e, "grads": g}
    if kind == "points":
        return {"energies": state["b"].run(state["gates"])}
    state["dm"].handle.reset()
    state["dm"].handle.run()
    return {"rho": state["out"]}


# ---- what a pass cannot do without -------------------------------------------------------

def _gate_flops(gates, n):
    """A dense one-qubit gate is 14 flops per amplitude (two complex products and a sum), a
    phase 6 on the amplitudes it changes; X, CX and SWAP move amplitudes."""
    dim = float(1 << n)
    per = {OP["CX"]: 0, OP["SWAP"]: 0, OP["X"]: 0, OP["CZ"]: 0.5, OP["CU1"]: 1.5, OP["RZZ"]: 3, OP["T"]: 3,
           OP["S"]: 0, OP["SDG"]: 0, OP["RZ"]: 3, OP["RX"]: 6, OP["RY"]: 6, OP["H"]: 4}
    ops, counts = np.unique(gates["op"], return_counts=True)
    return float(sum(per.get(int(o), 14) * c for o, c in zip(ops, counts))) * dim


def work(case):
    kind = case["kind"]
    if kind == "circuit":
        g = _gates(case, 0)
        amp = (8 if case["fp32"] else 16) * float(1 << case["n"])
        # the final state is written once, and read once more to be sampled
        return {"bytes": amp * (2 if case["shots"] else 1) + g.nbytes, "flops": _gate_flops(g, case["n"])}
    if kind == "adjoint":
        a = circuits.hardware_efficient_ansatz(case["n"], case["layers"])
        # forward, then psi and lambda backwards; two inner products per layer and qubit
        return {"bytes": 2 * 16.0 * (1 << case["n"]) + a.gates.nbytes,
                "flops": 3 * _gate_flops(a.gates, case["n"]) + 8.0 * len(a.params) * (1 << case["n"])}
    if kind == "qaoa":
        amps = sum(float(1 << i.n) for i in _instances(case, 0))
        mean = (case["n_min"] + case["n_max"]) / 2
        # per layer: a phase (6) and an RX per qubit (6), forwards and on both states backwards
        return {"bytes": amps * (8 if case["fp32"] else 16) + 8.0 * case["count"] * (1 + 4 * case["p"]),
                "flops": 3 * case["p"] * amps * 6 * (1 + mean)}
    if kind == "points":
        a = circuits.hardware_efficient_ansatz(case["n"], case["layers"])
        return {"bytes": case["count"] * (16.0 * (1 << case["n"]) + a.gates.nbytes),
                "flops": case["count"] * _gate_flops(a.gates, case["n"])}
    g = circuits.random_matching_circuit(case["n"], case["depth"], seed=0)
    # U on both indices of rho, and a 2 x 2 mix of its blocks per noise channel
    qubits = float(np.sum(np.where(g["op"] == OP["CX"], 2, 1)))
    return {"bytes": 16.0 * 4 ** case["n"],
            "flops": 2 * _gate_flops(g, 2 * case["n"]) + 6 * qubits * float(4 ** case["n"])}


def tolerance(case):
    """About four times the relative error against `exact` that was measured (largest of the
    ranges): FP64 states 2e-15, energies and gradients 8e-15, noisy rho 1.1e-14; FP32 states
    2.9e-6 after 1,680 gates, FP32 energies and gradients 2.1e-6."""
    kind = case["kind"]
    if kind == "circuit" and case["fp32"]:
        return {"rel": 1.2e-5, "max": 2e-4}
    if kind == "circuit":
        # the samples: a CDF entry moves by the amplitudes' rounding
        return {"rel": 1.2e-14, "max": 1e-12, "differ": 0.005}
    if kind == "qaoa" and case["fp32"]:
        return {"rel": 1e-5, "max": 1e-3}
    if kind in ("adjoint", "points"):
        return {"rel": 4e-13, "max": 1e-11}    # an energy is a sum whose terms cancel: 4e-14 off where it is small
    return {"rel": 5e-14, "max": 2e-12}


# ---- the same in plain torch, 64 bits ----------------------------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _mat(op, th, ph, la):
    c, s, r = math.cos(th / 2), math.sin(th / 2), math.sqrt(0.5)

    def e(x):
        return complex(math.cos(x), math.sin(x))

    return {"U3": [[c, -e(la) * s], [e(ph) * s, e(ph + la) * c]], "U2": [[r, -e(la) * r], [e(ph) * r, e(ph + la) * r]],
            "H": [[r, r], [r, -r]], "X": [[0, 1], [1, 0]], "RX": [[c, -1j * s], [-1j * s, c]], "RY": [[c, -s], [s, c]],
            "T": [[1, 0], [0, e(math.pi / 4)]], "S": [[1, 0], [0, 1j]], "SDG": [[1, 0], [0, -1j]],
            "RZ": [[1, 0], [0, e(ph)]]}[op]


def _one(psi, q, m):
    v = psi.view(*psi.shape[:-1], -1, 2, 1 << q)
    a, b = v[..., 0, :].clone(), v[..., 1, :].clone()
    v[..., 0, :] = m[0][0] * a + m[0][1] * b
    v[..., 1, :] = m[1][0] * a + m[1][1] * b


def _four(psi, a, b):
    """Views of psi by (bit a, bit b): x[i][j]."""
    lo, hi = min(a, b), max(a, b)
    v = psi.view(*psi.shape[:-1], -1, 2, 1 << (hi - lo - 1), 2, 1 << lo)
    pick = [[v[..., i, :, j, :] for j in range(2)] for i in range(2)]     # [hi][lo]
    return pick if a == hi else [[pick[j][i] for j in range(2)] for i in range(2)]


def _swap_blocks(x, y):
    t = x.clone()
    x.copy_(y)
    y.copy_(t)


def _gate(psi, g, conj=False, shift=0):
    op = _NAMES[int(g["op"])]
    a, b = int(g["qb"][0]) + shift, int(g["qb"][1]) + shift
    th, ph, la = float(g["theta"]), float(g["phi"]), float(g["lam"])
    if op in ("CX", "CZ", "CU1", "RZZ", "SWAP"):
        x = _four(psi, a, b)
        if op == "CX":
            _swap_blocks(x[1][0], x[1][1])
        elif op == "SWAP":
            _swap_blocks(x[0][1], x[1][0])
        elif op == "CZ":
            x[1][1].neg_()
        elif op == "CU1":
            x[1][1].mul_(complex(math.cos(la), math.sin(la)))
        else:                                  # the reference's RZZ: e^{i theta} where the bits differ
            x[0][1].mul_(complex(math.cos(th), math.sin(th)))
            x[1][0].mul_(complex(math.cos(th), math.sin(th)))
        return
    m = _mat(op, th, ph, la)
    _one(psi, a, [[complex(z).conjugate() for z in r] for r in m] if conj else m)


_NAMES = {v: k for k, v in OP.items()}


def _zero(n, lead=()):
    psi = torch.zeros(*lead, 1 << n, dtype=torch.complex128, device=_dev())
    psi[..., 0] = 1
    return psi


def _samples(prob, u):
    cdf = torch.cumsum(prob, 0)
    j = torch.searchsorted(cdf, torch.from_numpy(u).to(cdf.device), right=True)
    return torch.where(j < len(cdf), j, 0).cpu().numpy()


def _hamiltonian(psi, n):
    """(sum_i Z_i Z_{i+1} + 0.5 sum_i X_i) psi."""
    z = torch.arange(1 << n, device=psi.device)
    d = torch.zeros(1 << n, dtype=torch.float64, device=psi.device)
    for i in range(n):
        d += 1.0 - 2.0 * (((z >> i) ^ (z >> ((i + 1) % n))) & 1)
    out = psi * d
    for i in range(n):
        out += 0.5 * psi.view(*psi.shape[:-1], -1, 2, 1 << i).flip(-2).reshape(psi.shape)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "circuit":
        if case["n"] > 28:
            return None                        # tens of seconds and 16 GiB and more of complex128
        psi = _zero(case["n"])
        for g in _gates(case, seed):
            _gate(psi, g)
        out = {"state": torch.view_as_real(psi).to(torch.float64)}
        if case["shots"]:
            p = psi.real ** 2 + psi.imag ** 2
            if not case["fp32"]:
                out["samples"] = _samples(p, _uniforms(case, seed))
            out["total"] = float(p.sum())
        return out
    if kind == "adjoint":
        a = circuits.hardware_efficient_ansatz(case["n"], case["layers"], seed=seed)
        psi = _zero(a.n)
        for g in a.gates:
            _gate(psi, g)
        lam = _hamiltonian(psi, a.n)
        energy = torch.vdot(psi, lam).real
        grad = np.zeros(len(a.params))
        for g, b in zip(a.gates[::-1], a.binding[::-1]):
            op, q = _NAMES[int(g["op"])], int(g["qb"][0])
            if op == "CX":
                _gate(psi, g)
                _gate(lam, g)
                continue
            t = psi.clone()
            if op == "RY":                     # d/dtheta = -i Y / 2
                _one(t, q, [[0, -0.5], [0.5, 0]])
                m, k = _mat("RY", -float(g["theta"]), 0, 0), int(b["idx"][0])
            else:                              # diag(1, e^{i phi}): d/dphi = i |1><1|
                _one(t, q, [[0, 0], [0, 1j]])
                m, k = _mat("RZ", 0, -float(g["phi"]), 0), int(b["idx"][1])
            grad[k] += 2 * float(torch.vdot(lam, t).real)
            _one(psi, q, m)
            _one(lam, q, m)
        return {"energy": energy, "grad": torch.from_numpy(grad)}
    if kind == "qaoa":
        es, gs = [], []
        for inst in _instances(case, seed):
            cost = torch.zeros(1 << inst.n, dtype=torch.float64, device=_dev())
            z = torch.arange(1 << inst.n, device=_dev())
            for (a, b), w in zip(inst.edges, inst.weights):
                cost += float(w) * (((z >> int(a)) ^ (z >> int(b))) & 1).to(torch.float64)
            psi = torch.full((1 << inst.n,), 2.0 ** (-inst.n / 2), dtype=torch.complex128, device=_dev())
            for ga, be in zip(inst.gammas, inst.betas):
                psi *= torch.exp(-1j * float(ga) * cost)
                for q in range(inst.n):
                    _one(psi, q, _mat("RX", 2 * float(be), 0, 0))
            lam = cost * psi
            es.append(torch.vdot(psi, lam).real)
            both, p = torch.stack([psi, lam]), len(inst.gammas)
            g = [None] * (2 * p)
            for k in range(p - 1, -1, -1):
                xs = sum(both[0].view(-1, 2, 1 << q).flip(1).reshape(-1) for q in range(inst.n))
                g[p + k] = 2 * torch.vdot(both[1], xs).imag
                for q in range(inst.n):
                    _one(both, q, _mat("RX", -2 * float(inst.betas[k]), 0, 0))
                g[k] = 2 * torch.vdot(both[1], cost * both[0]).imag
                both *= torch.exp(1j * float(inst.gammas[k]) * cost)
            gs.append(torch.stack(g))
        return {"energies": torch.stack(es), "grads": torch.stack(gs)}
    if kind == "points":
        a, points = _points(case, seed)
        out = []
        for first in range(0, len(points), 16):
            ps = points[first:first + 16]
            psi = _zero(a.n, (len(ps),))
            for g, b in zip(a.gates, a.binding):
                op, q = _NAMES[int(g["op"])], int(g["qb"][0])
                if op == "CX":
                    _gate(psi, g)
                    continue
                if op == "RY":
                    ms = np.array([_mat("RY", t, 0, 0) for t in ps[:, int(b["idx"][0])]], dtype=complex)
                else:
                    ms = np.array([_mat("RZ", 0, t, 0) for t in ps[:, int(b["idx"][1])]], dtype=complex)
                t = torch.from_numpy(ms).to(psi.device)
                _one(psi, q, [[t[:, i, j].view(-1, 1, 1) for j in range(2)] for i in range(2)])
            h = _hamiltonian(psi, a.n)
            out.append((psi.conj() * h).sum(-1).real)
        return {"energies": torch.cat(out)}
    n = case["n"]
    rho = _zero(2 * n)
    for g in circuits.random_matching_circuit(n, case["depth"], seed=seed):
        _gate(rho, g)
        _gate(rho, g, conj=True, shift=n)
        for q in {int(g["qb"][0])} | ({int(g["qb"][1])} if int(g["op"]) == OP["CX"] else set()):
            # depolarizing: (1 - 4p/3) rho + (4p/3) (1/2 on q, the rest traced over q)
            x = _four(rho, q, q + n)
            mix = (2 * NOISE / 3) * (x[0][0] + x[1][1])
            rho *= 1 - 4 * NOISE / 3
            x[0][0].add_(mix)
            x[1][1].add_(mix)
    return {"rho": torch.view_as_real(rho)}
