"""The calls that are timed: what users have the engine do, through its public entry points.

Sizes follow this repository's workloads (bench.py, workloads.py, the tests): brickwork
circuits up to 30 qubits and depth 40, QFT on a random state, the gate mix with Pauli
rotations, batched gradients of 16-qubit ansatz circuits, noisy trajectories, density
matrices, Pauli expectations, shot sampling, period finding, and single gates without fusion.

A case is a dict of plain values; ``kind`` says which call it is.  All amplitudes are
complex128 (the engine's only amplitude type).
"""
from __future__ import annotations

import cmath
import math
import random

import numpy as np
import torch

import litequantumcomputingsimulator_b200 as lq
from litequantumcomputingsimulator_b200 import algorithms, torch_ops
from litequantumcomputingsimulator_b200.simulator import CompiledCircuit

TAU = 2.0 * math.pi


def listed():
    return [
        # the smallest call: a textbook-size circuit sampled, all latency and launches
        {"name": "sample_8q", "kind": "sample", "qubits": 8, "depth": 4, "shots": 1024},
        # an ordinary sampled run: 620 gates, 4096 shots, state far smaller than L2
        {"name": "sample_20q", "kind": "sample", "qubits": 20, "depth": 20, "shots": 4096},
        # the largest: a compiled 1800-gate circuit applied to a 16 GiB state
        {"name": "brickwork_30q", "kind": "brickwork", "qubits": 30, "depth": 40},
        # diagonal-heavy circuit on a given state, an odd qubit count
        {"name": "qft_27q", "kind": "qft", "qubits": 27, "width": 27},
        # a state from |0..0>: dense gates, entanglers, rotations and Pauli strings mixed
        {"name": "mix_26q", "kind": "mix", "qubits": 26, "depth": 16},
        # interactive use: gates applied one at a time, no fusion (the streaming kernels)
        {"name": "gates_26q", "kind": "gates", "qubits": 26, "gates": 10},
        # a gradient batch: 256 parameter sets, 200 Pauli rotations, 500 Hamiltonian terms
        {"name": "gradient_16q", "kind": "gradient", "qubits": 16, "gates": 200, "terms": 500,
         "sets": 256, "grads": True},
        # one step of an optimiser: energy and gradient of one parameter set through autograd
        {"name": "vqe_step_10q", "kind": "vqe", "qubits": 10, "layers": 4},
        # an observable of many Pauli terms measured on a prepared state
        {"name": "expectation_24q", "kind": "expectation", "qubits": 24, "terms": 100},
        # noisy shots: depolarizing and amplitude-damping trajectories, 64 states resident
        {"name": "trajectories_22q", "kind": "trajectories", "qubits": 22, "depth": 20, "shots": 64},
        # exact noise: the density matrix of 10 qubits (a 2^20-element matrix)
        {"name": "density_10q", "kind": "density", "qubits": 10, "depth": 20},
        # period finding: controlled permutations, inverse QFT and 64 shots
        {"name": "period_21q", "kind": "period", "modulus": 119, "shots": 64},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["sample", "brickwork", "qft", "mix", "gates", "gradient", "vqe",
                       "expectation", "trajectories", "density", "period"])
    if kind == "sample":
        return {"kind": kind, "qubits": rng.randint(3, 24), "depth": log_int(1, 40),
                "shots": log_int(16, 16384)}
    if kind == "brickwork":
        return {"kind": kind, "qubits": rng.randint(12, 29), "depth": log_int(1, 40)}
    if kind == "qft":
        n = rng.randint(5, 28)
        return {"kind": kind, "qubits": n, "width": rng.randint(max(2, n - 12), n)}
    if kind == "mix":
        return {"kind": kind, "qubits": rng.randint(8, 27), "depth": log_int(1, 24)}
    if kind == "gates":
        return {"kind": kind, "qubits": rng.randint(6, 28), "gates": log_int(1, 60)}
    if kind == "gradient":
        return {"kind": kind, "qubits": rng.randint(5, 16), "gates": log_int(8, 200),
                "terms": log_int(1, 500), "sets": log_int(1, 256), "grads": rng.random() < 0.7}
    if kind == "vqe":
        return {"kind": kind, "qubits": rng.randint(3, 14), "layers": log_int(1, 8)}
    if kind == "expectation":
        return {"kind": kind, "qubits": rng.randint(5, 26), "terms": log_int(1, 200)}
    if kind == "trajectories":
        return {"kind": kind, "qubits": rng.randint(5, 22), "depth": log_int(1, 20),
                "shots": log_int(4, 64)}
    if kind == "density":
        return {"kind": kind, "qubits": rng.randint(3, 11), "depth": log_int(1, 20)}
    return {"kind": kind, "modulus": 2 * rng.randint(5, 110) + 1, "shots": log_int(16, 1024)}


# ---------------------------------------------------------------- workloads
# A circuit is a list of (name, angles, qubits[, pauli]); the same list drives the engine and
# the plain evaluation below.

def _angles(rng, k):
    return [TAU * rng.random() for _ in range(k)]


def _brickwork_layer(rng, n):
    ops = [("u", _angles(rng, 3), [q]) for q in range(n)]
    order = list(range(n))
    rng.shuffle(order)
    return ops + [("cx", [], order[k:k + 2]) for k in range(0, n - 1, 2)]


def _brickwork(rng, n, depth):
    return [op for _ in range(depth) for op in _brickwork_layer(rng, n)]


def _random_pauli(rng, w):
    return "".join(rng.choice("XYZ") for _ in range(w))


def _mix(rng, n, depth):
    ops = []
    for _ in range(n * depth):
        r = rng.random()
        if r < 0.5:
            ops.append(("u", _angles(rng, 3), [rng.randrange(n)]))
        elif r < 0.8:
            ops.append((rng.choice(["cx", "cz"]), [], rng.sample(range(n), 2)))
        elif r < 0.9:
            ops.append(("rzz", _angles(rng, 1), rng.sample(range(n), 2)))
        else:
            w = rng.randint(2, min(8, n))
            ops.append(("rp", [TAU * rng.random() - math.pi], rng.sample(range(n), w),
                        _random_pauli(rng, w)))
    return ops


def _qft(n):
    ops = []
    for i in range(n - 1, -1, -1):
        ops.append(("h", [], [i]))
        ops += [("cp", [math.pi / (1 << (i - j))], [j, i]) for j in range(i - 1, -1, -1)]
    return ops + [("swap", [], [i, n - 1 - i]) for i in range(n // 2)]


def _gates(rng, n, count):
    ops = []
    for k in range(count):
        q = rng.sample(range(n), 4)
        ops.append([("h", [], [q[0] if k else 0]), ("u", _angles(rng, 3), [q[0]]),
                    ("t", [], [q[0]]), ("cx", [], q[:2]), ("ccx", [], q[:3]),
                    ("h", [], [n - 1]), ("rzz", _angles(rng, 1), q[:2]), ("swap", [], q[:2]),
                    ("rp", _angles(rng, 1), q, _random_pauli(rng, 4)),
                    ("cp", _angles(rng, 1), q[:2])][k % 10])
    return ops


def _noisy(rng, n, depth):
    """Brickwork with the noise of the trajectory workload: depolarizing 1e-3 after each
    one-qubit gate, 1e-2 after each CX, amplitude damping 1e-3 per qubit and layer."""
    ops = []
    for _ in range(depth):
        for op in _brickwork_layer(rng, n):
            ops.append(op)
            ops += [("dep", [1e-3 if op[0] == "u" else 1e-2], [q]) for q in op[2]]
        ops += [("damp", [1e-3], [q]) for q in range(n)]
    return ops


def _circuit(n, ops, clbits=0):
    qc = lq.QuantumCircuit(n, clbits)
    channel = {}
    for name, p, q, *rest in ops:
        if name == "rp":
            qc.rp(p[0], rest[0], q)
        elif name in ("dep", "damp"):
            make = lq.KrausChannel.depolarizing if name == "dep" else lq.KrausChannel.amplitude_damping
            qc.kraus(channel.setdefault((name, p[0]), make(p[0])), q[0])
        else:
            getattr(qc, name)(*p, *q)
    return qc


def _hamiltonian(rng, n, terms):
    return [(rng.gauss(0.0, 1.0), "".join(rng.choice("IXYZ") for _ in range(n - 1)) + rng.choice("XYZ"))
            for _ in range(terms)]


def _ising(rng, n):
    z = [(rng.gauss(0.0, 1.0), "".join("Z" if q in (k, k + 1) else "I" for q in range(n)))
         for k in range(n - 1)]
    return z + [(rng.gauss(0.0, 1.0), "".join("X" if q == k else "I" for q in range(n)))
                for k in range(n)]


def _ansatz(case, rng):
    """[(pauli, qubits) of a rotation with a parameter, or ("cx", [control, target])]"""
    n = case["qubits"]
    if case["kind"] == "gradient":
        out = []
        for _ in range(case["gates"]):
            w = rng.randint(2, min(8, n))
            out.append((_random_pauli(rng, w), rng.sample(range(n), w)))
        return out
    out = []
    for _ in range(case["layers"]):
        out += [(p, [q]) for q in range(n) for p in "YZ"]
        out += [("cx", [q, q + 1]) for q in range(n - 1)]
    return out


def _parametric(n, ansatz):
    pc = lq.ParametricCircuit(n)
    for pauli, q in ansatz:
        if pauli == "cx":
            pc.cx(*q)
        elif len(q) == 1:
            (pc.ry if pauli == "Y" else pc.rz)(q[0])
        else:
            pc.rp(pauli, q)
    return pc


def _base(rng, modulus):
    while True:
        a = rng.randrange(2, modulus)
        if math.gcd(a, modulus) == 1:
            return a


def _random_state(amps, seed):
    """iid complex Gaussian amplitudes, normalised, into the device tensor `amps`."""
    g = torch.Generator(device=amps.device)
    g.manual_seed(seed)
    flat = torch.view_as_real(amps).view(-1)
    flat.normal_(generator=g)
    total = 0.0
    for part in flat.split(1 << 28):
        total += float(torch.dot(part, part))
    flat.mul_(1.0 / math.sqrt(total))
    return amps


def _ops(case, seed):
    """(circuit of a gate-list case, the generator after it)"""
    rng = random.Random(seed)
    kind, n = case["kind"], case["qubits"]
    if kind == "qft":
        return _qft(case["width"]), rng   # on the lowest qubits of the register
    if kind == "gates":
        return _gates(rng, n, case["gates"]), rng
    if kind == "mix":
        return _mix(rng, n, case["depth"]), rng
    if kind == "trajectories":
        return _noisy(rng, n, case["depth"]), rng
    return _brickwork(rng, n, case["depth"]), rng


# ---------------------------------------------------------------- the measured calls

def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "period":
        rng = random.Random(seed)
        modulus = case["modulus"]
        work = modulus.bit_length()
        count = 2 * work
        qc = lq.QuantumCircuit(count + work, count)
        qc.x(count)
        for j in range(count):
            qc.h(j)
        qc.compose(algorithms.modular_exponentiation(_base(rng, modulus), modulus, count, work))
        qc.compose(algorithms.qft_inverse(count))
        for j in range(count):
            qc.measure(j, j)
        state.update(circuit=qc, sim=lq.StatevectorSimulator(seed=seed), shots=case["shots"])
        return state
    n = case["qubits"]
    if kind in ("gradient", "vqe"):
        rng = random.Random(seed)
        ansatz = _ansatz(case, rng)
        state["ansatz"] = _parametric(n, ansatz)
        state["hamiltonian"] = _hamiltonian(rng, n, case["terms"]) if kind == "gradient" else _ising(rng, n)
        params = _parameters(case, seed, ansatz)
        if kind == "gradient":
            state.update(params=params, grads=case["grads"])
        else:
            state["params"] = torch.tensor(params[0], device="cuda", requires_grad=True)
        return state
    if kind == "expectation":
        state["hamiltonian"] = _hamiltonian(random.Random(seed), n, case["terms"])
        state["sv"] = lq.Statevector(n)
        _random_state(state["sv"].to_torch(), seed)
        return state
    ops, rng = _ops(case, seed)
    if kind in ("brickwork", "qft", "gates"):
        qc = _circuit(n, ops)
        state["sv"] = lq.Statevector(n)
        _random_state(state["sv"].to_torch(), seed)
        if kind == "brickwork":
            state["program"] = CompiledCircuit(qc)
        else:
            state["circuit"] = qc
        return state
    if kind == "mix":
        state.update(circuit=_circuit(n, ops), sim=lq.StatevectorSimulator())
        return state
    if kind == "density":
        noise = lq.NoiseModel().add_all_qubit_channel(lq.KrausChannel.depolarizing(1e-3))
        noise.add_all_qubit_channel(lq.KrausChannel.amplitude_damping(1e-3))
        state.update(circuit=_circuit(n, ops), sim=lq.DensityMatrixSimulator(noise=noise))
        return state
    qc = _circuit(n, ops, n)
    qc.measure_all()
    resident = 64 if kind == "trajectories" else 0
    state.update(circuit=qc, shots=case["shots"],
                 sim=lq.StatevectorSimulator(seed=seed, max_resident=resident))
    return state


def _parameters(case, seed, ansatz):
    k = sum(1 for pauli, _ in ansatz if pauli != "cx")
    sets = case.get("sets", 1)
    return (np.random.RandomState(seed % (1 << 32)).random_sample((sets, k)) * 2.0 - 1.0) * math.pi


def run(state):
    kind = state["kind"]
    if kind in ("sample", "trajectories", "period"):
        return state["sim"].run_registers(state["circuit"], state["shots"])
    if kind == "brickwork":
        return state["program"].apply(state["sv"]).to_torch()
    if kind == "qft":
        return state["sv"].apply(state["circuit"]).to_torch()
    if kind == "gates":
        return state["sv"].apply(state["circuit"], fuse_gates=False).to_torch()
    if kind == "mix":
        return state["sim"].run_statevector(state["circuit"]).to_torch()
    if kind == "expectation":
        return algorithms.expectation(state["sv"], state["hamiltonian"])
    if kind == "density":
        return state["sim"].run_density_matrix(state["circuit"]).probabilities()
    if kind == "gradient":
        call = algorithms.adjoint_gradient if state["grads"] else algorithms.batched_energy
        return call(state["hamiltonian"], state["ansatz"], state["params"])
    params = state["params"]
    params.grad = None
    energy = torch_ops.expectation(params, state["ansatz"], state["hamiltonian"])
    energy.backward()
    return energy.detach(), params.grad


# ---------------------------------------------------------------- work

def _flops(ops, n):
    """Real multiplies and adds of the gates one by one (2 x 2 gate: 14 per amplitude,
    rotation or diagonal: 6, phase: 6 on the amplitudes it changes, moves: none)."""
    per = {"u": 14.0, "h": 4.0, "t": 3.0, "cz": 0.5, "cp": 1.5, "rzz": 6.0, "rp": 6.0}
    return sum(per.get(op[0], 0.0) for op in ops) * float(1 << n)


def work(case):
    kind = case["kind"]
    if kind == "period":
        w = case["modulus"].bit_length()
        amps = float(1 << (3 * w))
        return {"bytes": 16.0 * amps + 8.0 * case["shots"], "flops": (4.0 * w + 1.5 * w * (2 * w - 1)) * amps}
    n = case["qubits"]
    amps = float(1 << n)
    if kind in ("gradient", "vqe"):
        k = case["gates"] if kind == "gradient" else 2 * n * case["layers"]
        terms = case["terms"] if kind == "gradient" else 2 * n - 1
        sets = case.get("sets", 1)
        back = 16.0 * k if case.get("grads", True) else 0.0
        return {"bytes": 16.0 * sets * (k + 1) + 16.0 * terms,
                "flops": amps * sets * (6.0 * k + 4.0 * terms + 4.0 + back)}
    if kind == "expectation":
        return {"bytes": 16.0 * amps, "flops": 4.0 * case["terms"] * amps}
    ops, _ = _ops(case, 1)
    flops = _flops(ops, n)
    if kind in ("brickwork", "qft", "gates"):
        return {"bytes": 32.0 * amps, "flops": flops}
    if kind == "density":
        # a gate on both sides; the 4 x 4 map of a channel has 8 non-zero entries
        touched = sum(len(op[2]) for op in ops)
        return {"bytes": 8.0 * amps, "flops": amps * (2.0 * flops + 2 * touched * 8.0 * amps)}
    if kind == "trajectories":
        return {"bytes": 8.0 * case["shots"], "flops": flops * case["shots"]}
    return {"bytes": 16.0 * amps + 8.0 * case.get("shots", 0), "flops": flops}


# ---------------------------------------------------------------- plain 64-bit evaluation

def _matrix(name, p):
    r = math.sqrt(0.5)
    if name == "h":
        return [[r, r], [r, -r]]
    c, s = math.cos(p[0] / 2), math.sin(p[0] / 2)   # u(theta, phi, lambda)
    return [[c, -cmath.exp(1j * p[2]) * s],
            [cmath.exp(1j * p[1]) * s, cmath.exp(1j * (p[1] + p[2])) * c]]


def _one_qubit(psi, m, q):
    v = psi.view(-1, 2, 1 << q)
    a, b = v[:, 0].clone(), v[:, 1].clone()
    v[:, 0] = m[0][0] * a + m[0][1] * b
    v[:, 1] = m[1][0] * a + m[1][1] * b


def _where(psi, fixed):
    """A view of the amplitudes whose qubits have the given bits: {qubit: bit}."""
    n = psi.numel().bit_length() - 1
    shape, index, above = [], [], n
    for q in sorted(fixed, reverse=True):
        shape += [1 << (above - 1 - q), 2]
        index += [slice(None), fixed[q]]
        above = q
    return psi.view(*shape, 1 << above)[tuple(index)]


def _exchange(psi, one, other):
    a, b = _where(psi, one), _where(psi, other)
    t = a.clone()
    a.copy_(b)
    b.copy_(t)


def _masks(pauli, qubits):
    """X, Z masks and the number of Y of a string whose last character acts on qubits[0]."""
    x = z = y = 0
    for ch, q in zip(reversed(pauli), qubits):
        x |= (ch in "XY") << q
        z |= (ch in "YZ") << q
        y += ch == "Y"
    return x, z, y


def _signs(index, z):
    v = index & z
    for s in (32, 16, 8, 4, 2, 1):
        v = v ^ (v >> s)
    return (1 - 2 * (v & 1)).to(torch.float64)


def _pauli(psi, index, x, z, y):
    """P psi for states along the last axis."""
    from_ = index ^ x
    out = psi[..., from_] if x else psi.clone()
    out *= _signs(from_, z)
    return out * (1, 1j, -1, -1j)[y % 4] if y % 4 else out


def _evolve(psi, ops, shift=0, conj=False):
    """The gates on `psi` in place; shift, conj: the bra side of a density matrix."""
    index = None
    for name, p, q, *rest in ops:
        q = [k + shift for k in q]
        if name in ("u", "h"):
            m = _matrix(name, p)
            _one_qubit(psi, [[complex(e).conjugate() if conj else e for e in row] for row in m], q[0])
        elif name == "cx":
            _exchange(psi, {q[0]: 1, q[1]: 0}, {q[0]: 1, q[1]: 1})
        elif name == "ccx":
            _exchange(psi, {q[0]: 1, q[1]: 1, q[2]: 0}, {q[0]: 1, q[1]: 1, q[2]: 1})
        elif name == "swap":
            _exchange(psi, {q[0]: 0, q[1]: 1}, {q[0]: 1, q[1]: 0})
        elif name in ("t", "cz", "cp"):
            ph = {"t": math.pi / 4, "cz": math.pi}.get(name, p[0] if p else 0.0)
            _where(psi, {k: 1 for k in q}).mul_(cmath.exp(1j * ph))
        elif name == "rzz":
            for bits in ((0, 0), (0, 1), (1, 0), (1, 1)):
                sign = 1 if bits[0] == bits[1] else -1
                _where(psi, dict(zip(q, bits))).mul_(cmath.exp(-0.5j * p[0] * sign))
        else:
            if index is None:
                index = torch.arange(psi.numel(), device=psi.device)
            moved = _pauli(psi, index, *_masks(rest[0], q))
            psi.mul_(math.cos(p[0] / 2)).add_(moved, alpha=-1j * math.sin(p[0] / 2))
    return psi


def _channel(rho, kraus, q, n):
    total = torch.zeros_like(rho)
    for k in kraus:
        part = rho.clone()
        _one_qubit(part, k, q)
        _one_qubit(part, [[complex(e).conjugate() for e in row] for row in k], q + n)
        total += part
    return total


def exact(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind in ("sample", "trajectories", "period"):
        return None   # whole numbers
    n = case["qubits"]
    if kind in ("gradient", "vqe"):
        return _exact_gradient(case, seed, dev)
    if kind == "expectation":
        psi = _random_state(torch.empty(1 << n, dtype=torch.complex128, device=dev), seed)
        index, total = torch.arange(1 << n, device=dev), 0.0
        for c, pauli in _hamiltonian(random.Random(seed), n, case["terms"]):
            total += c * float(torch.vdot(psi, _pauli(psi, index, *_masks(pauli, range(n)))).real)
        return total
    ops, _ = _ops(case, seed)
    if len(ops) * 16.0 * (1 << n) > 2e12 or n > 28:
        return None
    if kind == "density":
        rho = torch.zeros(1 << (2 * n), dtype=torch.complex128, device=dev)
        rho[0] = 1.0
        d, g = 1e-3, 1e-3
        a, b = math.sqrt(1.0 - 0.75 * d), math.sqrt(d / 4.0)
        noise = [[[[a, 0], [0, a]], [[0, b], [b, 0]], [[0, -1j * b], [1j * b, 0]], [[b, 0], [0, -b]]],
                 [[[1, 0], [0, math.sqrt(1.0 - g)]], [[0, math.sqrt(g)], [0, 0]]]]
        for op in ops:
            _evolve(rho, [op])
            _evolve(rho, [op], shift=n, conj=True)
            for kraus in noise:
                for q in op[2]:
                    rho = _channel(rho, kraus, q, n)
        return rho.view(1 << n, 1 << n).diagonal().real.clone()
    psi = torch.zeros(1 << n, dtype=torch.complex128, device=dev)
    if kind == "mix":
        psi[0] = 1.0
    else:
        _random_state(psi, seed)
    return _evolve(psi, ops)


def _exact_gradient(case, seed, dev):
    n = case["qubits"]
    rng = random.Random(seed)
    ansatz = _ansatz(case, rng)
    ham = _hamiltonian(rng, n, case["terms"]) if case["kind"] == "gradient" else _ising(rng, n)
    params = torch.tensor(_parameters(case, seed, ansatz), device=dev)
    sets = params.shape[0]
    index = torch.arange(1 << n, device=dev)
    psi = torch.zeros(sets, 1 << n, dtype=torch.complex128, device=dev)
    psi[:, 0] = 1.0

    def step(v, gate, k, sign):
        if gate[0] == "cx":
            c, t = gate[1]
            return v[:, index ^ (((index >> c) & 1) << t)]
        half = sign * params[:, k:k + 1] / 2
        return torch.cos(half) * v - 1j * torch.sin(half) * _pauli(v, index, *_masks(*gate))

    k = 0
    for gate in ansatz:
        psi = step(psi, gate, k, 1.0)
        k += gate[0] != "cx"
    lam = torch.zeros_like(psi)
    for c, pauli in ham:
        lam += c * _pauli(psi, index, *_masks(pauli, range(n)))
    energies = (psi.conj() * lam).sum(1).real
    if not case.get("grads", True):
        return energies
    grads = torch.zeros_like(params)
    for gate in reversed(ansatz):
        if gate[0] != "cx":
            k -= 1
            grads[:, k] = (lam.conj() * _pauli(psi, index, *_masks(*gate))).sum(1).imag
        psi, lam = step(psi, gate, k, -1.0), step(lam, gate, k, -1.0)
    return (energies, grads) if case["kind"] == "gradient" else (energies[0], grads[0])
