"""Register passes in rotation form: one-qubit gates as diagonal, real rotation, diagonal;
CX as CZ between two H; negated and sign-carrying tile bits.

The circuits collect what the factoring has special cases for: exact X, Y and anti-diagonal
gates (bits stored negated), rotations by 0, pi/2 and pi, angles next to them, runs of one-qubit
gates that multiply to the identity, CX with and without neighbours on the target, chains of CX
on one target, CZ and CP whose qubits lie in the tile, half outside and outside, more sign masks
than a pass's sign word holds, RZZ next to and away from one-qubit gates, SWAPs, controlled
gates that look at a bit (which may then not be negated), and Pauli rotations on negated bits.

Tolerance: 1e-12 per amplitude, the engine's bound against the oracle.
"""
import math

import numpy as np
import pytest

import litequantumcomputingsimulator_b200 as lq
from litequantumcomputingsimulator_b200 import workloads as W
from test_reg_emulation import PLANNED, emulate

TOL = 1e-12
EDGE_ANGLES = [0.0, math.pi / 2, math.pi, -math.pi, 1e-9, math.pi - 1e-9, 2 * math.pi]


def edge_circuit(n, n_gates, seed):
    rng = np.random.default_rng(seed)
    qc = lq.QuantumCircuit(n)

    def angle():
        return float(rng.choice(EDGE_ANGLES)) if rng.random() < 0.5 else float(rng.uniform(-7, 7))

    for _ in range(n_gates):
        a, b, c, d = (int(v) for v in rng.permutation(n)[:4])
        k = int(rng.integers(20))
        if k < 5:
            getattr(qc, ["x", "y", "h", "t", "sx"][k])(a)
        elif k < 8:
            getattr(qc, ["rx", "ry", "rz"][k - 5])(angle(), a)
        elif k < 11:
            qc.u(angle(), angle(), angle(), a)
        elif k < 13:
            qc.cx(a, b)
        elif k == 13:
            qc.cz(a, b)
        elif k == 14:
            qc.rzz(angle(), a, b)
        elif k == 15:
            qc.swap(a, b)
        elif k == 16:
            qc.ccx(a, b, c)
        elif k == 17:
            (qc.crx if rng.random() < 0.5 else qc.crz)(angle(), a, b)
        elif k == 18:
            (qc.iswap if rng.random() < 0.5 else qc.cy)(a, b)
        else:
            qc.rp(angle(), "XYZ"[int(rng.integers(3))] + "ZY" + "X", [a, b, c, d])
    return qc


def cz_layers(n, layers, seed):
    """Rotations on every qubit between layers of CZ on every pair of neighbours in a random
    order: far more signs per pass than its sign word holds."""
    rng = np.random.default_rng(seed)
    qc = lq.QuantumCircuit(n)
    for _ in range(layers):
        for q in range(n):
            qc.ry(float(rng.uniform(-3, 3)), q)
        order = rng.permutation(n)
        for k in range(n - 1):
            qc.cz(int(order[k]), int(order[k + 1]))
    return qc


def ladder(n, seed):
    """CX chains on one target, runs that multiply to the identity, and CX with no one-qubit
    gate next to their targets."""
    qc = W.brickwork(n, 1, seed)
    for q in range(1, n):
        qc.cx(0, q)
    for q in range(n - 1):
        qc.cx(q, n - 1).h(n - 1).h(n - 1).cx(q, n - 1).x(q).x(q)
    for q in range(n - 1):
        qc.cx(q, q + 1)
    return qc.ry(math.pi, 0).rx(math.pi, n - 1)


CIRCUITS = [(n, kind, seed) for n in (12, 13, 16) for kind, seed in
            (("edge", 1), ("edge", 2), ("edge", 3), ("cz", 4), ("ladder", 5))]


def make(n, kind, seed):
    if kind == "edge":
        return edge_circuit(n, 150, 10 * n + seed)
    return cz_layers(n, 6, seed) if kind == "cz" else ladder(n, seed)


@pytest.fixture(scope="module")
def port():
    from oracle.oracle import Port
    return Port()


@pytest.mark.parametrize("n,kind,seed", CIRCUITS)
def test_rotation_form_records(port, n, kind, seed):
    """The lowered records, executed on the host, against the oracle; no races."""
    qc = make(n, kind, seed)
    state = np.zeros(1 << n, dtype=np.complex128)
    state[0] = 1.0
    got, _p, races, report = emulate(qc, PLANNED, state, grid=4)
    assert races == 0, report
    assert np.max(np.abs(got - port.run_statevector(qc, fuse=False))) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("n,kind,seed", CIRCUITS)
def test_rotation_form_kernel(port, n, kind, seed):
    """The same circuits through the kernel, from a random state, against gate by gate."""
    qc = make(n, kind, seed)
    psi = W.gaussian_state(n, seed)
    got = lq.Statevector.from_numpy(psi).apply(qc).to_numpy()
    want = lq.Statevector.from_numpy(psi).apply(qc, fuse_gates=False).to_numpy()
    assert np.max(np.abs(got - want)) < TOL
