"""Circuits that leave a register pass without records: X gates (bits stored negated), SWAPs of
qubits on registers (bits stored elsewhere), identities; alone, several, and as the last pass of a
longer circuit.  Every amplitude of a random state equals the permuted one exactly."""
import numpy as np
import pytest

import litequantumcomputingsimulator_b200 as lq
from litequantumcomputingsimulator_b200 import workloads as W
from litequantumcomputingsimulator_b200.simulator import CompiledCircuit

pytestmark = pytest.mark.gpu


def circuits(n):
    yield "x low", lq.QuantumCircuit(n).x(0)
    yield "x high", lq.QuantumCircuit(n).x(n - 1)
    yield "x several", lq.QuantumCircuit(n).x(2).x(7).x(n - 2)
    allx = lq.QuantumCircuit(n)
    for q in range(n):
        allx.x(q)
    yield "x all", allx
    yield "x twice", lq.QuantumCircuit(n).x(3).x(3)
    yield "swap registers", lq.QuantumCircuit(n).swap(n - 1, n - 2)
    yield "swap lanes", lq.QuantumCircuit(n).swap(0, n - 1)
    yield "swap and x", lq.QuantumCircuit(n).swap(n - 1, n - 3).x(n - 1)
    yield "identity", lq.QuantumCircuit(n).i(4)
    yield "barrier", lq.QuantumCircuit(n).barrier() if hasattr(lq.QuantumCircuit, "barrier") else lq.QuantumCircuit(n)
    yield "nothing", lq.QuantumCircuit(n)


def permuted(psi, qc):
    i = np.arange(psi.size)
    for inst in qc.instructions():
        name, q = inst.gate.type.name, list(inst.qubits)
        if name == "X":
            i = i ^ (1 << q[0])
        elif name == "SWAP":
            d = ((i >> q[0]) ^ (i >> q[1])) & 1
            i = i ^ (d << q[0]) ^ (d << q[1])
    out = np.empty_like(psi)
    out[i] = psi
    return out


@pytest.mark.parametrize("n", [9, 12, 13, 16, 20])
def test_passes_without_records(n):
    psi = W.gaussian_state(n, n)
    for name, qc in circuits(n):
        want = permuted(psi, qc)
        got = lq.Statevector.from_numpy(psi).apply(qc).to_numpy()
        assert np.array_equal(got, want), name
        sv = lq.Statevector.from_numpy(psi)
        prog = CompiledCircuit(qc, fusion_mode=4)   # the tile planner, also below 12 qubits
        prog.apply(sv)
        assert np.array_equal(sv.to_numpy(), want), name
        prog.profile(sv)


def test_basis_states_run():
    """The bits a circuit of X gates sets, sampled, and under noise that changes none of them."""
    for n in (12, 14):
        qc = lq.QuantumCircuit(n, n).x(1).x(n - 1).measure_all()
        want = (1 << 1) | (1 << (n - 1))
        assert np.all(lq.StatevectorSimulator(seed=1).run_registers(qc, 50) == want)
        noise = lq.NoiseModel().add_all_qubit_channel(lq.KrausChannel.phase_flip(0.3))
        assert np.all(lq.StatevectorSimulator(seed=1, noise=noise).run_registers(qc, 50) == want)


@pytest.mark.parametrize("n", [12, 14])
def test_gate_counts(n):
    """Every source gate is counted, also where products of gates turn out to be the identity."""
    for qc, gates in ((lq.QuantumCircuit(n).x(3).x(3), 2), (lq.QuantumCircuit(n).h(0).h(0).x(1), 3),
                      (lq.QuantumCircuit(n).cx(0, 1).cx(0, 1).i(2), 3), (lq.QuantumCircuit(n), 0)):
        assert CompiledCircuit(qc).n_gates == gates
