"""Register passes stay in rotation form where their matrices outgrow the shared-memory stage (2048
entries: passes that hold a whole 12-qubit circuit): such a pass takes compact diagonal tables.

The lowered records, executed on the host, against the oracle (1e-12 per amplitude, the engine's
bound); on the GPU the same circuits, and noisy trajectories whose passes hold per-state matrices,
against the paths without passes."""
import numpy as np
import pytest

import litequantumcomputingsimulator_b200 as lq
from litequantumcomputingsimulator_b200 import algorithms as A
from litequantumcomputingsimulator_b200 import workloads as W
from test_reg_emulation import PLANNED, emulate
from test_rotation_form import cz_layers, edge_circuit

TOL = 1e-12


def mix(n, seed):
    rng = np.random.default_rng(seed)
    qc = lq.QuantumCircuit(n)
    for _ in range(10 * n):
        a, b, c = (int(v) for v in rng.permutation(n)[:3])
        ang = float(rng.uniform(-3, 3))
        k = int(rng.integers(6))
        if k < 2:
            qc.u(ang, 1.0 - ang, 0.4 * ang, a)
        elif k == 2:
            qc.cx(a, b)
        elif k == 3:
            qc.rzz(ang, a, b)
        elif k == 4:
            qc.rp(ang, "XYZ", [a, b, c])
        else:
            qc.cp(ang, a, b)
    return qc


CIRCUITS = ([("qft", 12, 0)] + [("brickwork", 12, d) for d in (8, 10, 13, 16, 20)] +
            [("brickwork", 10, 20), ("brickwork", 13, 20), ("mix", 12, 1), ("mix", 12, 2),
             ("edge", 12, 3), ("cz", 12, 12)])


def make(kind, n, k):
    return {"qft": lambda: A.qft(n), "brickwork": lambda: W.brickwork(n, k, 7 + k), "mix": lambda: mix(n, k),
            "edge": lambda: edge_circuit(n, 300, k), "cz": lambda: cz_layers(n, k, k)}[kind]()


@pytest.fixture(scope="module")
def port():
    from oracle.oracle import Port
    return Port()


@pytest.mark.parametrize("kind,n,k", CIRCUITS)
def test_no_dense_fallback(port, kind, n, k):
    qc = make(kind, n, k)
    state = np.zeros(1 << n, dtype=np.complex128)
    state[0] = 1.0
    got, passes, races, report = emulate(qc, PLANNED, state, grid=2)
    assert races == 0, report
    assert report == f"{passes} of {passes} passes in rotation form"
    assert np.max(np.abs(got - port.run_statevector(qc, fuse=False))) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("kind,n,k", CIRCUITS)
def test_compact_tables_kernel(kind, n, k):
    qc = make(kind, n, k)
    psi = W.gaussian_state(n, 5)
    got = lq.Statevector.from_numpy(psi).apply(qc).to_numpy()
    want = lq.Statevector.from_numpy(psi).apply(qc, fuse_gates=False).to_numpy()
    assert np.max(np.abs(got - want)) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("n,depth", [(12, 10), (12, 16), (13, 14)])
def test_compact_tables_per_state(monkeypatch, n, depth):
    """Noise as per-state matrices in passes this full: the registers of unfused trajectories."""
    qc = W.brickwork(n, depth, n + depth, measure=True)
    noise = lq.NoiseModel().add_all_qubit_channel(lq.KrausChannel.depolarizing(0.01))
    noise.add_all_qubit_channel(lq.KrausChannel.amplitude_damping(0.001))

    def run():
        return lq.StatevectorSimulator(seed=3, noise=noise).run_registers(qc, 24)

    got = run()
    monkeypatch.setenv("LQCS_TRAJ_FUSED", "0")
    assert np.array_equal(got, run())
