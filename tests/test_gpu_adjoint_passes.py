"""Register passes of the batched adjoint: tiles that are cosets of the rotations' X masks, and
Clifford gates moved to the end of the circuit.

Energies and gradients against one launch per step (LQCS_ADJ_TILES=0, fixed gates applied where
they stand), at the edges of the kernels: 8 qubits (shared-memory tiles), 9..12 (one tile of each
size forward and backward), 13 and above (several tiles); one set and several; strings with no X,
with X on every qubit, equal and dependent X masks; every Clifford gate and fixed rotation the
frame knows, and one it does not (T-controlled, CCX), which keeps the gates in place.

Tolerance: 1e-12 relative to the coefficients' sum (energies) and to twice it (gradients): the
two orders of rounding differ by a few 1e-16 per rotation.
"""
import numpy as np
import pytest

import litequantumcomputingsimulator_b200 as lq
from litequantumcomputingsimulator_b200 import algorithms as A
from litequantumcomputingsimulator_b200 import workloads as W

pytestmark = pytest.mark.gpu


def ansatz(n, gates, seed, ccx=False):
    rng = np.random.default_rng(seed)
    pc = lq.ParametricCircuit(n)
    last = None
    for k in range(gates):
        q = [int(v) for v in rng.permutation(n)]
        c = int(rng.integers(8))
        if c == 0:
            (pc.rx, pc.ry, pc.rz)[int(rng.integers(3))](q[0])
        elif c == 1:
            pc.rp("Z" * 3, q[:3])
        elif c == 2:
            pc.rp("X" * n, list(range(n)))
        elif c == 3 and last:
            pc.rp(*last)   # the same string again
        else:
            w = int(rng.integers(1, min(8, n) + 1))
            last = ("".join("XYZ"[int(v)] for v in rng.integers(0, 3, w)), q[:w])
            pc.rp(*last)
        if k % 2:
            name = ["x", "y", "z", "h", "s", "sdg", "sx", "t", "cx", "cy", "cz", "swap"][int(rng.integers(12))]
            getattr(pc, name)(*q[:2 if name in ("cx", "cy", "cz", "swap") else 1])
        if ccx and k == gates // 2:
            pc.ccx(*q[:3])
    return pc


@pytest.mark.parametrize("n,sets,ccx", [(8, 3, False), (9, 1, False), (10, 5, False), (11, 4, True),
                                        (12, 3, False), (13, 2, True), (15, 6, False), (16, 1, False)])
def test_passes_equal_one_launch_per_step(monkeypatch, n, sets, ccx):
    pc = ansatz(n, 60, 100 + n, ccx)
    ham = W.random_hamiltonian(n, 40, seed=n)
    scale = sum(abs(c) for c, _ in ham)
    params = W.random_parameter_sets(pc.num_parameters(), sets, seed=n + 1)
    energies, grads = A.adjoint_gradient(ham, pc, params)
    only = A.batched_energy(ham, pc, params)
    again = A.adjoint_gradient(ham, pc, params)   # replayed graph
    A.release_caches()
    monkeypatch.setenv("LQCS_ADJ_TILES", "0")
    want_e, want_g = A.adjoint_gradient(ham, pc, params)
    A.release_caches()
    assert np.max(np.abs(energies - want_e)) < 1e-12 * scale
    assert np.max(np.abs(grads - want_g)) < 2e-12 * scale
    assert np.array_equal(only, energies)
    assert np.array_equal(again[0], energies) and np.array_equal(again[1], grads)


@pytest.mark.parametrize("n", [20, 21])   # the backward tiles' size changes between them
def test_tile_sizes_of_large_registers(monkeypatch, n):
    pc = ansatz(n, 14, 200 + n)
    ham = W.random_hamiltonian(n, 6, seed=n)
    scale = sum(abs(c) for c, _ in ham)
    params = W.random_parameter_sets(pc.num_parameters(), 2, seed=n + 1)
    energies, grads = A.adjoint_gradient(ham, pc, params)
    A.release_caches()
    monkeypatch.setenv("LQCS_ADJ_TILES", "0")
    want_e, want_g = A.adjoint_gradient(ham, pc, params)
    A.release_caches()
    assert np.max(np.abs(energies - want_e)) < 1e-12 * scale
    assert np.max(np.abs(grads - want_g)) < 2e-12 * scale


def test_gradient_against_central_differences():
    pc = ansatz(10, 30, 5)
    ham = W.random_hamiltonian(10, 20, seed=6)
    params = W.random_parameter_sets(pc.num_parameters(), 1, seed=7)[0]
    _e, grad = A.adjoint_gradient(ham, pc, params)
    h = 1e-4
    for k in range(0, params.size, 5):
        up, down = params.copy(), params.copy()
        up[k] += h
        down[k] -= h
        e = A.batched_energy(ham, pc, np.stack([up, down]))
        assert abs((e[0] - e[1]) / (2 * h) - grad[k]) < 1e-6
