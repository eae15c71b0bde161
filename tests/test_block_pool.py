"""The pool of device blocks: its bookkeeping on the host with a fake device (block_pool_check.cpp:
blocks whose work may be pending, refused frees, the bound on idle memory), and on the GPU that
freeing buffers in one thread and capturing graphs in another leave each other alone."""
import subprocess
import threading
from pathlib import Path

import numpy as np
import pytest

import litequantumcomputingsimulator_b200 as lq
from litequantumcomputingsimulator_b200 import algorithms as A
from litequantumcomputingsimulator_b200 import workloads as W

ROOT = Path(__file__).resolve().parent.parent


def test_bookkeeping(tmp_path):
    exe = tmp_path / "check"
    subprocess.run(["g++", "-std=c++20", "-O1", "-Wall", "-Werror", "-I",
                    str(ROOT / "litequantumcomputingsimulator_b200" / "csrc"),
                    str(ROOT / "tests" / "block_pool_check.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
    assert res.stdout == "ok\n"


def test_release_waits_for_one_stream():
    """CUDA refuses a device-wide wait while any stream is being captured, and it breaks the capture:
    no part of the engine issues one."""
    for src in (ROOT / "litequantumcomputingsimulator_b200" / "csrc").glob("*.c*"):
        assert "cudaDeviceSynchronize(" not in src.read_text(), src.name


@pytest.mark.gpu
def test_frees_beside_captures():
    """One thread builds, captures and replays adjoint plans, the other makes and frees states and
    programs: results as without the other."""
    def gradient(k):
        pc, _ = W.random_pauli_ansatz(9, 30, 50 + k % 3)
        ham = W.random_hamiltonian(9, 10, 60 + k % 3)
        return A.adjoint_gradient(ham, pc, W.random_parameter_sets(30, 2 + k % 5, 70 + k))

    circuits = [W.brickwork(6 + k % 7, 3, k) for k in range(20)]
    want_g = [gradient(k) for k in range(15)]
    want_s = [lq.Statevector(c.num_qubits()).apply(c).to_numpy() for c in circuits]
    A.release_caches()
    errors = []

    def guarded(f):
        def body():
            try:
                f()
            except Exception as e:   # noqa: BLE001 - reported by the assertion below
                errors.append(e)
        return body

    def gradients():
        for _ in range(4):
            for k, (e, g) in enumerate(want_g):
                for _ in range(3):
                    ge, gg = gradient(k)
                    assert np.array_equal(ge, e) and np.array_equal(gg, g)
            A.release_caches()

    def states():
        for r in range(10):
            for c, w in zip(circuits, want_s):
                sv = lq.Statevector(c.num_qubits())
                assert np.array_equal(sv.apply(c).to_numpy(), w)

    threads = [threading.Thread(target=guarded(f)) for f in (gradients, states, states)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


@pytest.mark.gpu
def test_idle_blocks_make_room_for_a_state():
    """A state that fits only where the idle blocks lie is not refused."""
    import torch
    A.release_caches()
    small = [lq.Statevector(21) for _ in range(8)]   # 8 blocks of 32 MiB
    del small                                        # idle now
    free, _total = torch.cuda.mem_get_info()
    need = 16 << 25                                  # 512 MiB
    filler = torch.empty(free - need + (128 << 20), dtype=torch.uint8, device="cuda")
    try:
        sv = lq.Statevector(25)
        assert sv.norm() == 1.0
        del sv
    finally:
        del filler
        torch.cuda.empty_cache()
        A.release_caches()
