"""Device buffers and state batches shared between calls: concurrent threads get the results of
one thread, plans of one shape may alternate, and the caches can be emptied at any time.

Results are compared bit for bit: every reduction on these paths has a fixed order."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import litequantumcomputingsimulator_b200 as lq
from litequantumcomputingsimulator_b200 import algorithms as A
from litequantumcomputingsimulator_b200 import workloads as W

pytestmark = pytest.mark.gpu


def gradient(n, gates, sets, seed):
    pc, _ = W.random_pauli_ansatz(n, gates, seed)
    ham = W.random_hamiltonian(n, 20, seed + 1)
    return A.adjoint_gradient(ham, pc, W.random_parameter_sets(gates, sets, seed + 2))


def jobs():
    out = []
    for s in range(3):
        out.append(lambda s=s: lq.StatevectorSimulator(seed=s).run_registers(
            W.brickwork(14 + s, 4, s, measure=True), 200))
        out.append(lambda s=s: np.concatenate([x.ravel() for x in gradient(9, 12, 3, 40 + s)]))
        # 2 * 48 * 2^15 * 16 B = 48 MiB of states: these plans share one pair of batches
        out.append(lambda s=s: np.concatenate([x.ravel() for x in gradient(15, 5, 48, 70 + s)]))
    return out


@pytest.mark.parametrize("threads", [1, 4])
def test_results_do_not_depend_on_what_shares_the_pool(threads):
    want = [j() for j in jobs()]
    A.release_caches()
    with ThreadPoolExecutor(threads) as ex:
        for _ in range(2):   # the second round replays captured graphs
            got = list(ex.map(lambda j: j(), jobs()))
            for g, w in zip(got, want):
                assert np.array_equal(g, w)
    A.release_caches()
    assert np.array_equal(jobs()[0](), want[0])
