"""Pauli expectations at the edges of their kernels: a block per term (to 14 qubits, down to one),
and passes over coset tiles above (15: eight tiles; 21: more tiles than blocks), with equal,
dependent, Z-only, full-width and identity strings, one term and more than a pass holds.

Against the oracle's sum in 64 bits; tolerance 1e-12 for a normalised state (sums of 2^n terms of
at most 1 in all, rounded in trees: well below 2^n/2 * 1e-16 * the largest term)."""
import numpy as np
import pytest

import litequantumcomputingsimulator_b200 as lq
from litequantumcomputingsimulator_b200 import algorithms as A
from litequantumcomputingsimulator_b200 import workloads as W

pytestmark = pytest.mark.gpu


def strings(n, count, seed):
    rng = np.random.default_rng(seed)
    out = ["I" * n, "Z" * n, "X" * n, "Y" * n, "I" * (n - 1) + "Y"]
    while len(out) < count:
        p = list("".join("IXYZ"[int(v)] for v in rng.integers(0, 4, n)))
        out.append("".join(p))
        flipped = "".join({"I": "Z", "Z": "I", "X": "Y", "Y": "X"}[c] for c in p)
        out.append(flipped)   # the same X mask
    return out[:count]


def plain(psi, pauli):
    n = len(pauli)
    i = np.arange(psi.size)
    x = sum(1 << (n - 1 - k) for k, c in enumerate(pauli) if c in "XY")
    z = sum(1 << (n - 1 - k) for k, c in enumerate(pauli) if c in "YZ")
    sign = 1 - 2 * (np.bitwise_count(i & z).astype(np.int64) & 1)
    return float((1j ** pauli.count("Y") * np.sum(sign * psi * np.conj(psi[i ^ x]))).real)


@pytest.mark.parametrize("n,count", [(1, 3), (4, 9), (8, 30), (14, 12), (15, 1), (15, 60), (16, 45), (21, 25)])
def test_expectation_terms(n, count):
    psi = W.gaussian_state(n, n)
    sv = lq.Statevector.from_numpy(psi)
    paulis = strings(n, count, n) if n > 1 else ["X", "Y", "Z"]
    got = A.expectation_terms(sv, paulis)
    want = [plain(psi, p) for p in paulis]
    assert np.max(np.abs(got - np.array(want))) < 1e-12
    assert np.array_equal(A.expectation_terms(sv, paulis), got)   # fixed order


@pytest.mark.parametrize("n,letters", [(15, "IZ"), (16, "IXYZ"), (20, "IZ")])
def test_many_terms_in_bounded_memory(n, letters):
    """More terms than are planned and summed at a time (1024), in every order of X masks; the scratch
    does not grow with the number of terms times blocks (20000 * 512 * 8 bytes = 78 MiB)."""
    import torch
    rng = np.random.default_rng(n)
    count = 20000 if letters == "IZ" else 2600
    paulis = ["".join(letters[int(v)] for v in rng.integers(0, len(letters), n)) for _ in range(count)]
    sv = lq.Statevector.from_numpy(W.gaussian_state(n, n))
    A.release_caches()
    A.expectation_terms(sv, paulis[:1])
    free, _total = torch.cuda.mem_get_info()
    got = A.expectation_terms(sv, paulis)
    assert free - torch.cuda.mem_get_info()[0] <= 32 << 20
    some = list(range(0, count, 97)) + [1023, 1024, count - 1]
    # the same terms with others about them: another pass, the same sum up to rounding
    want = np.concatenate([A.expectation_terms(sv, [paulis[k] for k in some[i:i + 50]])
                           for i in range(0, len(some), 50)])
    assert np.max(np.abs(got[some] - want)) < 1e-12


@pytest.mark.parametrize("n", [11, 12, 13, 15])
def test_hamiltonian_apply_over_tiles(n):
    """lambda = H psi on tiles of 2^12 amplitudes: one tile (to 12 qubits), and 2 and 8 tiles whose terms
    have X masks above the tile (several groups).  <psi|H|psi> of the adjoint against the sum of the
    terms' expectations; tolerance 1e-12 of the coefficients' sum."""
    rng = np.random.default_rng(n)
    ham = [(float(rng.normal()), "".join("IXYZ"[int(v)] for v in rng.integers(0, 4, n))) for _ in range(60)]
    pc, _ = W.random_pauli_ansatz(n, 20, n)
    params = W.random_parameter_sets(20, 3, n + 1)
    got = A.batched_energy(ham, pc, params)
    for e, p in zip(got, params):
        sv = lq.Statevector(n).apply(pc.bind(p))
        want = sum(c * v for (c, _s), v in zip(ham, A.expectation_terms(sv, [s for _c, s in ham])))
        assert abs(e - want) < 1e-12 * sum(abs(c) for c, _s in ham)
