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
