"""Marginal probabilities (k_marginal) where its split can go wrong: registers
smaller and larger than a chunk, selections below, above and across it, every
qubit in another order, none; both precisions.  Reference: numpy over the
returned statevector; sums of at most 2^17 terms in [0, 1] in FP64 differ by
less than 1e-13."""

import numpy as np
import pytest

from helpers import hea

import dqsim

pytestmark = pytest.mark.gpu


def selections(n):
    rng = np.random.default_rng(n)
    yield []
    yield [n - 1]
    yield [0]
    yield list(range(n))  # ascending: not the sampler's order
    if n > 2:
        yield [0, n - 1]
        yield list(range(n - 1, 0, -1))
        for k in {2, n // 2, n - 1, min(n, 13)}:
            yield [int(q) for q in rng.choice(n, size=k, replace=False)]
    if n > 13:
        yield list(range(12))
        yield list(range(n - 1, 11, -1))


def reference(psi, n, qubits):
    p = (np.abs(psi) ** 2).reshape((2,) * n)
    kept = sorted(qubits, reverse=True)
    p = p.sum(axis=tuple(n - 1 - q for q in range(n) if q not in qubits))
    return p.transpose([kept.index(q) for q in qubits]).ravel() if qubits else p.reshape(1)


@pytest.mark.parametrize("precision", ["complex128", "complex64"])
@pytest.mark.parametrize("n", [1, 2, 5, 8, 11, 12, 13, 17])
def test_marginals(n, precision):
    r = dqsim.StatevectorSimulator(seed=1, precision=precision).simulate(hea(n, 3, seed=n))
    psi = r.statevector
    for qubits in selections(n):
        got = np.zeros(1 << len(qubits))
        table = r.probabilities(qubits)
        got[list(table)] = list(table.values())
        np.testing.assert_allclose(got, reference(psi, n, qubits), atol=1e-13, rtol=0, err_msg=str(qubits))


@pytest.mark.parametrize("n,k", [(3, 3), (10, 0), (11, 1), (12, 1), (12, 2), (13, 3), (14, 3), (18, 8), (20, 10), (20, 9), (21, 11)])
def test_marginals_where_gathering_meets_chunks(n, k):
    """Up to 20 qubits and ten unselected ones, and just beyond either."""
    r = dqsim.StatevectorSimulator(seed=1).simulate(hea(n, 2, seed=n))
    psi = r.statevector
    qubits = [int(q) for q in np.random.default_rng(100 * n + k).choice(n, size=k, replace=False)]
    got = np.zeros(1 << k)
    table = r.probabilities(qubits)
    got[list(table)] = list(table.values())
    np.testing.assert_allclose(got, reference(psi, n, qubits), atol=1e-13, rtol=0)
