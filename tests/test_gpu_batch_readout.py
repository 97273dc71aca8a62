"""<Z0 Z1> and counts of a batch where its readout can go wrong: circuits
smaller and larger than a summed part (2^13 amplitudes) and a scan tile (2^11),
in an order that puts several in one tile.  <Z0 Z1> within 1e-12 of the
statevector's (1e-6 in single precision), counts equal to a single call's."""

import numpy as np
import pytest

import dqsim
from dqsim import _core, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["complex128", "complex64"])
def test_readout_of_uneven_circuits(precision):
    sizes = [2, 3, 11, 5, 12, 13, 14, 2, 15, 16]
    circuits = [workloads.hea(n, 3, seed=i, measure=True) for i, n in enumerate(sizes)]
    sim = dqsim.StatevectorSimulator(seed=3, precision=precision)
    batch = _core.BatchedCircuits(sim, circuits, shots=200)
    batch.run()
    zz = batch.expect_zz()
    for i, n in enumerate(sizes):
        p = np.abs(batch.statevector(i, n)) ** 2
        j = np.arange(1 << n)
        want = np.sum(np.where((j ^ (j >> 1)) & 1, -p, p))
        assert abs(zz[i] - want) <= (1e-12 if precision == "complex128" else 1e-6)
        if precision == "complex128":
            seed = (3 + i * _core.BATCH_SEED_STRIDE) % (1 << 64)
            assert batch.counts(i) == dqsim.StatevectorSimulator(seed=seed).simulate_shots(circuits[i], shots=200)
