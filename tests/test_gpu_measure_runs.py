"""Runs of measurements in one launch (k_measure_chain): seeded counts and
collapsed states equal to the oracle's where runs can go wrong: states below
and above the shared-memory limit, a qubit measured twice, two writes to one
classical bit, conditional measurements and resets between, runs of more than
64, and a state kept after the run."""

import numpy as np
import pytest

from helpers import Circuit, conditional, inst
from oracle import oracle as o

import dqsim
from dqsim import workloads

pytestmark = pytest.mark.gpu


def measure(q, c):
    return inst("measure", qubit=q, cbit=c)


def dynamic(n):
    ins = workloads.benchmark_layers(n, 2)
    ins += [measure(0, 0), measure(n - 1, 1), measure(0, 2)]  # a qubit twice in one run
    ins += [inst("reset", qubit=n - 1), conditional(measure(n // 2, 3), 1), conditional(inst("reset", qubit=0), 1)]
    ins += workloads.benchmark_layers(n, 1)
    ins += [measure(q, q % 7) for q in range(n)]  # later writes to a bit win
    return Circuit(n, ins, 7)


@pytest.mark.parametrize("precision", ["complex128", "complex64"])
@pytest.mark.parametrize("n", [2, 5, 11, 12, 13, 15])
def test_runs_of_measurements_match_the_oracle(n, precision):
    c = dynamic(n)
    got = dqsim.StatevectorSimulator(seed=5, precision=precision).simulate_shots(c, shots=80)
    want = o.OracleSimulator(seed=5).simulate_shots(c, shots=80)
    assert got == want


@pytest.mark.parametrize("n", [3, 12, 14])
def test_state_after_a_run(n):
    ins = workloads.benchmark_layers(n, 2) + [measure(q, q) for q in range(n // 2, n)] + [measure(n - 1, 0)]
    c = Circuit(n, ins + workloads.benchmark_layers(n, 1), n)
    got, want = dqsim.StatevectorSimulator(seed=9).simulate(c), o.OracleSimulator(seed=9).simulate(c)
    assert got.classical_bits == want.classical_bits
    assert np.max(np.abs(got.statevector - want.statevector)) <= 1e-12


def test_runs_of_more_than_64_measurements():
    n = 6
    ins = workloads.benchmark_layers(n, 2) + [inst("reset", qubit=0)] + workloads.benchmark_layers(n, 1)
    c = Circuit(n, ins + [measure(i % n, i) for i in range(70)], 70)
    assert (dqsim.StatevectorSimulator(seed=2).simulate_shots(c, shots=50)
            == o.OracleSimulator(seed=2).simulate_shots(c, shots=50))
