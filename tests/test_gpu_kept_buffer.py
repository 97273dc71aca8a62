"""The statevector buffer a simulator keeps after a result goes: given back before
a call makes one of another size, and with the simulator."""

import pytest

from helpers import Circuit, inst

import dqsim
from dqsim import _core

pytestmark = pytest.mark.gpu
MB = 1 << 20  # the large state holds 512; the pool and the small states 64 at most


def free():
    return _core.device_memory(0)["free"]


def test_a_call_of_another_size_gives_the_kept_buffer_back():
    sim = dqsim.StatevectorSimulator(seed=1)
    small, large = Circuit(10, [inst("h", qubit=0)]), Circuit(25, [inst("h", qubit=0)])
    sim.simulate(small)  # the device's context and the engine's pool are there from now on
    before = free()
    held = sim.simulate(large)
    assert free() <= before - 448 * MB
    del held
    assert free() <= before - 448 * MB  # kept for the next call of its size
    held = sim.simulate(small)
    assert free() >= before - 64 * MB
    del held


def test_the_simulator_gives_the_kept_buffer_back():
    keeper = dqsim.StatevectorSimulator(seed=1)  # keeps the device's pool as it is
    sim = dqsim.StatevectorSimulator(seed=1)
    keeper.simulate(Circuit(10, [inst("h", qubit=0)]))
    before = free()
    sim.simulate(Circuit(25, [inst("h", qubit=0)]))
    assert free() <= before - 448 * MB
    del sim
    assert free() >= before - 64 * MB
