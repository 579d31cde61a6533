"""The launches a simulation's statistics count: a sort is one kernel for its digits,
one a leading byte and three to place and settle the sheets."""
import ctypes

import pytest

import wendy_gb300
from wendy_gb300 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bytes_", [(1 << 17, 4), ((1 << 17) + 1, 5), ((1 << 22) + 1, 6)])
def test_launches_of_a_first_output_and_of_its_energy(n, bytes_):
    sim = wendy_gb300.Simulation(*ics.gaussian(n, seed=1), 1., -1.)
    sim.step(1e-5, 3, ctypes.c_double(0.))
    first = sim.stats()["launches"]
    # drift, sort, layout; three sub-steps; outputs
    assert first == 2 + (4 + bytes_) + 3 + 1
    sim.energy()
    # a copy of the layout (two), drift, sort, force, two for the sums
    assert sim.stats()["launches"] == first + 2 + 2 + (4 + bytes_) + 2
    sim.close()
