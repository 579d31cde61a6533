"""Several exact simulations alive at once: their steps do not depend on which was
set up last (the golden trajectories themselves are in test_gpu_exact.py)."""
import numpy
import pytest

import wendy_gb300
from wendy_gb300 import ics

pytestmark = pytest.mark.gpu


def _outputs(gen, k):
    return [tuple(a.copy() for a in next(gen)[:2]) for _ in range(k)]


@pytest.mark.parametrize("omega", [None, 1.1])
def test_steps_of_simulations_of_different_sizes_interleave(omega):
    # 2001 sheets take more shared memory than a block has without asking, 51 less
    runs = {n: ics.sech2_disk(n, seed=n) for n in (2001, 51, 901)}
    dt = 0.002

    def start(n):
        return wendy_gb300.nbody(*runs[n], dt, omega=omega)

    want = {n: _outputs(start(n), 3) for n in runs}
    gens = {n: start(n) for n in runs}
    got = {n: [] for n in runs}
    for _ in range(3):
        for n in runs:
            got[n] += _outputs(gens[n], 1)
    for n in runs:
        for (gx, gv), (wx, wv) in zip(got[n], want[n]):
            assert numpy.array_equal(gx, wx) and numpy.array_equal(gv, wv)
