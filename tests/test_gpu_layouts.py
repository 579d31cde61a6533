"""Ensembles whose step has few buckets, so that members are laid out in buckets
smaller than the tuned ones: every member gives the bits it gives alone (prefix
masses are exact sums, every sheet's arithmetic is the same), and no sheet is
lost whatever the sizes beside it."""
import ctypes

import numpy
import pytest

import wendy_gb300
from wendy_gb300 import ics
from wendy_gb300.ensemble import Pool

pytestmark = pytest.mark.gpu


def _sizes(which):
    if which == "mixed":
        return [int(round(s)) for s in numpy.geomspace(500, 20000, 90)]
    return {"400 x 1200": [1200] * 400, "410 x 1280": [1280] * 410, "210 x 1500": [1500] * 210,
            "220 x 3000": [3000] * 220, "one large": [500000, 1200, 1100, 5791],
            "330 x 1024": [1024] * 330}[which]


@pytest.mark.parametrize("which", ["400 x 1200", "410 x 1280", "210 x 1500", "220 x 3000",
                                   "330 x 1024", "one large", "mixed"])
def test_members_of_small_buckets_match_single_runs(which):
    sizes = _sizes(which)
    mem = [ics.sech2_disk(n, seed=k, masses="lognormal" if k % 2 else "equal")
           for k, n in enumerate(sizes)]
    with Pool() as pool:
        ids = [pool.add(x, v, m, omega=0.5) for x, v, m in mem]
        t = numpy.zeros(len(ids))
        for _ in range(2):
            pool.step(ids, numpy.full(len(ids), 0.005), 6, t)
        got = [pool.download(i) for i in ids]
    for (x, v, m), (gx, gv) in zip(mem, got):
        sim = wendy_gb300.Simulation(x, v, m, float(numpy.sum(m)), 0.25)
        ts = ctypes.c_double(0.)
        for _ in range(2):
            sim.step(0.005, 6, ts)
        ax, av = numpy.empty(len(x)), numpy.empty(len(x))
        sim.download(ax, av)
        sim.close()
        assert numpy.array_equal(gx, ax) and numpy.array_equal(gv, av)
