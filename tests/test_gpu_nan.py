"""Positions that are not numbers: an external force may have no value somewhere.
Such a sheet is ordered by its key like any other (first or last, by the sign of
its NaN), on all paths, so the other sheets do not depend on which path ran."""
import ctypes

import numpy
import pytest

import wendy_gb300
from wendy_gb300 import ics
from wendy_gb300.ensemble import Pool
from wendy_gb300.extforce import Expression

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [20, 700, 1500])
@pytest.mark.parametrize("dt", [0.4, 0.01])
@pytest.mark.parametrize("expr", ["0.1*sqrt(40.0-x)", "-(0.1*sqrt(40.0-x))"])
def test_sheets_beside_one_without_a_position(n, dt, expr):
    # the rightmost sheet gets no force; with the longer step every sheet passes
    # many others in a sub-step
    x, v, m = ics.gaussian(n, seed=n, masses="lognormal")
    k = int(numpy.argmax(x))
    x[k], v[k] = 50., 0.
    ext = Expression(expr)
    tot = float(numpy.sum(m))
    sim = wendy_gb300.Simulation(x, v, m, tot, -1., ext)
    t = ctypes.c_double(0.)
    with Pool() as pool:
        i = pool.add(x, v, m, ext_force=ext)
        tp = numpy.zeros(1)
        for _ in range(3):
            sim.step(dt, 5, t)
            pool.step([i], numpy.array([dt]), 5, tp)
            sx, sv = numpy.empty(n), numpy.empty(n)
            sim.download(sx, sv)
            px, pv = pool.download(i)
            assert numpy.isnan(sx[k]) and numpy.isfinite(numpy.delete(sx, k)).all()
            assert numpy.array_equal(sx, px, equal_nan=True)
            assert numpy.array_equal(sv, pv, equal_nan=True)
    sim.close()
