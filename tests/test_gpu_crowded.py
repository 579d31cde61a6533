"""Sorts of positions that share the leading bytes of their keys by the thousand:
systems far from the origin against their width, and systems crowded about a few
places.  Orders are exact; calls on them take no more than a few times as long as on
a system about the origin."""
import ctypes
import time

import numpy
import pytest

import wendy_gb300
from wendy_gb300 import ics
from wendy_gb300.ensemble import Pool

pytestmark = pytest.mark.gpu


def _crowded(n, kind):
    rng = numpy.random.default_rng(n)
    g = rng.normal(0., 1., n)
    if kind == "cores":  # two cores, and a third of the sheets around them
        x = numpy.where(rng.random(n) < 0.5, 1. + 1e-5 * g, -1. + 1e-6 * g)
        x[::3] = rng.normal(0., 3., len(x[::3]))
        return x
    if kind == "equal":  # a few places, each with a core around it
        x = rng.integers(0, 7, n) * 0.5
        x[::2] += 2. ** -51 * rng.integers(-9, 9, len(x[::2]))
        return x
    return g + float(kind)


# sizes at the tiles of 2048 sheets and about the smallest crowd that is sorted whole
# (2048 sheets and a 256th of all), and one beyond each choice of leading bytes
@pytest.mark.parametrize("n", [2049, 2057, 2058, 4096, 4097, 6144, 20011, 100003, (1 << 18) + 5,
                               1000003, (1 << 22) + 9])
@pytest.mark.parametrize("kind", ["1e4", "1e6", "-1e9", "1e13", "cores", "equal"])
def test_orders_of_crowded_positions(n, kind):
    x = _crowded(n, kind)
    m = numpy.random.default_rng(1).lognormal(0., 0.5, n)
    tot = float(numpy.sum(m))
    got, perm = wendy_gb300.accel(x, m, tot)
    order = numpy.argsort(x, kind="stable")
    assert numpy.array_equal(perm, order)
    ms = m[order].astype(numpy.longdouble)
    ref = numpy.empty(n)
    ref[order] = (tot - 2. * numpy.cumsum(ms) + ms).astype(numpy.float64)
    assert numpy.max(numpy.abs(got - ref)) <= 1e-12 * tot


@pytest.mark.parametrize("shift", [0., 2. ** 20, 2. ** 33])
def test_equal_positions_come_by_index_whatever_their_order(shift):
    # a slab falling through its centre overflows its buckets; the re-sorts start
    # from the buckets' order, not that of the indices, and far from the origin many
    # positions are equal.  A single simulation and a pool sort by different passes
    n = 1 << 17
    rng = numpy.random.default_rng(9)
    x = rng.uniform(-1., 1., n)
    v = -60. * x + 0.3 * rng.normal(size=n)
    m = rng.lognormal(0., 0.5, n) / n
    tot = float(numpy.sum(m))
    sim = wendy_gb300.Simulation(x + shift, v, m, tot, -1.)
    t = ctypes.c_double(0.)
    with Pool() as pool:
        i = pool.add(x + shift, v, m)
        for _ in range(3):
            sim.step(0.002, 8, t)
            pool.step([i], numpy.array([0.002]), 8, numpy.zeros(1))
            sim.energy()  # (sorts a copy of the sheets)
            sx, sv = numpy.empty(n), numpy.empty(n)
            sim.download(sx, sv)
            px, pv = pool.download(i)
            assert numpy.array_equal(sx, px) and numpy.array_equal(sv, pv)
    assert sim.stats()["sorts_full"] > 1
    sim.close()


@pytest.mark.parametrize("n,shift", [(100003, 1e9), (1000003, 1e9), (4000037, 1e4)])
def test_systems_far_from_the_origin_take_about_as_long(n, shift):
    x, _, m = ics.gaussian(n, seed=n)

    def best(y):
        out = []
        for _ in range(5):
            t0 = time.perf_counter()
            wendy_gb300.accel(y, m, 1.)
            out.append(time.perf_counter() - t0)
        return min(out)

    assert best(x + shift) <= 2.5 * best(x)
