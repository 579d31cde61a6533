"""Splitters predicted from samples, one per quantile: a bucket that has grown to
many times its target publishes all of them, so the layouts (seen here as the
fullest bucket of every sub-step) do not depend on which samples came first."""
import ctypes

import numpy
import pytest

import wendy_gb300
from wendy_gb300 import autotune

pytestmark = pytest.mark.gpu


def _fullest(x, v, m, dt, steps):
    sim = wendy_gb300.Simulation(x, v, m, float(numpy.sum(m)), -1.)
    t, out = ctypes.c_double(0.), []
    for _ in range(steps):
        sim.step(dt, 1, t)
        out.append(sim.stats()["last_max_count"])
    assert sim.stats()["substeps_predicted"] > 0
    sim.close()
    return out


def test_buckets_of_many_targets_publish_all_their_samples():
    # sheets at rest, and two groups that each meet in a point: the first makes a
    # bucket overflow, which switches prediction on, the second crowds buckets to
    # up to thirty targets while it is
    saved = autotune.load_table() or [dict(n_min=0, **autotune.current(0))]
    n, dt = 60000, 1e-3
    rng = numpy.random.default_rng(n)
    x, v = rng.uniform(-1., 1., n), numpy.zeros(n)
    g = (x > 0.) & (rng.random(n) < 0.5)
    v[g] = (0.5 - x[g]) / (4 * dt)
    g = (x < 0.) & (rng.random(n) < 0.4)
    v[g] = (-0.5 + 0.01 * rng.normal(size=g.sum()) - x[g]) / (12 * dt)
    try:
        autotune.apply([dict(n_min=0, target=64, window=64, sort_bits=11, ctas_per_sm=2)])
        runs = [_fullest(x, v, numpy.full(n, 1e-9), dt, 20) for _ in range(6)]
    finally:
        autotune.apply(saved)
    assert all(r == runs[0] for r in runs), runs
