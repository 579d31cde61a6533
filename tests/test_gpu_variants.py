"""The kernel variants and where the library changes from one to another:
simulations run in one launch, bucket layouts of different targets, equal and
unequal masses, launches by kind of external force, sort and force tiles of
different sizes.

Tolerances, fixed beforehand:
  * two variants of the same computation (a simulation alone and as a member
    of an ensemble; equal masses with and without a massless tracer beside
    them, which turns the equal-mass form off) give the same bits: prefix
    masses are exact sums, every sheet's arithmetic is the same;
  * against the oracle 1e-10 absolute after an output, as in the other parity
    tests (unit-scale systems; rounding of the oracle's running sum is below
    1e-13 a sub-step, dt and the number of sub-steps keep its growth below 10);
  * accelerations 1e-12 of the acceleration scale, orders exact;
  * powers by products: half an ulp and a few 2^-53 of it, against a library
    power within one ulp: 2 x 2^-52 relative; quotients: the same bits.
"""
import ctypes
import threading

import numpy
import pytest

import wendy_gb300
from oracle import oracle as O
from wendy_gb300 import _lib, ics
from wendy_gb300.ensemble import Pool
from wendy_gb300.extforce import Expression, Harmonic, PulseTanh, evaluate_on_device

pytestmark = pytest.mark.gpu

PULSE = PulseTanh(0.3, 5.0, 1.0, 0.5)
BREATHING = "-0.5*(1.0+0.3*sin(2.0*t))*x**3/(1.0+x**2)"


def _alone(x, v, m, omega, ext, dt, nleap, t0=4.0, nout=1, totmass=None):
    tot = float(numpy.sum(m)) if totmass is None else totmass
    sim = wendy_gb300.Simulation(x, v, m, tot, -1. if omega is None else omega ** 2, ext)
    t = ctypes.c_double(t0)
    for _ in range(nout):
        sim.step(dt, nleap, t)
    gx, gv = numpy.empty(len(x)), numpy.empty(len(x))
    sim.download(gx, gv)
    sim.close()
    return gx, gv


def _members(members, dt, nleap, t0=4.0, nout=1):
    with Pool() as pool:
        ids = [pool.add(x, v, m, omega=omega, ext_force=ext) for x, v, m, omega, ext in members]
        t = numpy.full(len(ids), t0)
        for _ in range(nout):
            pool.step(ids, numpy.full(len(ids), dt), nleap, t)
        return [pool.download(i) for i in ids]


def _same(a, b):
    return numpy.array_equal(a[0], b[0]) and numpy.array_equal(a[1], b[1])


def _near_oracle(got, x, v, m, omega, ext, dt, nleap, t0=4.0):
    rx, rv = next(O.nbody_approx(x, v, m, dt * nleap, nleap, t0=t0, omega=omega, ext=ext))
    assert numpy.max(numpy.abs(got[0] - rx)) <= 1e-10
    assert numpy.max(numpy.abs(got[1] - rv)) <= 1e-10


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 257, 1023, 1024, 1025, 2047, 2048, 2049])
@pytest.mark.parametrize("masses", ["equal", "lognormal"])
def test_small_simulations(n, masses):
    # up to 2048 sheets one launch runs the whole call; 40 sub-steps are more
    # than the lanes of a warp
    x, v, m = ics.gaussian(n, seed=n, masses=masses)
    for omega, ext in ((None, None), (1.1, PULSE)):
        got = _alone(x, v, m, omega, ext, 0.001, 40)
        assert _same(got, _members([(x, v, m, omega, ext)], 0.001, 40)[0])
        _near_oracle(got, x, v, m, omega, ext, 0.001, 40)


@pytest.mark.parametrize("n", [1535, 1536, 1537])
def test_small_simulations_with_an_expression(n):
    x, v, m = ics.gaussian(n, seed=n)
    e = Expression(BREATHING)
    got = _alone(x, v, m, None, e, 0.002, 40, t0=0.3)
    assert _same(got, _members([(x, v, m, None, e)], 0.002, 40, t0=0.3)[0])
    _near_oracle(got, x, v, m, None, e, 0.002, 40, t0=0.3)


@pytest.mark.parametrize("n", [40, 1000, 2048])
def test_small_simulations_with_long_steps_and_coincident_sheets(n):
    # every sheet passes many others in a sub-step, and some share a position
    x, v, m = ics.gaussian(n, seed=n, masses="lognormal")
    k = n // 10
    x[k:3 * k] = x[:2 * k]
    v[k:2 * k] = v[:k]
    got = _alone(x, v, m, 0.7, None, 0.4, 5, nout=3)
    assert _same(got, _members([(x, v, m, 0.7, None)], 0.4, 5, nout=3)[0])


@pytest.mark.parametrize("n", [2049, 3000, 384 * 456 + 1, 700417])
@pytest.mark.parametrize("family", ["sech2", "tophat"])
def test_bucket_layouts(n, family):
    # from the smallest targets up to those that take more than one round
    x, v, m = ics.FAMILIES[family](n, seed=n, masses="lognormal")
    _near_oracle(_alone(x, v, m, 1.1, PULSE, 0.002, 6), x, v, m, 1.1, PULSE, 0.002, 6)


@pytest.mark.parametrize("n", [5, 1999, 40001, 300001])
def test_equal_masses_give_the_bits_of_the_general_form(n):
    x, v, m = ics.sech2_disk(n, seed=n)
    tot = float(numpy.sum(m))
    got = _alone(x, v, m, None, PULSE, 0.002, 8, nout=2, totmass=tot)
    tracer = (numpy.append(x, 1e3), numpy.append(v, 0.), numpy.append(m, 0.))
    gen = _alone(*tracer, None, PULSE, 0.002, 8, nout=2, totmass=tot)
    assert numpy.array_equal(got[0], gen[0][:n]) and numpy.array_equal(got[1], gen[1][:n])


def test_equal_masses_through_overflowing_buckets():
    # a slab falling through its centre in a few sub-steps: layouts overflow, are
    # compacted and laid out again
    n = 1 << 18
    rng = numpy.random.default_rng(9)
    x = rng.uniform(-1., 1., n)
    v = -60. * x + 0.3 * rng.normal(size=n)
    m = numpy.full(n, 1. / n)
    got = _alone(x, v, m, None, None, 0.002, 8, nout=3, totmass=1.)
    tracer = (numpy.append(x, 1e3), numpy.append(v, 0.), numpy.append(m, 0.))
    gen = _alone(*tracer, None, None, 0.002, 8, nout=3, totmass=1.)
    assert numpy.array_equal(got[0], gen[0][:n]) and numpy.array_equal(got[1], gen[1][:n])
    other = ics.sech2_disk(3000, seed=1, masses="lognormal")
    for mem in ([(x, v, m, None, None)], [(x, v, m, None, None), (*other, None, None)]):
        assert _same(got, _members(mem, 0.002, 8, nout=3)[0])
    sim = wendy_gb300.Simulation(x, v, m, 1., -1.)
    sim.step(0.002, 8, ctypes.c_double(4.))
    st = sim.stats()
    sim.close()
    assert st["sorts_full"] > 1  # it did overflow


@pytest.mark.parametrize("n", [900, 40001])
def test_stateless_calls_whose_masses_change(n):
    # equal masses for two calls, unequal ones in the third, equal in the fourth
    x, v, m0 = ics.sech2_disk(n, seed=n)
    m1 = ics.sech2_disk(n, seed=n + 1, masses="lognormal")[2]
    outs = []
    for which in ("gpu", "oracle"):
        xx, vv, a = x.copy(), v.copy(), numpy.zeros(n)
        xi = O.make_sheets(xx)
        t = 4.5
        for m in (m0, m0, m1, m0):
            tot = float(numpy.sum(m))
            if which == "gpu":
                t, _el = wendy_gb300.approx_onestep(xi, xx, vv, m, a, tot, 0.002, 5, t,
                                                    omega2=-1., ext_force=PULSE)
            else:
                t, _el = O.onestep(xi, xx, vv, m, a, tot, 0.002, 5, t, -1., PULSE)
        outs.append((xi.copy(), xx, vv, a))
    assert numpy.array_equal(outs[0][0]["idx"], outs[1][0]["idx"])
    for p, q in zip(outs[0][1:], outs[1][1:]):
        assert numpy.max(numpy.abs(p - q)) <= 1e-10


@pytest.mark.parametrize("force", ["none", "closed", "expression"])
@pytest.mark.parametrize("masses", ["equal", "unequal", "both"])
def test_ensemble_launch_variants(force, masses):
    exts = {"none": [None, None, None], "closed": [None, PULSE, Harmonic(0.7)],
            "expression": [None, PULSE, Expression(BREATHING)]}[force]
    kinds = {"equal": ["equal"] * 3, "unequal": ["lognormal"] * 3,
             "both": ["lognormal", "equal", "lognormal"]}[masses]
    mem = []
    for k, n in enumerate((2500, 9001, 30000)):
        x, v, m = ics.gaussian(n, seed=k, masses=kinds[k])
        mem.append((x, v, m, 1.1 if k == 2 else None, exts[k]))
    for s, got in zip(mem, _members(mem, 0.003, 6, nout=2)):
        assert _same(got, _alone(*s, 0.003, 6, nout=2))


# one sheet on either side of the force tiles (512 sheets, up to 2^16; 2048
# above), of the sort's tiles (1024 keys up to 2^18 sheets; 4096 above, with 512
# threads up to one tile per SM of 152) and of its leading bytes (four up to 2^17,
# five up to 2^22, six above)
@pytest.mark.parametrize("n", [511, 512, 513, 1024, 1025, 65535, 65536, 65537, 1 << 17,
                               (1 << 17) + 1, 1 << 18, (1 << 18) + 1, 152 * 4096,
                               152 * 4096 + 1, 1 << 22, (1 << 22) + 1])
def test_force_evaluation_at_the_limits_of_its_tiles(n):
    # a third of the positions shares its leading bytes: runs of pairs, of equal
    # positions and of positions a few units in the last place apart
    rng = numpy.random.default_rng(n)
    x = rng.normal(0., 1., n)
    near = rng.permutation(n)[:n // 3]
    a, b, c = numpy.array_split(near, 3)
    x[a] = 1.0 + rng.integers(0, 1 << 22, len(a)) * 2. ** -52
    x[b] = -0.75 - rng.integers(0, 3, len(b)) * 2. ** -53
    x[c] = x[numpy.roll(c, 1)] * (1. + 2. ** -50)
    m = rng.lognormal(0., 0.5, n)
    tot = float(numpy.sum(m))
    got, perm = wendy_gb300.accel(x, m, tot, omega2=1.21)
    order = numpy.argsort(x, kind="stable")
    assert numpy.array_equal(perm, order)
    ms = m[order].astype(numpy.longdouble)
    cum = numpy.cumsum(ms)
    ref = numpy.empty(n)
    ref[order] = (tot - 2. * cum + ms).astype(numpy.float64) - 1.21 * x[order]
    scale = max(tot, float(numpy.max(numpy.abs(ref))))
    assert numpy.max(numpy.abs(got - ref)) <= 1e-12 * scale


@pytest.mark.parametrize("n", [70001, 300001, (1 << 22) + 3])
@pytest.mark.parametrize("step", [0.25, 0.25 + 2. ** -16, 0.25 + 2. ** -29])
def test_sort_of_positions_whose_bytes_are_partly_constant(n, step):
    # digits that are the same for every key are skipped, but not the pass that
    # halves the keys
    rng = numpy.random.default_rng(n)
    x = 4. + step * rng.integers(0, 8, n)
    got, perm = wendy_gb300.accel(x, numpy.full(n, 1. / n), 1.)
    assert numpy.array_equal(perm, numpy.argsort(x, kind="stable"))


@pytest.mark.parametrize("k", ["2", "3", "4", "7", "8", "9", "-3", "2.5", "3.5", "16"])
def test_powers_of_an_expression(k):
    rng = numpy.random.default_rng(5)
    x = numpy.concatenate([rng.normal(0., 3., 1001), 10. ** rng.uniform(-300., 300., 1000),
                           -10. ** rng.uniform(-300., 300., 1000),
                           [0., -0., 1., -1., 5e-324, -5e-324, numpy.inf, -numpy.inf,
                            numpy.nan, 1e-34, 1e-110, 1e38, 1e103]])
    with numpy.errstate(all="ignore"):
        got = evaluate_on_device(Expression("x**(%s)" % k), x, 0.)
        ref = numpy.power(x, float(k))
        fin = numpy.isfinite(ref) & (numpy.abs(ref) >= 2. ** -1021)
        assert numpy.all(numpy.abs(got[fin] - ref[fin]) <= 2. * 2. ** -52 * numpy.abs(ref[fin]))
        # below that, a unit in the last place is 2^-1074
        low = numpy.isfinite(ref) & ~fin
        assert numpy.all(numpy.abs(got[low] - ref[low]) <= 2. * 2. ** -1074)
        assert numpy.array_equal(numpy.signbit(got[fin | low]), numpy.signbit(ref[fin | low]))
        rest = ~(fin | low)
        assert numpy.array_equal(got[rest], ref[rest], equal_nan=True)


@pytest.mark.parametrize("t", [1., -3., 0.1, 1e-150, 2. ** -501, 2. ** -500, 1.9999 * 2. ** 499,
                               2. ** 500, 1e-300, 5e-324, 1e308, 0., -0.])
def test_quotients_of_an_expression(t):
    # the same bits as the division: dividends and divisors over the whole
    # range, at the limits of the shorter form, and mantissas of few and many ones
    rng = numpy.random.default_rng(6)
    e = numpy.concatenate([rng.integers(-1074, 1024, 4000), rng.integers(-30, 30, 4000),
                           rng.integers(-503, -497, 500), rng.integers(497, 503, 500)])
    f = rng.choice([1., 1.5, 2. - 2. ** -52, 1. + 2. ** -52, 1. + 2. ** -23], len(e))
    f[::2] = rng.uniform(1., 2., len(f[::2]))
    x = numpy.concatenate([numpy.ldexp(f * rng.choice([-1., 1.], len(e)), e),
                           [0., -0., numpy.inf, -numpy.inf, numpy.nan, t]])
    with numpy.errstate(all="ignore"):
        for prog, ref in (("x/t", x / t), ("t/x", t / x)):
            got = evaluate_on_device(Expression(prog), x, t)
            assert numpy.array_equal(got, ref, equal_nan=True)
            num = ~numpy.isnan(ref)
            assert numpy.array_equal(numpy.signbit(got[num]), numpy.signbit(ref[num]))


def test_simulations_of_several_threads_share_no_memory():
    # what a simulation releases is handed to the next one that asks for it,
    # also of another thread and size; everything is given back when the free
    # memory is asked for
    cases = [(1, 3), (101, 40), (3000, 8), (70001, 6), (2048, 20), (250000, 4)]
    ics_of = {n: ics.sech2_disk(n, seed=n, masses="lognormal" if n % 2 else "equal")
              for n, _ in cases}

    def run(n, nleap):
        return _alone(*ics_of[n], 1.1, PULSE, 0.002, nleap)

    def free_bytes():
        sms, free, total = ctypes.c_int(), ctypes.c_int64(), ctypes.c_int64()
        assert _lib.lib().wg_device_info(ctypes.byref(sms), ctypes.byref(free),
                                         ctypes.byref(total)) == 0
        return free.value

    want = {n: run(n, nl) for n, nl in cases}
    free0 = free_bytes()
    bad = []

    def work(k):
        for r in range(4):
            for n, nl in cases[k:] + cases[:k]:
                if not _same(run(n, nl), want[n]):
                    bad.append((k, r, n))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad
    assert free_bytes() >= free0 - (64 << 20)
