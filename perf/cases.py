"""The calls this package is timed on, each through a public entry point.

A case is a dict of plain values; ``kind`` names the entry point:

nbody     one output of the approximate generator, ``next(nbody(...))``
run       a whole approximate run from the initial conditions: set-up and a
          number of outputs of one simulation
dropin    outputs of ``approx_onestep`` on the caller's buffers, handed back
          from call to call as wendy's generator does
pool      one output of an ensemble: ``Pool.step`` and ``Pool.download_many``
diag      ``Simulation.step``, ``.energy`` and ``.download``: an output with
          its conserved quantities
accel     ``accel``: one force evaluation on host arrays
noalloc   ``wg_accel_noalloc``: one force evaluation on device arrays the
          caller owns
exact     one output of the exact event-driven generator

Initial conditions are the package's three families (sech^2 disk, cold
top-hat, Gaussian blob) and ``slab``: the cold top-hat at a later phase of its
collapse, in closed form.
"""
import ctypes
import math

import numpy
import torch

import wendy_gb300
from wendy_gb300 import _lib
from wendy_gb300.ensemble import Pool
from wendy_gb300.extforce import Expression, PulseTanh

# The pulsed force of the top-hat workload, and an anharmonic time-dependent
# restoring force given as an expression.
PULSE = (0.3, 5.0, 1.0, 0.5)
BREATHING = "-0.5*(1.0+0.3*sin(2.0*t))*x**3/(1.0+x**2)"


def listed():
    return [
        # wendy's own small approximate tests: a hundred sheets, many short
        # sub-steps per output; nothing but latency
        dict(name="nbody_101", kind="nbody", family="sech2", masses="equal", n=101, dt=0.05,
             nleap=1000, omega=0.0, force="none"),
        # the usual notebook-sized disk
        dict(name="nbody_1e4", kind="nbody", family="sech2", masses="equal", n=10000, dt=0.05,
             nleap=10, omega=0.0, force="none"),
        # a medium run of odd size with unequal masses, a harmonic background
        # and a force written as an expression
        dict(name="nbody_300007_expr", kind="nbody", family="gaussian", masses="lognormal",
             n=300007, dt=0.02, nleap=10, omega=0.5, force="breathing"),
        # the large disk: lognormal masses in a harmonic background
        dict(name="nbody_2p24_omega", kind="nbody", family="sech2", masses="lognormal",
             n=1 << 24, dt=0.02, nleap=20, omega=1.1, force="none"),
        # the largest workload: the cold top-hat with the pulsed force
        dict(name="nbody_2p27_pulse", kind="nbody", family="tophat", masses="equal", n=1 << 27,
             dt=0.01, nleap=10, omega=0.0, force="pulse"),
        # a run through the collapse of a cold slab, where the flow crowds the
        # sheets and the local repair of the order gives way to full sorts
        dict(name="run_collapse_1e6", kind="run", family="slab", masses="equal", n=1000003,
             phase=1.5, dt=0.01, nleap=10, outputs=12, omega=0.0, force="none"),
        # wendy's step function replaced call by call in an existing program
        dict(name="dropin_400009_pulse", kind="dropin", family="sech2", masses="equal", n=400009,
             dt=0.01, nleap=10, outputs=4, omega=0.0, force="pulse", t0=4.0),
        # an ensemble: uneven members, each with its own time step and omega
        dict(name="pool_192", kind="pool", members=192, lo=1000, hi=1000000, nleap=10),
        # an output with its energy and momentum
        dict(name="diag_2p21", kind="diag", family="sech2", masses="lognormal", n=(1 << 21) + 77,
             dt=0.02, nleap=10, omega=1.1, force="none"),
        # one force evaluation on a program's own arrays (initial
        # accelerations, diagnostics)
        dict(name="accel_150001", kind="accel", family="gaussian", masses="lognormal", n=150001,
             omega=1.1, force="none"),
        # the same inside a program that owns the device memory and cannot
        # have it allocated behind its back
        dict(name="noalloc_20011", kind="noalloc", family="sech2", masses="lognormal", n=20011,
             omega=0.5, force="pulse"),
        # the exact solver as the cross-check of a small run
        dict(name="exact_1001", kind="exact", family="sech2", masses="equal", n=1001, dt=0.05,
             omega=0.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["nbody", "nbody", "nbody", "nbody", "run", "dropin", "pool", "diag",
                       "accel", "noalloc", "exact"])
    fam = rng.choice(["sech2", "gaussian"])
    masses = rng.choice(["equal", "lognormal"])
    omega = rng.choice([0.0, 0.5, 1.1])
    force = rng.choice(["none", "none", "pulse", "breathing", "harmonic"])
    dt = rng.uniform(0.005, 0.05)
    if kind == "nbody":
        n = _log(rng, 64, 1 << 26)
        nleap = max(3, min(rng.choice([5, 10, 20, 100, 1000]), int(5e8) // n))
        if n > 1 << 18 and rng.random() < 0.3:
            fam, omega, dt = "tophat", 0.0, 0.002
        return dict(kind=kind, family=fam, masses=masses, n=n, dt=dt, nleap=nleap, omega=omega,
                    force=force)
    if kind == "run":
        return dict(kind=kind, family="slab", masses=masses, n=_log(rng, 20000, 1500000),
                    phase=rng.uniform(1.35, 1.55), dt=0.01, nleap=10, outputs=rng.randint(4, 12),
                    omega=0.0, force="none")
    if kind == "dropin":
        return dict(kind=kind, family=fam, masses=masses, n=_log(rng, 1000, 4000000), dt=dt,
                    nleap=rng.choice([5, 10, 20]), outputs=rng.randint(2, 5), omega=omega,
                    force=force, t0=rng.uniform(0.0, 6.0))
    if kind == "pool":
        return dict(kind=kind, members=_log(rng, 4, 256), lo=rng.choice([500, 1000, 3000]),
                    hi=rng.choice([20000, 200000, 1000000]), nleap=rng.choice([5, 10, 20]))
    if kind == "diag":
        return dict(kind=kind, family=fam, masses=masses, n=_log(rng, 1000, 1 << 23), dt=dt,
                    nleap=rng.choice([5, 10, 20]), omega=omega, force=force)
    if kind == "accel":
        return dict(kind=kind, family=fam, masses=masses, n=_log(rng, 100, 1 << 22), omega=omega,
                    force=force)
    if kind == "noalloc":
        force = "pulse" if force == "breathing" else force
        return dict(kind=kind, family=fam, masses=masses,
                    n=_log(rng, 50, _lib.NOALLOC_MAX_SHEETS), omega=omega, force=force)
    n = _log(rng, 51, 4001)
    return dict(kind="exact", family="sech2", masses=masses, n=n,
                dt=min(0.05, 5000.0 / (0.094 * n * n)), omega=rng.choice([0.0, 0.0, 1.1]))


# ---- initial conditions ------------------------------------------------------
def _sheets(case, seed, n=None, family=None, masses=None):
    """x, v, m on the GPU, from the seed alone."""
    n = case["n"] if n is None else n
    family = case["family"] if family is None else family
    masses = case.get("masses", "equal") if masses is None else masses
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * seed + n)
    f8 = dict(dtype=torch.float64, device="cuda", generator=g)
    if family == "sech2":
        x = 2.0 * torch.atanh(2.0 * torch.rand(n, **f8).clamp_(1e-15, 1.0 - 1e-15) - 1.0)
        v = torch.randn(n, **f8)
    elif family == "gaussian":
        x = torch.randn(n, **f8)
        v = torch.randn(n, **f8)
    else:
        x = 2.0 * torch.rand(n, **f8) - 1.0
        v = 1e-3 * torch.randn(n, **f8)
        if family == "slab":
            # a uniform cold slab of unit mass on [-1, 1] feels a = -x
            c, s = math.cos(case["phase"]), math.sin(case["phase"])
            x, v = x * c + v * s, v * c - x * s
    if masses == "lognormal":
        m = torch.exp(0.5 * torch.randn(n, **f8))
        m /= m.sum()
    else:
        m = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    return x, v, m


def _host(*arrays):
    return tuple(a.cpu().numpy() for a in arrays)


def _force(case):
    name = case.get("force", "none")
    if name == "pulse":
        return PulseTanh(*PULSE)
    if name == "breathing":
        return Expression(BREATHING)
    if name == "harmonic":
        return wendy_gb300.Harmonic(0.4)
    return None


def _omega(case):
    return case["omega"] if case["omega"] > 0 else None


def _members(case):
    """Size, time step, omega, family and masses of each member of an ensemble."""
    k = case["members"]
    out = []
    for i in range(k):
        n = int(round(case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / k)))
        out.append((n, 0.005 + 0.045 * ((7 * i) % k) / k, (0.0, 0.5, 1.1)[i % 3],
                    ("sech2", "gaussian")[i % 2], ("equal", "lognormal")[(i // 2) % 2]))
    return out


# ---- what a program has in hand before the call ----------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "pool":
        pool, ids, dts, total = Pool(), [], [], 0
        for i, (n, dt, om, fam, masses) in enumerate(_members(case)):
            x, v, m = _host(*_sheets(case, seed + 7919 * i, n, fam, masses))
            ids.append(pool.add(x, v, m, omega=om if om > 0 else None))
            dts.append(dt / case["nleap"])
            total += n
        return dict(case=case, pool=pool, ids=numpy.array(ids, dtype=numpy.int32),
                    dts=numpy.array(dts), x=_lib.pinned_empty(total), v=_lib.pinned_empty(total))
    if kind == "noalloc":
        x, _, m = _sheets(case, seed)
        force = _force(case)
        params = _lib.ext_params(force.params if force else ())
        return dict(case=case, x=x, m=m, tot=float(m.sum()), a=torch.empty_like(x),
                    perm=torch.empty(case["n"], dtype=torch.int32, device="cuda"),
                    kind=force.kind if force else 0, params=params,
                    np=len(force.params) if force else 0)
    x, v, m = _host(*_sheets(case, seed))
    if kind == "nbody":
        # the generator with its first output taken: set up, in its loop
        g = wendy_gb300.nbody(x, v, m, case["dt"], approx=True, nleap=case["nleap"],
                              omega=_omega(case), ext_force=_force(case))
        next(g)
        return dict(case=case, gen=g)
    if kind == "exact":
        g = wendy_gb300.nbody(x, v, m, case["dt"], omega=_omega(case), maxcoll=10 ** 7)
        next(g)
        return dict(case=case, gen=g)
    if kind == "run":
        return dict(case=case, x=x, v=v, m=m)
    if kind == "diag":
        om = case["omega"]
        sim = wendy_gb300.Simulation(x, v, m, numpy.sum(m), om ** 2 if om > 0 else -1.0,
                                     _force(case))
        return dict(case=case, sim=sim, t=ctypes.c_double(0.0), x=x, v=v)
    if kind == "accel":
        return dict(case=case, x=x, m=m, tot=numpy.sum(m), force=_force(case))
    n = case["n"]
    xi = numpy.zeros(n, dtype=_lib.SHEET_DTYPE)
    xi["idx"] = numpy.arange(n, dtype=numpy.int32)
    xi["val"] = x
    return dict(case=case, xi=xi, x=x, v=v, m=m, a=numpy.zeros(n), tot=numpy.sum(m),
                t=case["t0"], force=_force(case))


# ---- one pass ---------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("nbody", "exact"):
        x, v = next(state["gen"])
        return {"x": x, "v": v}
    if kind == "run":
        g = wendy_gb300.nbody(state["x"], state["v"], state["m"], case["dt"], approx=True,
                              nleap=case["nleap"], omega=_omega(case), ext_force=_force(case))
        for _ in range(case["outputs"]):
            x, v = next(g)
        g.close()
        return {"x": x, "v": v}
    if kind == "dropin":
        om = case["omega"]
        for _ in range(case["outputs"]):
            state["t"], _el = wendy_gb300.approx_onestep(
                state["xi"], state["x"], state["v"], state["m"], state["a"], state["tot"],
                case["dt"] / case["nleap"], case["nleap"], state["t"],
                om ** 2 if om > 0 else -1.0, state["force"])
        return {"x": state["x"], "v": state["v"], "a": state["a"], "idx": state["xi"]["idx"],
                "val": state["xi"]["val"]}
    if kind == "pool":
        state["pool"].step(state["ids"], state["dts"], case["nleap"])
        x, v = state["pool"].download_many(state["ids"], state["x"], state["v"])
        return {"x": x, "v": v}
    if kind == "diag":
        sim = state["sim"]
        sim.step(case["dt"] / case["nleap"], case["nleap"], state["t"])
        energy, momentum = sim.energy(omega=_omega(case))
        sim.download(state["x"], state["v"])
        return {"x": state["x"], "v": state["v"], "energy": energy, "momentum": momentum}
    om = case["omega"]
    omega2 = om ** 2 if om > 0 else -1.0
    if kind == "accel":
        a, perm = wendy_gb300.accel(state["x"], state["m"], state["tot"], omega2, state["force"],
                                    4.2)
        return {"a": a, "perm": perm}
    _lib.check(_lib.lib().wg_accel_noalloc(
        case["n"], state["x"].data_ptr(), state["m"].data_ptr(), state["tot"], omega2,
        state["kind"], state["params"], state["np"], 4.2, state["a"].data_ptr(),
        state["perm"].data_ptr(), torch.cuda.current_stream().cuda_stream), "wg_accel_noalloc")
    return {"a": state["a"], "perm": state["perm"]}


def work(case):
    """56 bytes per sheet and sub-step (28 read, 28 written) and 16 per sheet
    and output for the approximate paths; the inputs and outputs alone for a
    force evaluation; the state of the sheets in and out, and three pair
    times per crossing, for the exact solver."""
    kind = case["kind"]
    if kind == "pool":
        n = sum(m[0] for m in _members(case))
        return {"bytes": n * (56.0 * case["nleap"] + 16), "flops": 20.0 * n * case["nleap"]}
    n = float(case["n"])
    if kind in ("accel", "noalloc"):
        return {"bytes": 28.0 * n, "flops": 10.0 * n}
    if kind == "exact":
        events = 0.094 * n * n * case["dt"]
        return {"bytes": 80.0 * n, "flops": 60.0 * events}
    steps = case["nleap"] * case.get("outputs", 1)
    per_output = {"nbody": 16.0, "run": 16.0, "dropin": 72.0, "diag": 44.0}[kind]
    return {"bytes": n * (56.0 * steps + per_output * case.get("outputs", 1)),
            "flops": 20.0 * n * steps}


# ---- the same quantities in 64 bits, by sorting and summing ------------------------
def _ext(case, x, t):
    name = case.get("force", "none")
    if name == "pulse":
        a, t0, tau, h = PULSE
        return a * math.exp(-(t - t0) ** 2 / (2 * tau ** 2)) * torch.tanh(x / h)
    if name == "breathing":
        return -0.5 * (1 + 0.3 * math.sin(2 * t)) * x ** 3 / (1 + x ** 2)
    if name == "harmonic":
        return -(0.4 ** 2) * x
    return 0.0


def _accel(case, x, m, tot, omega, t, external=True):
    order = torch.sort(x, stable=True).indices
    ms = m[order]
    a = torch.empty_like(x)
    a[order] = tot - 2.0 * (torch.cumsum(ms, 0) - ms) - ms
    if omega > 0:
        a -= omega ** 2 * x
    if external:
        a += _ext(case, x, t)
    return a, order


def _leapfrog(case, x, v, m, dt, nleap, omega, t):
    """One output of drift-kick-drift sub-steps; the time of the force lags."""
    tot = m.sum().item()
    h = dt / nleap
    x = x + 0.5 * h * v
    for i in range(nleap):
        a, order = _accel(case, x, m, tot, omega, t)
        t += h
        v = v + h * a
        x = x + (h if i < nleap - 1 else 0.5 * h) * v
    return x, v, a, order, t


def exact(case, seed):
    kind = case["kind"]
    if kind == "exact":
        return _exact_events(case, seed)
    if kind == "pool":
        xs, vs = [], []
        for i, (n, dt, om, fam, masses) in enumerate(_members(case)):
            x, v, m = _sheets(case, seed + 7919 * i, n, fam, masses)
            x, v, _, _, _ = _leapfrog(case, x, v, m, dt, case["nleap"], om, 0.0)
            xs.append(x)
            vs.append(v)
        return {"x": torch.cat(xs), "v": torch.cat(vs)}
    x, v, m = _sheets(case, seed)
    if kind in ("accel", "noalloc"):
        a, _ = _accel(case, x, m, m.sum().item(), case["omega"], 4.2)
        return {"a": a, "perm": None}
    t = case.get("t0", 0.0)
    outputs = 2 if kind == "nbody" else case.get("outputs", 1)
    for _ in range(outputs):
        x, v, a, order, t = _leapfrog(case, x, v, m, case["dt"], case["nleap"], case["omega"], t)
    if kind == "dropin":
        return {"x": x, "v": v, "a": a, "idx": None, "val": x[order]}
    if kind == "diag":
        g, _ = _accel(case, x, m, m.sum().item(), 0.0, 0.0, external=False)
        energy = (m * v * v).sum() / 2 + case["omega"] ** 2 * (m * x * x).sum() / 2 \
            - (m * x * g).sum()
        return {"x": x, "v": v, "energy": energy.item(), "momentum": (m * v).sum().item()}
    return {"x": x, "v": v}


def _exact_events(case, seed):
    """The first two outputs, crossing by crossing (no harmonic background)."""
    if case["omega"] > 0 or case["n"] > 4001:
        return None
    x, v, m = _host(*_sheets(case, seed))
    n = len(x)
    order = numpy.argsort(x)
    ms = m[order]
    below = numpy.cumsum(ms) - ms
    acc = numpy.empty(n)
    acc[order] = (ms.sum() - below - ms) - below
    x, v, acc, m = x.tolist(), v.tolist(), acc.tolist(), m.tolist()
    order = order.tolist()
    clock = [0.0] * n
    now = 0.0

    def at(s):
        d = now - clock[s]
        return x[s] + v[s] * d + 0.5 * acc[s] * d * d, v[s] + acc[s] * d

    def meet(i):
        """Time at which the pair at places i, i + 1 (x_i < x_j) meets."""
        p, q = order[i], order[i + 1]
        (xp, vp), (xq, vq) = at(p), at(q)
        b, c = (vp - vq) / (acc[p] - acc[q]), 2.0 * (xp - xq) / (acc[p] - acc[q])
        return now - b + math.sqrt(max(b * b - c, 0.0))

    pairs = numpy.array([meet(i) for i in range(n - 1)])
    end = 2 * case["dt"]
    while True:
        i = int(numpy.argmin(pairs))
        if pairs[i] >= end:
            break
        now = float(pairs[i])
        p, q = order[i], order[i + 1]
        for s in (p, q):
            x[s], v[s] = at(s)
            clock[s] = now
        order[i], order[i + 1] = q, p
        dm = m[q] - m[p]
        acc[p], acc[q] = acc[q] - dm, acc[p] - dm
        # the pair just met: the other root of its quadratic
        pairs[i] = now + 2.0 * (v[p] - v[q]) / (acc[q] - acc[p])
        if i > 0:
            pairs[i - 1] = meet(i - 1)
        if i + 2 < n:
            pairs[i + 1] = meet(i + 1)
    now = end
    for s in range(n):
        x[s], v[s] = at(s)
    return {"x": numpy.array(x), "v": numpy.array(v)}
