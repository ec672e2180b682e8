"""Performance cases: the simulations that a user of the backend runs.

Every case is one call (or a pause and its resume) through the package's
public Python API on a scenario object and, where a program keeps one, a
`Simulation` (validated scenario, SpatiallyExplicit tables on the device) or
a resident `Batch`.  The outputs are the whole reported event stream and the
outcome's numbers.

The sizes come from the repository's benchmark configurations (synthetic.py),
its tests and the command line's defaults, and from log-uniform ranges around
them.
"""
import importlib
import math

import numpy as np

nb = importlib.import_module("necsim-rust_b200")
syn = importlib.import_module("necsim-rust_b200.synthetic")

CENTRE = 0xFFFFFFFF // 2


def listed():
    return [
        # one small simulation from scratch, as the command line runs it:
        # context, set-up, a few thousand events, tear-down
        dict(name="nonspatial_oneshot", family="oneshot", width=30, height=20, deme=2, nu=0.01),
        # the benchmark's NonSpatial configuration: 100,000 lineages
        dict(name="nonspatial_100k", family="nonspatial", width=100, height=100, deme=10, nu=1e-3),
        # ten million lineages: set-up, bulk rounds and merging dominate
        dict(name="nonspatial_10m", family="nonspatial", width=1000, height=1000, deme=10, nu=1e-3),
        # the CUDA algorithm's sampler with the command line's arguments for it
        dict(name="nonspatial_exp", family="exp", width=100, height=100, deme=10, nu=1e-3),
        # dispersal events reported (Csv, GlobalCoverage and Counter users)
        dict(name="nonspatial_dispersal", family="dispersal", width=40, height=30, deme=2, nu=5e-3),
        # a local community that is paused half way and resumed from its
        # remaining lineages
        dict(name="implicit_pause_resume", family="resume", local=30011, meta=10_000_000, migration=0.05,
             nu=1e-4, pause=150.0),
        # the batched parameter sweep, 64 simulations, plain schedule
        dict(name="implicit_sweep", family="sweep", n_sims=64, log_local_max=5.5, log_nu_min=-5.0, learned=False),
        # the same sweep with the learned lifetime schedule
        dict(name="implicit_sweep_learned", family="sweep", n_sims=64, log_local_max=5.5, log_nu_min=-5.0,
             learned=True),
        # the benchmark's AlmostInfinite configuration: Normal dispersal
        dict(name="infinite_normal", family="infinite", radius=100, nu=1e-5, sigma=10.0, shape_u=0.0, tail_p=0.0),
        # fat-tailed dispersal on an odd-sized sample
        dict(name="infinite_clark2dt", family="infinite", radius=37, nu=1e-4, sigma=0.0, shape_u=4.0, tail_p=0.5),
        # the benchmark's 64 x 64 map with dense dispersal
        dict(name="explicit_map", family="explicit", width=64, height=64, p_zero=0.15, habitat_max=50, sigma=3.0,
             nu=1e-4, turnover_map=False),
        # the command line's default noise habitat
        dict(name="wrapping_noise", family="noise", width=120, height=95, coverage=0.5, octaves=16, sigma=3.0,
             nu=1e-3),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _area(rng, lo, hi, deme_max):
    """(width, height, deme) of about a log-uniform number of individuals."""
    deme = rng.randint(1, deme_max)
    cells = max(2.0, _log(rng, lo, hi) / deme)
    width = max(1, round(math.sqrt(cells) * _log(rng, 0.5, 2.0)))
    return dict(width=width, height=max(1, round(cells / width)), deme=deme)


def draw(rng):
    family = rng.choice(["oneshot", "nonspatial", "nonspatial", "exp", "dispersal", "resume", "sweep", "sweep",
                         "infinite", "infinite", "explicit", "explicit", "noise"])
    if family == "oneshot":
        return dict(family=family, **_area(rng, 200, 2e4, 10), nu=_log(rng, 2e-3, 5e-2))
    if family == "nonspatial":
        return dict(family=family, **_area(rng, 1e3, 9e6, 10), nu=_log(rng, 2e-4, 1e-2))
    if family == "exp":
        return dict(family=family, **_area(rng, 1e3, 1e5, 10), nu=_log(rng, 1e-3, 1e-2))
    if family == "dispersal":
        return dict(family=family, **_area(rng, 200, 3e3, 5), nu=_log(rng, 5e-3, 2e-2))
    if family == "resume":
        return dict(family=family, local=round(_log(rng, 1e3, 5e4)), meta=round(_log(rng, 1e5, 1e7)),
                    migration=rng.uniform(0.01, 0.2), nu=_log(rng, 1e-4, 1e-3), pause=round(_log(rng, 20, 400), 1))
    if family == "sweep":
        return dict(family=family, n_sims=rng.randint(5, 64), log_local_max=rng.uniform(4.0, 5.5),
                    log_nu_min=rng.uniform(-5.0, -4.0), learned=rng.random() < 0.5)
    if family == "infinite":
        clark = rng.random() < 0.4
        return dict(family=family, radius=rng.randint(6, 100), nu=_log(rng, 2e-5, 2e-3),
                    sigma=0.0 if clark else _log(rng, 2.0, 20.0), shape_u=_log(rng, 1.0, 20.0) if clark else 0.0,
                    tail_p=rng.choice([0.5, 1.0, rng.uniform(0.4, 1.5)]) if clark else 0.0)
    if family == "explicit":
        return dict(family=family, width=rng.randint(9, 64), height=rng.randint(9, 64),
                    p_zero=rng.uniform(0.0, 0.3), habitat_max=round(_log(rng, 5, 100)), sigma=rng.uniform(1.0, 4.0),
                    nu=_log(rng, 1e-4, 5e-3), turnover_map=rng.random() < 0.4)
    return dict(family="noise", width=rng.randint(20, 120), height=rng.randint(20, 95),
                coverage=rng.uniform(0.2, 0.8), octaves=rng.randint(2, 16), sigma=_log(rng, 1.5, 6.0),
                nu=_log(rng, 1e-3, 2e-2))


def _sweep(case, seed):
    """Scenarios, speciation probabilities and seeds of a SpatiallyImplicit
    parameter sweep (the benchmark's ranges, bounded as the case says)."""
    n = case["n_sims"]
    u = [syn.unit(seed, n, k) for k in range(3)]
    local = np.floor(10.0 ** (3.0 + (case["log_local_max"] - 3.0) * u[0])).astype(int)
    migration = 0.01 + 0.19 * u[1]
    nu = 10.0 ** (case["log_nu_min"] + (-3.0 - case["log_nu_min"]) * u[2])
    scenarios = [nb.SpatiallyImplicit((int(local[s]), 1), 1, (10_000_000, 1), 1, float(migration[s]))
                 for s in range(n)]
    return scenarios, [float(v) for v in nu], [seed * 1000 + s for s in range(n)]


def _model(seed):
    """A lifetime model trained on traces of a few short simulations."""
    train = dict(n_sims=8, log_local_max=4.0, log_nu_min=-4.0)
    scenarios, nus, seeds = _sweep(train, seed + 7)
    X, y = nb.collect_traces(scenarios, [10.0 * v for v in nus], seeds, nb.CUDA(resident=True),
                             snapshot_rounds=32, max_rows=1 << 15)
    model = nb.LifetimeModel(seed=seed)
    model.train(X, y, epochs=4, seed=seed)
    return model


def _scenario(case, seed):
    family = case["family"]
    if family in ("oneshot", "nonspatial", "exp", "dispersal"):
        return nb.NonSpatial((case["width"], case["height"]), case["deme"])
    if family == "resume":
        return nb.SpatiallyImplicit((case["local"], 1), 1, (case["meta"], 1), 1, case["migration"])
    if family == "infinite":
        dispersal = nb.Normal(case["sigma"]) if case["sigma"] else nb.Clark2Dt(case["shape_u"], case["tail_p"])
        return nb.AlmostInfinite(nb.Circle(case["radius"], (CENTRE, CENTRE)), dispersal)
    if family == "noise":
        return nb.WrappingNoise(seed, case["coverage"], 0.07, 0.5, case["octaves"],
                                nb.Rectangle((1000, 2000), case["width"], case["height"]), case["sigma"])
    habitat = syn.habitat_map(case["width"], case["height"], case["p_zero"], case["habitat_max"], seed)
    dispersal = syn.dispersal_map(habitat, case["sigma"])
    turnover = 0.5
    if case["turnover_map"]:
        turnover = 0.1 + 0.9 * syn.unit(seed, habitat.size, 2).reshape(habitat.shape)
    return nb.SpatiallyExplicit(habitat, dispersal, turnover)


def prepare(case, seed):
    family = case["family"]
    state = dict(case=case, family=family, seed=seed)
    if family == "sweep":
        scenarios, nus, seeds = _sweep(case, seed)
        if case["learned"]:
            state["model"] = _model(seed)  # stays alive beside the batch
            algorithm = nb.CUDA(resident=True, schedule="learned", model=state["model"])
        else:
            algorithm = nb.CUDA(resident=True)
        state["batch"] = nb.Batch(scenarios, nus, seeds, algorithm)
        _result_buffers(state, case["n_sims"] * int(10.0 ** case["log_local_max"]), 1e-3)
        return state
    scenario = _scenario(case, seed)
    if family == "explicit":
        n = case["width"] * case["height"] * case["habitat_max"]
    elif family == "infinite":
        n = (2 * case["radius"] + 1) ** 2
    elif family == "noise":
        n = case["width"] * case["height"]
    else:
        n = _lineages(case)
    _result_buffers(state, n, case["nu"])
    if family == "oneshot":
        state["scenario"] = scenario
        return state
    algorithm = nb.CUDA()
    if family == "exp":
        algorithm = nb.CUDA(event_time_sampler="exp", delta_t=3.0, step_slice=150)
    elif family == "dispersal":
        algorithm = nb.CUDA(report_dispersal=True)
    state["sim"] = nb.Simulation(scenario, case["nu"], algorithm)
    return state


NUMBERS = ("steps", "n_initial", "n_remaining", "n_speciation", "biodiversity", "n_rounds", "n_dedup")
FIELDS = (("gref", np.uint64), ("prior_time", np.float64), ("event_time", np.float64), ("x", np.uint32),
          ("y", np.uint32), ("index", np.uint32))


def _event_capacity(n, nu):
    """Room for the speciation events of n lineages: one each at most, and
    for many lineages well above the few that speciate before they merge."""
    return min(n, 20_000 + int(60 * nu * n))


def _result_buffers(state, n, nu):
    """The program's own arrays, which the events of a pass are copied into
    (the number of events depends on the seed, the arrays' size does not)."""
    def events():
        return {name: np.zeros(_event_capacity(n, nu), dtype=t) for name, t in FIELDS}

    if state["family"] == "resume":
        state["out"] = [events(), events()]
        return
    state["out"] = events()
    if state["family"] == "dispersal":
        # a lineage that never merged would take 1 / nu events
        rows = 20_000 + int(1.3 * n / nu)
        state["out"]["dispersal"] = np.zeros((rows, nb.DISPERSAL_DTYPE.itemsize // 8), dtype=np.uint64)


def _fill(out, events):
    for name, _ in FIELDS:
        out[name][:len(events)] = events[name]


def _result(out, outcome):
    _fill(out, outcome.speciation)
    out["time"] = float(outcome.time)
    out["numbers"] = np.array([getattr(outcome, name) for name in NUMBERS], dtype=np.int64)
    return out


def run(state):
    case, family, seed, out = state["case"], state["family"], state["seed"], state["out"]
    if family == "oneshot":
        return _result(out, nb.simulate(case["nu"], state["scenario"], seed))
    if family == "sweep":
        outcomes = state["batch"].run(collect=True)
        _fill(out, np.concatenate([o.speciation for o in outcomes]))
        out["time"] = np.array([o.time for o in outcomes])
        out["numbers"] = np.array([[getattr(o, name) for name in NUMBERS] for o in outcomes], dtype=np.int64)
        return out
    if family == "resume":
        first = state["sim"].simulate(seed, pause_before=case["pause"])
        left = first.remaining if first.remaining is not None else np.zeros(0, dtype=nb.LINEAGE_DTYPE)
        second = state["sim"].resume(left, case["pause"], seed)
        return [_result(out[0], first), _result(out[1], second)]
    outcome = state["sim"].simulate(seed)
    out = _result(out, outcome)
    if family == "dispersal":
        words = outcome.dispersal.view(np.uint64).reshape(len(outcome.dispersal), -1)
        out["dispersal"][:len(words)] = words
    return out


# The hash work of one event (3.3 primes and 7.6 draws, 14 multiply-folds of
# 64 x 64 -> 128 bits: four 32 x 32 products and their additions each) and its
# share of diffusions, as 32-bit integer operations.
EVENT_OPERATIONS = 300.0


def _lineages(case):
    family = case["family"]
    if family in ("oneshot", "nonspatial", "exp", "dispersal"):
        return case["width"] * case["height"] * case["deme"]
    if family == "resume":
        return case["local"]
    if family == "infinite":
        return math.pi * case["radius"] ** 2
    if family == "noise":
        return case["width"] * case["height"] * case["coverage"]
    return case["width"] * case["height"] * (1.0 - case["p_zero"]) * 0.5 * (case["habitat_max"] + 1)


def work(case):
    """Events of n lineages that coalesce at the pace of a neutral community
    (n / (1 + t) lineages after t events each, until 1 / nu): n ln(1 + 1 / nu);
    each event's hash operations, and the events reported (40 bytes, 56 for a
    dispersal event).  Tables are read once."""
    if case["family"] == "sweep":
        lo, hi = 3.0 * math.log(10), case["log_local_max"] * math.log(10)
        mean = (math.exp(hi) - math.exp(lo)) / (hi - lo)
        n, nu = case["n_sims"] * mean, 10.0 ** (0.5 * (case["log_nu_min"] - 3.0))
    else:
        n, nu = _lineages(case), case["nu"]
    events = n * math.log1p(1.0 / nu)
    read = 0.0
    if case["family"] == "explicit":
        cells = case["width"] * case["height"]
        read = 32.0 * cells + 16.0 * min(events, (cells * (1.0 - case["p_zero"])) ** 2)
    written = 40.0 * max(1.0, nu * events)
    if case["family"] == "dispersal":
        written += 56.0 * events
    return dict(bytes=read + written, flops=EVENT_OPERATIONS * events)


# ---- the NonSpatial simulation with the Poisson sampler in plain numpy ----

_U = np.uint64
_P0, _P1, _P2, _P5 = (_U(v) for v in (0xA0761D6478BD642F, 0xE7037ED1A0B428DB, 0x8EBC6AF09C88C6E3,
                                      0xEB44ACCAB455D165))
_K, _PHI = _U(0x6EED0E9DA4D94A4F), _U(0x9E3779B97F4A7C15)
_M64 = (1 << 64) - 1


def _mum(a, b):
    m, s = _U(0xFFFFFFFF), _U(32)
    a0, a1, b0, b1 = a & m, a >> s, b & m, b >> s
    mid = a1 * b0 + ((a0 * b0) >> s)
    mid2 = a0 * b1 + (mid & m)
    high = a1 * b1 + (mid >> s) + (mid2 >> s)
    return (a ^ (a * b)) ^ (b ^ high)


def _diffuse(x):
    x = x * _K
    x = x ^ ((x >> _U(32)) >> (x >> _U(60)))
    return x * _K


def _swap(x):
    return (x << _U(32)) | (x >> _U(32))


def _prime(loc, t):
    return _mum(_mum(loc, _swap(_diffuse(t)) ^ _P2), _U(16) ^ _P5)


def _draw(s, k):
    v = s + _U((k * int(_P0)) & _M64)
    return _diffuse(_mum(v ^ _P1, v))


def _unit(d):
    return (d >> _U(11)).astype(np.float64) * 2.0 ** -53


def _next_events(loc, before, threshold, lam_dt):
    """Next event time after `before` at each location and its re-prime index."""
    n = len(loc)
    at, index = np.zeros(n), np.zeros(n, dtype=np.uint64)
    step = np.floor(before / 2.0).astype(np.uint64)
    todo = np.arange(n)
    while len(todo):
        s = _prime(loc[todo], step[todo])
        u = _unit(_draw(s, 1))
        count = (u[:, None] > threshold[None, :]).sum(axis=1)
        best, which = np.full(len(todo), np.inf), np.zeros(len(todo), dtype=np.uint64)
        for k in range(int(count.max(initial=0))):
            t = (step[todo].astype(np.float64) + _unit(_draw(s, k + 2))) * 2.0
            ok = (k < count) & (t > before[todo]) & (t < best)
            best[ok], which[ok] = t[ok], k
        found = np.isfinite(best)
        hit = todo[found]
        at[hit] = best[found]
        index[hit] = step[hit] + _PHI * (which[found] + _U(1))
        todo = todo[~found]
        step[todo] += _U(1)
    return at, index


def _simulate_nonspatial(width, height, deme, nu, wyhash_seed):
    lam, lam_dt = 0.5, 1.0
    threshold, prod, acc = [], math.exp(-lam_dt), math.exp(-lam_dt)
    for n in range(1, 40):
        threshold.append(acc)
        prod *= lam_dt / n
        acc += prod
    threshold = np.array(threshold)
    cells = width * height
    n0 = cells * deme
    gref = np.arange(n0, dtype=np.uint64)
    cell, idx = gref // _U(deme), gref % _U(deme)
    last, steps = np.zeros(n0), np.zeros(n0, dtype=np.int64)
    total = dict(steps=0, n_rounds=0, n_dedup=0, time=0.0)
    events, horizon = [], 0.0
    seed = _U(wyhash_seed)
    while len(gref):
        per = min(max(-(-(1 << 20) // len(gref)), 10), 1024)
        horizon += per / lam
        total["n_rounds"] += 1
        live, gone = np.arange(len(gref)), np.zeros(len(gref), dtype=bool)
        while len(live):
            loc = _swap(_diffuse(cell[live] * _U(deme) + idx[live])) ^ (seed ^ _P0)
            at, index = _next_events(loc, last[live], threshold, lam_dt)
            go = at < horizon
            live, loc, at, index = live[go], loc[go], at[go], index[go]
            s = _prime(loc, index)
            steps[live] += 1
            spec = _unit(_draw(s, 1)) < nu
            lost = live[spec]
            gone[lost] = True
            events.append((gref[lost], last[lost], at[spec], cell[lost], idx[lost]))
            total["steps"] += int(steps[lost].sum())
            live, s, at = live[~spec], s[~spec], at[~spec]
            target = np.minimum(np.floor(_unit(_draw(s, 2)) * float(cells)), cells - 1)
            cell[live] = target.astype(np.uint64)
            idx[live] = np.floor(_unit(_draw(s, 3)) * float(deme)).astype(np.uint64)
            last[live] = at
        keep = np.flatnonzero(~gone)
        order = keep[np.lexsort((gref[keep], last[keep], idx[keep], cell[keep]))]
        same = np.zeros(len(order), dtype=bool)
        same[1:] = ((cell[order[1:]] == cell[order[:-1]]) & (idx[order[1:]] == idx[order[:-1]])
                    & (last[order[1:]] == last[order[:-1]]))
        total["n_dedup"] += int(same.sum())
        total["steps"] += int(steps[order[same]].sum())
        total["time"] = max(total["time"], last[order].max(initial=0.0))
        order = np.sort(order[~same])
        gref, cell, idx, last, steps = (v[order] for v in (gref, cell, idx, last, steps))
    g, prior, at, cell, idx = (np.concatenate(v) for v in zip(*events))
    x, y = cell % _U(width), cell // _U(width)
    order = np.lexsort((g, prior, idx, y, x, at))
    g, prior, at, x, y, idx = (v[order] for v in (g, prior, at, x, y, idx))
    differ = np.ones(len(g), dtype=bool)
    differ[1:] = (x[1:] != x[:-1]) | (y[1:] != y[:-1]) | (idx[1:] != idx[:-1]) | (at[1:] != at[:-1])
    capacity = _event_capacity(n0, nu)
    padded = {}
    for name, values in zip(("gref", "prior_time", "event_time", "x", "y", "index"), (g, prior, at, x, y, idx)):
        padded[name] = np.zeros(capacity, dtype=dict(FIELDS)[name])
        padded[name][:len(g)] = values
    numbers = [total["steps"], n0, 0, len(g), int(differ.sum()), total["n_rounds"], total["n_dedup"]]
    return dict(padded, time=max(total["time"], float(at.max())), numbers=np.array(numbers, dtype=np.int64))


def _wyhash_seed(seed):
    """The WyHash seed word of `rng: Seed(seed)`: eight bytes expanded by PCG32."""
    state, out = seed & _M64, 0
    for chunk in range(2):
        state = (state * 6364136223846793005 + 11634580027462260723) & _M64
        x = (((state >> 18) ^ state) >> 27) & 0xFFFFFFFF
        r = state >> 59
        out |= (((x >> r) | (x << (32 - r))) & 0xFFFFFFFF if r else x) << (32 * chunk)
    return out


def exact(case, seed):
    """The small NonSpatial simulations restated in numpy (every operation is
    one 64-bit integer or f64 operation); others take too long that way."""
    if case["family"] not in ("oneshot", "nonspatial"):
        return None
    if case["nu"] < 9e-4 or _lineages(case) > 120_000:
        return None
    with np.errstate(over="ignore"):
        return _simulate_nonspatial(case["width"], case["height"], case["deme"], case["nu"], _wyhash_seed(seed))
