"""The lone-lineage kernel form (chain_run) at the edges of its rule: worlds of
one cell, 2^32 - 1 cells and beyond, a metacommunity that reaches into the
local extent, time buckets with many events or almost none, delta_t that is no
power of two (the general form), every event a speciation or a migration,
interrupted rounds and wide displacements, all against the oracle's canonical
schedule bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import same_stream

pytestmark = pytest.mark.gpu

M32 = 0xFFFFFFFF


def ns(w, h, deme, nu):
    return dict(kind=0, speciation_probability=nu, width=w, height=h, deme=deme)


def si(local, deme, meta, meta_deme, migration, nu, height=1, meta_height=1):
    return dict(kind=1, speciation_probability=nu, width=local, height=height, deme=deme, meta_width=meta,
                meta_height=meta_height, meta_deme=meta_deme, migration_probability=migration)


def ai(radius, sigma, nu, centre=(M32 // 2, M32 // 2)):
    return dict(kind=2, speciation_probability=nu, sigma=sigma, radius=radius, centre_x=centre[0],
                centre_y=centre[1])


CASES = {
    # name: (scenario, kernel arguments, resumed lineages (None: every origin))
    "one_cell": (ns(1, 1, 1, 0.02), {}, None),
    "one_column": (ns(1, 37, 3, 0.01), {}, None),
    "every_event_speciates": (ns(9, 5, 2, 1.0), {}, None),
    "cells_below_2_32": (ns(65535, 65537, 7, 0.01), {}, 40),   # 2^32 - 1 cells
    "cells_2_32": (ns(65536, 65536, 7, 0.01), {}, 40),         # the general form
    "cells_above_2_32": (ns(M32, 3, 2, 0.01), {}, 40),
    "many_events_per_bucket": (ns(20, 11, 3, 0.004), dict(delta_t=32.0), None),
    "four_events_per_bucket": (ns(20, 11, 3, 0.004), dict(delta_t=8.0), None),
    "few_events_per_bucket": (ns(12, 7, 3, 0.01), dict(delta_t=0.0625), None),
    "delta_t_no_power_of_two": (ns(20, 11, 3, 0.004), dict(delta_t=3.0), None),
    "short_rounds": (ns(20, 11, 3, 0.004), dict(step_slice=1, min_round_events=1), None),
    "local_only_by_chance": (si(15, 2, 1000, 3, 1e-3, 0.01), {}, None),
    "every_event_migrates": (si(15, 2, 1000, 3, 1.0, 0.01), {}, None),
    "demes_and_rows": (si(6, 5, 40, 4, 0.2, 0.01, height=4, meta_height=9), {}, None),
    "meta_inside_local": (si(50, 2, M32, 3, 0.3, 0.01), {}, None),
    "meta_cells_above_2_32": (si(50, 2, 70000, 3, 0.3, 0.01, meta_height=70000), {}, None),
    "meta_many_events": (si(15, 2, 1000, 3, 0.1, 0.01), dict(delta_t=16.0), None),
    "wide_displacements": (ai(4, 3e8, 0.01), {}, None),
    "no_displacement": (ai(4, 0.0, 0.01, centre=(1, M32)), {}, None),
    "narrow_displacements": (ai(5, 0.4, 0.01, centre=(1, M32)), {}, None),
    "sigma_64": (ai(5, 64.0, 0.002), {}, None),  # the widest that 32-bit arithmetic decides
    "sigma_above_64": (ai(5, 64.0001, 0.002), {}, None),
    "clark_tiny": (dict(kind=4, speciation_probability=0.005, shape_u=1e-9, tail_p=3.0, radius=4, centre_x=2,
                        centre_y=M32 - 1), {}, None),
    "clark_wide": (dict(kind=4, speciation_probability=0.01, shape_u=1e9, tail_p=1.0, radius=4, centre_x=2,
                        centre_y=M32 - 1), {}, None),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("batch", [False, True])
def test_matches_oracle(nb, syn, oracle, name, batch):
    desc, kw, resumed = CASES[name]
    oracle_kw = dict(dict(step_slice=10, min_round_events=1 << 20), **kw)
    if resumed is not None:
        lins = np.zeros(resumed, dtype=nb.LINEAGE_DTYPE)
        u = syn.splitmix64(3, 3 * resumed)
        lins["x"] = u[:resumed] % np.uint64(desc["width"])
        lins["y"] = u[resumed:2 * resumed] % np.uint64(desc["height"])
        lins["index"] = u[2 * resumed:] % np.uint64(desc["deme"])
        lins["gref"] = np.arange(resumed)
        if batch:
            pytest.skip("batches start from every origin")
        with nb.Simulation(syn.to_scenario(desc), desc["speciation_probability"], nb.CUDA(**kw)) as sim:
            g = sim.resume(lins, 0.0, 5)
        c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, lineages=lins, step_slice_max=1024, **oracle_kw)
    elif batch:
        # beside another simulation and in the resident kernel
        other = dict(desc, speciation_probability=min(1.0, 2.0 * desc["speciation_probability"]))
        pair = [desc, other]
        g = nb.simulate_batch([syn.to_scenario(d) for d in pair], [d["speciation_probability"] for d in pair],
                              [5, 6], nb.CUDA(resident=True, **kw), collect=True)[0]
        c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice_max=1024, **oracle_kw)
    else:
        with nb.Simulation(syn.to_scenario(desc), desc["speciation_probability"], nb.CUDA(**kw)) as sim:
            g = sim.simulate(5)
        c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice_max=1024, **oracle_kw)
    assert same_stream(g.speciation, c.speciation)
    assert (g.steps, g.n_rounds, g.n_dedup, g.time) == (c.steps, c.n_rounds, c.n_dedup, c.time)


@pytest.mark.parametrize("name", ["four_events_per_bucket", "demes_and_rows", "narrow_displacements"])
@pytest.mark.parametrize("pause", [7.25, 40.0])
def test_pause_and_dispersal_events(nb, syn, oracle, name, pause):
    """The peek kept over a pause, and every executed event reported."""
    desc, kw, _ = CASES[name]
    algo = nb.CUDA(report_dispersal=True, **kw)
    with nb.Simulation(syn.to_scenario(desc), desc["speciation_probability"], algo) as sim:
        g = sim.simulate(5, pause_before=pause)
    c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice=10, min_round_events=1 << 20,
                        step_slice_max=1024, pause_before=pause, report_dispersal=True, dispersal_cap=1 << 20, **kw)
    assert same_stream(g.speciation, c.speciation)
    a = np.sort(g.dispersal, order=("event_time", "gref"))
    b = np.sort(c.dispersal, order=("event_time", "gref"))
    assert len(a) == len(b) > 0
    for f in ("gref", "prior_time", "event_time", "x", "y", "index", "tx", "ty", "tindex"):
        assert np.array_equal(a[f], b[f]), f
    rem, crem = np.sort(g.remaining, order="gref"), np.sort(c.remaining, order="gref")
    for f in ("gref", "x", "y", "index", "last_event_time"):
        assert np.array_equal(rem[f], crem[f]), f


@pytest.mark.parametrize("n", [147, 148, 149, 296, 297, 592, 593, 2368, 2369, 9471, 9472, 9473, 9600, 18944, 18945])
@pytest.mark.parametrize("kind", [0, 2])
def test_round_sizes(nb, syn, oracle, n, kind):
    """Lineage counts at the edges of the warps, blocks and kernels that take
    a round (148 SMs, four warps per block, four lineages per resident warp)."""
    if kind == 0:
        desc = ns(n, 1, 1, 0.05)
    else:
        desc = dict(kind=2, speciation_probability=0.05, sigma=2.0, sample=(7, 9, n, 1))
    with nb.Simulation(syn.to_scenario(desc), 0.05, nb.CUDA(step_slice=2, min_round_events=1)) as sim:
        g = sim.simulate(5)
    c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice_max=1024, step_slice=2, min_round_events=1)
    assert same_stream(g.speciation, c.speciation)
    assert (g.steps, g.n_rounds, g.n_dedup, g.time) == (c.steps, c.n_rounds, c.n_dedup, c.time)


def se(syn, w, h, sigma, nu, cell=12, p_zero=0.2, dispersal=None, seed=3, **kw):
    hab = syn.habitat_map(w, h, p_zero, cell, seed)
    hab.flat[0] = max(1, hab.flat[0])
    disp = syn.dispersal_map(hab, sigma) if dispersal is None else dispersal(hab)
    return dict(kind=3, speciation_probability=nu, width=w, height=h, habitat=hab, dispersal=disp, **kw)


def only_self(hab):
    return np.diag((hab.reshape(-1) > 0).astype(np.float64))


def never_self(hab):
    d = np.tile((hab.reshape(-1) > 0).astype(np.float64), (hab.size, 1))
    np.fill_diagonal(d, 0.0)
    d[hab.reshape(-1) == 0] = 0.0
    return d


SE_CASES = {
    # name: (scenario, kernel arguments)
    "one_cell": (lambda syn: se(syn, 1, 1, 1.0, 0.02, p_zero=0.0), {}),
    "one_row": (lambda syn: se(syn, 23, 1, 1.0, 0.01), {}),
    "self_only": (lambda syn: se(syn, 7, 5, 1.0, 0.01, dispersal=only_self), {}),
    "self_never": (lambda syn: se(syn, 7, 5, 1.0, 0.01, dispersal=never_self), {}),
    "narrow": (lambda syn: se(syn, 11, 9, 0.3, 0.01), {}),
    "many_events_per_bucket": (lambda syn: se(syn, 11, 9, 2.0, 0.005), dict(delta_t=16.0)),
    "few_events_per_bucket": (lambda syn: se(syn, 11, 9, 2.0, 0.02), dict(delta_t=0.125)),
    "delta_t_no_power_of_two": (lambda syn: se(syn, 11, 9, 2.0, 0.005), dict(delta_t=3.0)),
    "short_rounds": (lambda syn: se(syn, 11, 9, 2.0, 0.01), dict(step_slice=1, min_round_events=1)),
    "every_event_speciates": (lambda syn: se(syn, 5, 4, 2.0, 1.0), {}),
    "turnover_map": (lambda syn: se(syn, 11, 9, 2.0, 0.005,
                                    turnover_map=0.1 + 3.0 * syn.unit(9, 99, 4).reshape(9, 11)), {}),
}


@pytest.mark.parametrize("name", sorted(SE_CASES))
@pytest.mark.parametrize("batch", [False, True])
def test_explicit_matches_oracle(nb, syn, oracle, name, batch):
    """SpatiallyExplicit: every candidate reads its own alias atom and record."""
    make, kw = SE_CASES[name]
    desc = make(syn)
    nu = desc["speciation_probability"]
    if batch:
        g = nb.simulate_batch([syn.to_scenario(desc)] * 2, [nu, min(1.0, 2 * nu)], [5, 6],
                              nb.CUDA(resident=True, **kw), collect=True)[0]
    else:
        with nb.Simulation(syn.to_scenario(desc), nu, nb.CUDA(**kw)) as sim:
            g = sim.simulate(5)
    oracle_kw = dict(dict(step_slice=10, min_round_events=1 << 20), **kw)
    c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice_max=1024, **oracle_kw)
    assert g.steps == c.steps > 0
    assert same_stream(g.speciation, c.speciation)
    assert (g.n_rounds, g.n_dedup, g.time) == (c.n_rounds, c.n_dedup, c.time)


def test_explicit_dispersal_events(nb, syn, oracle):
    desc = se(syn, 11, 9, 1.0, 0.01)
    with nb.Simulation(syn.to_scenario(desc), 0.01, nb.CUDA(report_dispersal=True)) as sim:
        g = sim.simulate(5, pause_before=60.0)
    c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice=10, min_round_events=1 << 20,
                        step_slice_max=1024, pause_before=60.0, report_dispersal=True, dispersal_cap=1 << 20)
    assert same_stream(g.speciation, c.speciation)
    a = np.sort(g.dispersal, order=("event_time", "gref"))
    b = np.sort(c.dispersal, order=("event_time", "gref"))
    assert len(a) == len(b) > 0
    for f in ("gref", "prior_time", "event_time", "x", "y", "index", "tx", "ty", "tindex"):
        assert np.array_equal(a[f], b[f]), f
    rem, crem = np.sort(g.remaining, order="gref"), np.sort(c.remaining, order="gref")
    for f in ("gref", "x", "y", "index", "last_event_time"):
        assert np.array_equal(rem[f], crem[f]), f


@pytest.mark.parametrize("desc", [
    dict(kind=2, sigma=10.0), dict(kind=2, sigma=0.7), dict(kind=2, sigma=60.0),
    dict(kind=4, shape_u=4.0, tail_p=0.5), dict(kind=4, shape_u=1.0, tail_p=1.0), dict(kind=4, shape_u=20.0, tail_p=0.4),
], ids=lambda d: "-".join("%s" % v for v in d.values()))
def test_displacements_decided_in_32_bits(nb, syn, oracle, desc):
    """Some 10^6 events: several thousand targets are not decided by the 32-bit
    arithmetic; one wrong rounding would move a lineage for good.  (The steep
    Clark2Dt tails reach beyond 2^32 cells.)"""
    desc = dict(desc, speciation_probability=1e-3, radius=18, centre_x=M32 // 2, centre_y=3)
    g = nb.simulate(1e-3, syn.to_scenario(desc), 9)
    c = oracle.simulate(desc, 9, mode=oracle.MODE_CANONICAL, step_slice=10, min_round_events=1 << 20,
                        step_slice_max=1024)
    assert g.steps == c.steps > 500_000
    assert same_stream(g.speciation, c.speciation)


EXP_CASES = sorted(n for n in CASES if CASES[n][2] is None) + ["explicit-" + n for n in sorted(SE_CASES)]


@pytest.mark.parametrize("name", EXP_CASES)
@pytest.mark.parametrize("batch", [False, True])
def test_exponential_sampler(nb, syn, oracle, name, batch):
    """The exponential sampler's form: buckets that hold many samples or whose
    first sample is past the end, at the same edges."""
    if name.startswith("explicit-"):
        make, kw = SE_CASES[name[len("explicit-"):]]
        desc = make(syn)
    else:
        desc, kw, _ = CASES[name]
    nu = desc["speciation_probability"]
    kw = dict(dict(delta_t=3.0), **kw)
    algo = nb.CUDA(event_time_sampler="exp", resident=batch, **kw)
    if batch:
        g = nb.simulate_batch([syn.to_scenario(desc)] * 2, [nu, min(1.0, 2 * nu)], [5, 6], algo, collect=True)[0]
    else:
        with nb.Simulation(syn.to_scenario(desc), nu, algo) as sim:
            g = sim.simulate(5)
    oracle_kw = dict(dict(step_slice=10, min_round_events=1 << 20), **kw)
    c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice_max=1024, event_time_sampler=oracle.SAMPLER_EXP,
                        **oracle_kw)
    assert g.steps == c.steps > 0
    assert same_stream(g.speciation, c.speciation)
    assert (g.n_rounds, g.n_dedup, g.time) == (c.n_rounds, c.n_dedup, c.time)


@pytest.mark.parametrize("n", [147, 149, 1776, 1777, 7104, 7105, 9472, 9473])
def test_exponential_round_sizes(nb, syn, oracle, n):
    desc = ns(n, 1, 1, 0.05)
    algo = nb.CUDA(event_time_sampler="exp", step_slice=2, min_round_events=1)
    with nb.Simulation(syn.to_scenario(desc), 0.05, algo) as sim:
        g = sim.simulate(5)
    c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice_max=1024, step_slice=2, min_round_events=1,
                        event_time_sampler=oracle.SAMPLER_EXP)
    assert same_stream(g.speciation, c.speciation)
    assert (g.steps, g.n_rounds, g.n_dedup, g.time) == (c.steps, c.n_rounds, c.n_dedup, c.time)


@pytest.mark.parametrize("side", [45, 46])
@pytest.mark.parametrize("sampler", ["poisson", "exp"])
def test_explicit_table_sizes(nb, syn, oracle, side, sampler):
    """2025^2 and 2116^2 alias atoms: either side of the table size above which
    only the selected lane reads its atom.  (The tests above have tables on
    either side of the size that is read through L1.)"""
    desc = se(syn, side, side, 4.0, 0.02, cell=1, p_zero=0.0)
    desc["habitat"] = np.ones_like(desc["habitat"])
    desc["dispersal"] = np.ones((side * side, side * side))
    with nb.Simulation(syn.to_scenario(desc), 0.02, nb.CUDA(event_time_sampler=sampler, report_dispersal=True)) as sim:
        g = sim.simulate(5)
    c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice=10, min_round_events=1 << 20,
                        step_slice_max=1024, report_dispersal=True, dispersal_cap=1 << 20,
                        event_time_sampler=oracle.SAMPLER_EXP if sampler == "exp" else oracle.SAMPLER_POISSON)
    assert g.steps == c.steps > 50_000
    assert same_stream(g.speciation, c.speciation)
    a = np.sort(g.dispersal, order=("event_time", "gref"))
    b = np.sort(c.dispersal, order=("event_time", "gref"))
    for f in ("gref", "prior_time", "event_time", "x", "y", "index", "tx", "ty", "tindex"):
        assert np.array_equal(a[f], b[f]), f
    with nb.Simulation(syn.to_scenario(desc), 0.02, nb.CUDA(event_time_sampler=sampler)) as sim:
        assert same_stream(sim.simulate(5).speciation, c.speciation)
