"""Event streams large enough for the device's event sort: PackedEvent order
(event.rs:256-280) of everything delivered, ties included, at the edges of the
sort's tiles (2,048 records) and with more simulations than one digit holds."""
import numpy as np
import pytest

from test_gpu_parity import same_stream

pytestmark = pytest.mark.gpu


def packed_order(e):
    """np.lexsort keys of PackedEvent::cmp, last key first."""
    t = e["event_time"].view(np.uint64)
    if "tx" in e.dtype.names:
        return np.lexsort((e["gref"], e["prior_time"].view(np.uint64), e["tindex"], e["ty"], e["tx"], e["index"],
                           e["y"], e["x"], t))
    return np.lexsort((e["gref"], e["prior_time"].view(np.uint64), e["index"], e["y"], e["x"], t))


@pytest.mark.parametrize("n", [8191, 8192, 8193, 10239, 10240, 10241, 40000])
def test_speciation_stream(nb, syn, oracle, n):
    """nu = 1: every lineage speciates once."""
    desc = dict(kind=0, speciation_probability=1.0, width=n, height=1, deme=1)
    g = nb.simulate(1.0, syn.to_scenario(desc), 5)
    c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice=10, min_round_events=1 << 20,
                        step_slice_max=1024)
    assert len(g.speciation) == n and same_stream(g.speciation, c.speciation)
    assert g.biodiversity == c.biodiversity


def test_duplicates_share_their_event_time(nb, syn, oracle):
    """A small world in one long round: most speciations are reported by many
    lineages that have met and not merged yet."""
    desc = dict(kind=0, speciation_probability=0.01, width=60, height=50, deme=4)
    g = nb.simulate(0.01, syn.to_scenario(desc), 5, nb.CUDA(step_slice=1000))
    c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice=1000, min_round_events=1 << 20,
                        step_slice_max=1024)
    t = g.speciation["event_time"]
    assert len(t) > 8192 and len(np.unique(t)) < len(t) // 4
    assert same_stream(g.speciation, c.speciation) and g.biodiversity == c.biodiversity


def test_batch_of_many_simulations(nb, syn, oracle):
    n = 300
    descs = [dict(kind=0, speciation_probability=0.5, width=40 + s % 7, height=1, deme=1) for s in range(n)]
    g = nb.simulate_batch([syn.to_scenario(d) for d in descs], [0.5] * n, list(range(n)), nb.CUDA(), collect=True)
    assert sum(len(o.speciation) for o in g) > 8192
    for s in (0, 1, 6, 255, 256, 257, 299):
        c = oracle.simulate(descs[s], s, mode=oracle.MODE_CANONICAL, step_slice=10, min_round_events=1 << 20,
                            step_slice_max=1024)
        assert same_stream(g[s].speciation, c.speciation), s


@pytest.mark.parametrize("batch", [False, True])
def test_dispersal_stream(nb, syn, oracle, batch):
    desc = dict(kind=0, speciation_probability=0.02, width=40, height=30, deme=2)
    algo = nb.CUDA(report_dispersal=True)
    if batch:
        g = nb.simulate_batch([syn.to_scenario(desc)] * 2, [0.02, 0.03], [5, 6], algo, collect=True)[0]
    else:
        g = nb.simulate(0.02, syn.to_scenario(desc), 5, algo)
    c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice=10, min_round_events=1 << 20,
                        step_slice_max=1024, report_dispersal=True, dispersal_cap=1 << 20)
    assert same_stream(g.speciation, c.speciation)
    assert len(g.dispersal) == len(c.dispersal) > 50000
    want = c.dispersal[packed_order(c.dispersal)]
    for f in ("gref", "prior_time", "event_time", "x", "y", "index", "tx", "ty", "tindex"):
        assert np.array_equal(g.dispersal[f], want[f]), f
    assert not g.dispersal["pad"].any() and not g.dispersal["pad2"].any() and not g.speciation["pad"].any()
    # the interleaving: calls alternate between the kinds in time order
    at = {"s": 0, "d": 0}
    last = 0.0
    for kind, count in g.delivery:
        e = (g.speciation if kind == "s" else g.dispersal)[at[kind]:at[kind] + count]
        at[kind] += count
        assert e["event_time"][0] >= last
        last = e["event_time"][-1]
    assert (at["s"], at["d"]) == (len(g.speciation), len(g.dispersal))


@pytest.mark.parametrize("shift", [0, 20, 33])
def test_references_beyond_the_sorted_digits(nb, syn, oracle, shift):
    """Lineages that share their places from the start report the same events
    under references that differ in their low digits or only above them (the
    host settles the latter)."""
    desc = dict(kind=0, speciation_probability=0.01, width=20, height=7, deme=1)
    n = 600
    lins = np.zeros(n, dtype=nb.LINEAGE_DTYPE)
    u = syn.splitmix64(3, 2 * n)
    lins["x"] = u[:n] % np.uint64(20)
    lins["y"] = u[n:] % np.uint64(7)
    lins["gref"] = np.arange(n, 0, -1, dtype=np.uint64) << np.uint64(shift)
    with nb.Simulation(syn.to_scenario(desc), 0.01, nb.CUDA(report_dispersal=True, step_slice=60)) as sim:
        g = sim.resume(lins, 0.0, 5)
    c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, lineages=lins, step_slice=60, min_round_events=1 << 20,
                        step_slice_max=1024, report_dispersal=True, dispersal_cap=1 << 20)
    assert same_stream(g.speciation, c.speciation)
    assert len(g.dispersal) == len(c.dispersal) > 10000
    want = c.dispersal[packed_order(c.dispersal)]
    t = want["event_time"]
    assert (t[1:] == t[:-1]).sum() > 1000
    for f in ("gref", "prior_time", "event_time", "x", "y", "index", "tx", "ty", "tindex"):
        assert np.array_equal(g.dispersal[f], want[f]), f
