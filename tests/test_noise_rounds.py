"""WrappingNoise rounds on either side of the size at which they move from a
warp to a lane per lineage, and calls with cheap and with costly noise that
reuse one another's workspace (whose graph holds that size)."""
import numpy as np
import pytest

from test_gpu_parity import same_stream
from test_wrapping_noise import wn_desc

pytestmark = pytest.mark.gpu


def noise(oracle, octaves, coverage, width, height, nu=0.05):
    return wn_desc(oracle, nu, 4, coverage, 0.07, 0.6, octaves, (0xFFFFFFFF - 9, 300, width, height), 2.0)


def check(g, c):
    assert g.n_initial == c.n_initial and g.steps == c.steps > 0
    assert same_stream(g.speciation, c.speciation)
    assert (g.n_rounds, g.n_dedup, g.time) == (c.n_rounds, c.n_dedup, c.time)


def expect(oracle, desc, seed, sampler, **kw):
    return oracle.simulate(desc, seed, mode=oracle.MODE_CANONICAL, event_time_sampler=sampler == "exp",
                           **dict(dict(step_slice=10, min_round_events=1 << 20, step_slice_max=1024), **kw))


@pytest.mark.parametrize("sampler", ["poisson", "exp"])
@pytest.mark.parametrize("octaves,coverage,width,height", [
    (1, 1.0, 4500, 1), (1, 1.0, 4501, 1), (1, 1.0, 5000, 1), (1, 1.0, 5001, 1), (3, 1.0, 150, 100),
    (1, 0.5, 150, 160), (2, 0.7, 200, 140), (4, 0.3, 210, 150), (16, 0.5, 120, 100)])
def test_round_sizes(nb, syn, oracle, octaves, coverage, width, height, sampler):
    desc = noise(oracle, octaves, coverage, width, height)
    g = nb.simulate(0.05, syn.to_scenario(desc), 5, nb.CUDA(event_time_sampler=sampler))
    check(g, expect(oracle, desc, 5, sampler))


@pytest.mark.parametrize("resident", [False, True])
@pytest.mark.parametrize("sampler", ["poisson", "exp"])
def test_batches(nb, syn, oracle, sampler, resident):
    descs = [noise(oracle, o, c, w, 80, nu) for o, c, w, nu in
             ((1, 1.0, 70, 0.03), (2, 0.9, 90, 0.05), (1, 0.5, 60, 0.02), (5, 0.6, 1, 0.1))]
    got = nb.simulate_batch([syn.to_scenario(d) for d in descs], [d["speciation_probability"] for d in descs],
                            [3, 4, 5, 6], nb.CUDA(event_time_sampler=sampler, resident=resident), collect=True)
    assert sum(g.n_initial for g in got) > 10_000
    for s, (d, g) in enumerate(zip(descs, got)):
        check(g, expect(oracle, d, 3 + s, sampler))


def test_reused_workspaces(nb, syn, oracle):
    """Hundreds of rounds each, which move into a graph."""
    kw = dict(step_slice=1, min_round_events=1, step_slice_max=1)
    descs = [noise(oracle, o, c, 80, 100, 5e-3) for o, c in ((1, 1.0), (16, 0.9), (2, 1.0), (12, 0.8))]
    want = [expect(oracle, d, 5, "poisson", **kw) for d in descs]
    for k in (0, 1, 0, 2, 3, 1, 2):
        g = nb.simulate(5e-3, syn.to_scenario(descs[k]), 5, nb.CUDA(**kw))
        assert g.n_step_launches > 300  # a graph was built
        check(g, want[k])


def test_dispersal_events(nb, syn, oracle):
    desc = noise(oracle, 1, 0.9, 80, 80)
    g = nb.simulate(0.05, syn.to_scenario(desc), 5, nb.CUDA(report_dispersal=True))
    c = expect(oracle, desc, 5, "poisson", report_dispersal=True, dispersal_cap=1 << 20)
    assert same_stream(g.speciation, c.speciation)
    a = np.sort(g.dispersal, order=("event_time", "gref"))
    b = np.sort(c.dispersal, order=("event_time", "gref"))
    assert len(a) == len(b) > 50_000
    for f in ("gref", "prior_time", "event_time", "x", "y", "index", "tx", "ty", "tindex"):
        assert np.array_equal(a[f], b[f]), f
