"""SpatiallyExplicit lineages that a warp steps event by event: a delta_t that
is no power of two, in batches whose last lineages run rounds of their own and
are interrupted when the launch's other work is done."""
import pytest

from test_chain import se
from test_gpu_parity import same_stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(), dict(step_slice=1, min_round_events=1, step_slice_max=40)])
@pytest.mark.parametrize("resident", [False, True])
@pytest.mark.parametrize("n_sims", [1, 2, 7])
def test_matches_oracle(nb, syn, oracle, n_sims, resident, kw):
    descs = []
    for s in range(n_sims):
        d = se(syn, 11, 9, 2.0, 0.02 / (1 + 2 * s), cell=1 + 2 * s)
        if s % 2:
            d["turnover_map"] = 0.1 + 3.0 * syn.unit(9 + s, 99, 4).reshape(9, 11)
        descs.append(d)
    got = nb.simulate_batch([syn.to_scenario(d) for d in descs], [d["speciation_probability"] for d in descs],
                            list(range(30, 30 + n_sims)), nb.CUDA(delta_t=3.0, resident=resident, **kw), collect=True)
    for s, (d, g) in enumerate(zip(descs, got)):
        c = oracle.simulate(d, 30 + s, mode=oracle.MODE_CANONICAL, delta_t=3.0,
                            **dict(dict(step_slice=10, min_round_events=1 << 20, step_slice_max=1024), **kw))
        assert same_stream(g.speciation, c.speciation), s
        assert (g.steps, g.n_rounds, g.n_dedup, g.time) == (c.steps, c.n_rounds, c.n_dedup, c.time), s


@pytest.mark.parametrize("kind", ["ns", "se"])
def test_workspaces_across_delta_t(nb, syn, oracle, kind):
    """Calls of hundreds of rounds with and without a lone-lineage form reuse
    one another's workspace, whose graph holds the kernels of one of them."""
    if kind == "ns":
        desc = dict(kind=0, speciation_probability=2e-3, width=40, height=30, deme=2)
    else:
        desc = se(syn, 31, 29, 1.5, 2e-3, cell=3)
    kw = dict(step_slice=1, min_round_events=1, step_slice_max=1)
    want = {dt: oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, delta_t=dt, **kw) for dt in (2.0, 3.0, 0.5)}
    assert min(c.n_rounds for c in want.values()) > 500
    for dt in (2.0, 3.0, 2.0, 0.5, 3.0, 3.0, 2.0):
        g = nb.simulate(2e-3, syn.to_scenario(desc), 5, nb.CUDA(delta_t=dt, **kw))
        c = want[dt]
        assert g.n_step_launches > 300  # a graph was built
        assert same_stream(g.speciation, c.speciation), dt
        assert (g.steps, g.n_rounds, g.n_dedup, g.time) == (c.steps, c.n_rounds, c.n_dedup, c.time), dt
