"""Rounds without an event: a resume whose lineages last moved long before the
resume time passes through hundreds of them, and is not taken for hung before
64 graphs of rounds (1,024 by default), however the rounds are launched."""
import numpy as np
import pytest

from test_gpu_parity import same_stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("report_dispersal", [False, True])
@pytest.mark.parametrize("idle", [100, 200, 700, 1000])
def test_resume_long_after_the_last_events(nb, syn, oracle, idle, report_dispersal):
    desc = dict(kind=0, speciation_probability=0.05, width=9, height=5, deme=2)
    kw = dict(step_slice=10, step_slice_max=10, min_round_events=1)
    resume_time = idle * 10 / 0.5  # a round is ten events of the rate 1 / 2
    lins = np.zeros(60, dtype=nb.LINEAGE_DTYPE)
    lins["gref"] = np.arange(60)
    lins["x"], lins["y"], lins["index"] = np.arange(60) % 9, np.arange(60) // 9 % 5, np.arange(60) // 45
    with nb.Simulation(syn.to_scenario(desc), 0.05, nb.CUDA(report_dispersal=report_dispersal, **kw)) as sim:
        g = sim.resume(lins, resume_time, 3)
    c = oracle.simulate(desc, 3, mode=oracle.MODE_CANONICAL, lineages=lins, resume_time=resume_time, **kw)
    assert same_stream(g.speciation, c.speciation) and len(c.speciation) > 0
    assert (g.steps, g.n_rounds, g.n_dedup) == (c.steps, c.n_rounds, c.n_dedup)
    assert c.n_rounds > idle
    assert (g.speciation["event_time"] > resume_time).all()


def test_many_more_idle_rounds_time_out(nb, syn):
    """Far more idle rounds than the limit still end in the watchdog's error."""
    desc = dict(kind=0, speciation_probability=0.05, width=3, height=1, deme=1)
    lins = np.zeros(2, dtype=nb.LINEAGE_DTYPE)  # (one lineage alone runs rounds in one launch)
    lins["x"] = lins["gref"] = np.arange(2)
    with nb.Simulation(syn.to_scenario(desc), 0.05, nb.CUDA(step_slice_max=10, min_round_events=1)) as sim:
        with pytest.raises(nb.NecsimError) as e:
            sim.resume(lins, 5000 * 20.0, 3)
        assert e.value.code == -5
        assert sim.simulate(3).n_remaining == 0  # the context stays usable
