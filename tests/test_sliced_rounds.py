"""Batches whose rounds end in different launches: simulations of very
different sizes (10 to 1,024 events per lineage and round) share the step
kernel's launches, which run at most 128 events of a lineage; every simulation
keeps the oracle's canonical rounds, merges and events."""
import numpy as np
import pytest

from test_gpu_parity import same_stream

pytestmark = pytest.mark.gpu


def scenarios(kind, syn):
    sizes = [9000, 6000, 1, 30, 700, 1500, 128, 3000]
    if kind == "ns":
        return [dict(kind=0, speciation_probability=2e-3 * (1 + s % 3), width=n, height=1, deme=1)
                for s, n in enumerate(sizes)]
    if kind == "si":
        return [dict(kind=1, speciation_probability=2e-2, width=n, height=1, deme=1, meta_width=5000, meta_height=1,
                     meta_deme=1, migration_probability=0.05 + 0.05 * (s % 4)) for s, n in enumerate(sizes)]
    if kind == "ai":
        return [dict(kind=2, speciation_probability=1e-2, sigma=2.0 + s, sample=(3, 5, n, 1))
                for s, n in enumerate(sizes)]
    out = []
    for s, cell in enumerate((60, 40, 1, 3)):
        hab = syn.habitat_map(17, 13, 0.2, cell, 5 + s)
        out.append(dict(kind=3, speciation_probability=5e-3, width=17, height=13, habitat=hab,
                        dispersal=syn.dispersal_map(hab, 2.0)))
    return out * 3


@pytest.mark.parametrize("sampler", ["poisson", "exp"])
@pytest.mark.parametrize("resident", [False, True])
@pytest.mark.parametrize("kind", ["ns", "si", "ai", "se"])
def test_matches_oracle(nb, syn, oracle, kind, resident, sampler):
    descs = scenarios(kind, syn)
    nus = [d["speciation_probability"] for d in descs]
    seeds = list(range(40, 40 + len(descs)))
    got = nb.simulate_batch([syn.to_scenario(d) for d in descs], nus, seeds,
                            nb.CUDA(resident=resident, event_time_sampler=sampler), collect=True)
    assert sum(o.n_initial for o in got) > 9472  # the step kernel takes the first rounds
    for s, (d, o) in enumerate(zip(descs, got)):
        c = oracle.simulate(d, seeds[s], mode=oracle.MODE_CANONICAL, step_slice=10, min_round_events=1 << 20,
                            step_slice_max=1024, event_time_sampler=oracle.SAMPLER_EXP if sampler == "exp" else 0)
        assert same_stream(o.speciation, c.speciation), s
        assert (o.steps, o.n_rounds, o.n_dedup, o.time) == (c.steps, c.n_rounds, c.n_dedup, c.time), s


def test_pause_mid_round(nb, syn, oracle):
    descs = scenarios("ns", syn)
    for pause in (33.0, 500.25):
        got = nb.simulate_batch([syn.to_scenario(d) for d in descs], [d["speciation_probability"] for d in descs],
                                list(range(8)), nb.CUDA(), pause_before=pause, collect=True)
        for s, d in enumerate(descs):
            c = oracle.simulate(d, s, mode=oracle.MODE_CANONICAL, step_slice=10, min_round_events=1 << 20,
                                step_slice_max=1024, pause_before=pause)
            assert same_stream(got[s].speciation, c.speciation), s
            assert (got[s].steps, got[s].n_rounds, got[s].n_dedup, got[s].n_remaining) == \
                   (c.steps, c.n_rounds, c.n_dedup, c.n_remaining), s


def test_round_watchdog_counts_rounds_not_launches(nb, syn):
    descs = scenarios("ns", syn)
    args = ([syn.to_scenario(d) for d in descs], [d["speciation_probability"] for d in descs], list(range(8)))
    need = max(o.n_rounds for o in nb.simulate_batch(*args, nb.CUDA()))
    again = nb.simulate_batch(*args, nb.CUDA(max_rounds=need))
    assert max(o.n_rounds for o in again) == need
    with pytest.raises(nb.NecsimError) as e:
        nb.simulate_batch(*args, nb.CUDA(max_rounds=1, rounds_per_graph=2))
    assert e.value.code == -5
