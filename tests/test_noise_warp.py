"""WrappingNoise targets found by a whole warp, at the edges of its lane
groups (octaves around powers of two, more than a warp of them), with more
rejections than one batch of targets, and with every way a lineage reaches it
(single runs, batches with the resident kernel, both samplers): the oracle's
canonical schedule bit for bit.  The shortened lattice wrap is compared with
the oracle's full division on the host, too."""
import numpy as np
import pytest

from test_gpu_parity import same_stream
from test_wrapping_noise import wn_desc

M32 = 0xFFFFFFFF

CASES = {
    "octaves_1": (1, 0.5, 2.0),
    "octaves_2": (2, 0.5, 2.0),
    "octaves_3": (3, 0.5, 2.0),
    "octaves_17": (17, 0.5, 2.0),
    "octaves_32": (32, 0.5, 2.0),
    "octaves_33": (33, 0.5, 2.0),
    "octaves_65": (65, 0.4, 2.0),
    "many_rejections": (2, 0.03, 3.0),
    "many_rejections_16": (16, 0.06, 3.0),
    "own_cell_rejections": (4, 0.7, 0.3),
    "full": (5, 1.0, 0.3),
}


@pytest.mark.gpu
@pytest.mark.parametrize("sampler", ["poisson", "exp"])
@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_matches_oracle(nb, syn, oracle, name, batch, sampler):
    octaves, coverage, sigma = CASES[name]
    desc = wn_desc(oracle, 0.05, 4, coverage, 0.07, 0.6, octaves, (M32 - 9, 300, 40, 30), sigma)
    algo = nb.CUDA(event_time_sampler=sampler, resident=batch)

    def run():
        if batch:
            return nb.simulate_batch([syn.to_scenario(desc)] * 2, [0.05, 0.1], [5, 6], algo, collect=True)[0]
        return nb.simulate(0.05, syn.to_scenario(desc), 5, algo)

    try:
        c = oracle.simulate(desc, 5, mode=oracle.MODE_CANONICAL, step_slice=10, min_round_events=1 << 20,
                            step_slice_max=1024,
                            event_time_sampler=oracle.SAMPLER_EXP if sampler == "exp" else 0)
    except RuntimeError as e:
        # an isolated cell and a narrow dispersal: 2^20 targets in a row rejected
        assert name == "own_cell_rejections" and "status -6" in str(e)
        with pytest.raises(nb.NecsimError) as failed:
            run()
        assert failed.value.code == -11
        return
    g = run()
    assert g.steps == c.steps > 0
    assert same_stream(g.speciation, c.speciation)
    assert (g.n_rounds, g.n_dedup, g.time) == (c.n_rounds, c.n_dedup, c.time)


@pytest.mark.parametrize("octaves", [1, 22, 40])
@pytest.mark.parametrize("corner", [(0, 0), (M32 - 20, M32 - 20), (M32 - 20, 5)])
def test_host_noise_at_the_lattice_edges(nb, syn, oracle, octaves, corner):
    """Lattice points below zero, at the period and, with many octaves, of
    periods beyond 2^53."""
    desc = wn_desc(oracle, 0.5, 11, 0.5, 0.9, 0.9, octaves, corner + (41, 41), 2.0)
    o = nb.enumerate_origins(syn.to_scenario(desc))
    c = oracle.enumerate_origins(desc)
    assert 0 < len(c) < 41 * 41
    assert np.array_equal(o["x"], c["x"]) and np.array_equal(o["y"], c["y"])
