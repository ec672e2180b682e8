"""A lineage without an event before the horizon leaves the allocation-free
round as it came: the caller's own coordinates, which the round does not check
against the scenario, in both samplers' forms."""
import numpy as np
import pytest

from test_zz_no_alloc import SCENARIOS, _round

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sampler", ["poisson", "exp"])
@pytest.mark.parametrize("scenario", sorted(SCENARIOS))
def test_unmoved_lineages_keep_their_coordinates(nb, syn, scenario, sampler):
    torch = pytest.importorskip("torch")
    desc, seed = SCENARIOS[scenario]
    struct = nb._scenario_struct(syn.to_scenario(desc), 1e-9)
    n = 300
    lins = np.zeros(n, dtype=nb.LINEAGE_DTYPE)
    lins["gref"] = np.arange(n)
    # inside and outside the scenario's extent, with indices beyond its demes
    lins["x"], lins["y"], lins["index"] = 7 * np.arange(n), np.arange(n) // 3, np.arange(n) % 11
    out, _, steps = _round(nb, torch, struct, nb.seed_from_u64(seed), lins, 0.0, 1.0, sampler)
    assert 50 < steps
    out = out[np.argsort(out["gref"])]
    still = out[out["last_event_time"] == 0.0]
    assert len(still) > 100
    for f in ("x", "y", "index"):
        assert np.array_equal(still[f], lins[f][still["gref"].astype(np.int64)]), f
