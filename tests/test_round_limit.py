"""necsim_args.max_rounds bounds the rounds that the host launches: rounds that
a lone lineage runs within one launch, and rounds in the resident kernel, are
counted by n_rounds and not by the limit."""
import pytest

from test_gpu_parity import same_stream

pytestmark = pytest.mark.gpu


def lone(nb):
    # one lineage of 100,000 expected events, ten to a round
    return nb.NonSpatial((1, 1), 1), 1e-5, dict(step_slice_max=10, min_round_events=1)


def test_free_rounds_are_not_counted(nb, syn):
    scenario, nu, kw = lone(nb)
    free = nb.simulate(nu, scenario, 3, nb.CUDA(**kw))
    assert free.n_rounds > 2000
    for limit in (free.n_rounds // 16, 2 ** 64 - 1):
        g = nb.simulate(nu, scenario, 3, nb.CUDA(max_rounds=limit, **kw))
        assert same_stream(g.speciation, free.speciation) and g.n_rounds == free.n_rounds


def test_resident_rounds_are_not_counted(nb, syn):
    scenario = nb.NonSpatial((1000, 1), 1)
    args = ([scenario] * 2, [1e-3, 2e-3], [3, 4])
    kw = dict(step_slice_max=10, min_round_events=1, resident=256)
    free = nb.simulate_batch(*args, nb.CUDA(**kw), collect=True)
    need = max(o.n_rounds for o in free)
    # each simulation is handed over within the first graphs of rounds
    got = nb.simulate_batch(*args, nb.CUDA(max_rounds=need // 2, **kw), collect=True)
    for a, b in zip(got, free):
        assert same_stream(a.speciation, b.speciation) and a.n_rounds == b.n_rounds


@pytest.mark.parametrize("kw", [dict(), dict(report_dispersal=True)])
def test_launched_rounds_are(nb, syn, kw):
    with pytest.raises(nb.NecsimError) as e:
        nb.simulate(1e-4, nb.NonSpatial((20, 20), 1), 3,
                    nb.CUDA(max_rounds=16, step_slice_max=1, step_slice=1, min_round_events=1, **kw))
    assert e.value.code == -5
