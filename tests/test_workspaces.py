"""Calls that follow one another reuse a finished call's workspace: every mix
of sizes, scenario kinds, samplers, empty and failing calls, threads and long
runs (whose rounds move into a graph) gives what each call gives alone."""
import threading

import numpy as np
import pytest

from test_gpu_parity import same_stream

pytestmark = pytest.mark.gpu


def calls(nb, syn):
    ns = nb.NonSpatial
    return [
        (ns((30, 20), 2), 0.01, dict()),
        (ns((1, 1), 1), 0.05, dict()),
        (ns((90, 70), 3), 0.02, dict()),
        (ns((30, 20), 2), 0.01, dict(event_time_sampler="exp")),
        (ns((30, 20), 2), 0.01, dict(report_dispersal=True)),
        (ns((8, 9), 2), 0.02, dict(step_slice=1, min_round_events=1)),  # hundreds of rounds: a graph
        (ns((31, 20), 2), 0.01, dict(dedup_factor_pct=400)),
        (nb.SpatiallyImplicit((40, 3), 2, (500, 1), 2, 0.2), 0.01, dict()),
        (nb.WrappingNoise(3, 0.0, 0.07, 0.5, 2, nb.Rectangle((0, 0), 9, 8), 2.0), 0.05, dict()),
        (nb.WrappingNoise(3, 0.6, 0.07, 0.5, 2, nb.Rectangle((0, 0), 70, 81), 2.0), 0.05, dict()),
        (nb.WrappingNoise(3, 0.4, 0.07, 0.5, 2, nb.Rectangle((0, 0), 9, 8), 2.0), 0.05, dict()),
    ]


def outcome(nb, call, seed):
    scenario, nu, kw = call
    return nb.simulate(nu, scenario, seed, nb.CUDA(**kw))


def same(a, b):
    return (same_stream(a.speciation, b.speciation)
            and (a.steps, a.n_rounds, a.n_dedup, a.time, a.n_initial, a.biodiversity, a.n_dispersal)
            == (b.steps, b.n_rounds, b.n_dedup, b.time, b.n_initial, b.biodiversity, b.n_dispersal))


def test_mixed_calls_repeat(nb, syn):
    todo = calls(nb, syn)
    first = [outcome(nb, c, 5 + k) for k, c in enumerate(todo)]
    order = np.random.RandomState(3).permutation(np.repeat(np.arange(len(todo)), 4))
    for k in order:
        if k % 4 == 0:  # a call that fails gives its workspace back to nobody
            with pytest.raises(nb.NecsimError):
                nb.simulate(1e-4, nb.NonSpatial((30, 20), 2), 1, nb.CUDA(max_rounds=2, step_slice=1, min_round_events=1))
        assert same(outcome(nb, todo[k], 5 + k), first[k]), k
    # against a batch of one, which has an engine of its own
    for k in (0, 1, 2, 5, 7, 9):
        scenario, nu, kw = todo[k]
        alone = nb.simulate_batch([scenario], [nu], [5 + k], nb.CUDA(**kw), collect=True)[0]
        assert same(alone, first[k]), k


def test_threads(nb, syn):
    todo = calls(nb, syn)[:6]
    first = [outcome(nb, c, 11 + k) for k, c in enumerate(todo)]
    bad = []

    def work(t):
        for r in range(6):
            k = (t + r) % len(todo)
            if not same(outcome(nb, todo[k], 11 + k), first[k]):
                bad.append((t, k))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
