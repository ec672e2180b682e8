"""Order between the host's writes of device memory and the kernels that read
it.  The engines' streams are non-blocking: work on the default stream is
neither before nor after theirs, and cudaMemset and a host-to-device
cudaMemcpy may return before they have run."""
import os
import re

import numpy as np
import pytest

from test_event_sort import packed_order
from test_gpu_parity import same_stream

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "necsim-rust_b200", "csrc")


def calls(text, name):
    """The argument texts of every call of `name`."""
    for m in re.finditer(r"\b%s\(" % name, text):
        depth, at = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        yield text[m.end():at - 1]


@pytest.mark.parametrize("source", sorted(f for f in os.listdir(CSRC) if f.endswith((".cpp", ".cu"))))
def test_writes_of_device_memory_name_their_stream(source):
    with open(os.path.join(CSRC, source)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    assert not list(calls(text, "cudaMemset"))
    for args in calls(text, "cudaMemcpy"):
        assert "cudaMemcpyDeviceToHost" in args, args


@pytest.mark.gpu
def test_every_round_delivers_its_events(nb, syn, oracle):
    """Many rounds of few events each, delivered round by round."""
    desc = dict(kind=0, speciation_probability=5e-3, width=7, height=5, deme=3)
    kw = dict(step_slice=1, min_round_events=1, step_slice_max=1)
    for seed in range(3):
        g = nb.simulate(5e-3, syn.to_scenario(desc), seed, nb.CUDA(report_dispersal=True, **kw))
        c = oracle.simulate(desc, seed, mode=oracle.MODE_CANONICAL, report_dispersal=True, dispersal_cap=1 << 20, **kw)
        assert g.n_rounds == c.n_rounds > 50
        assert same_stream(g.speciation, c.speciation)
        assert g.n_dispersal == len(g.dispersal) == len(c.dispersal)
        # (a round's events are in order, and reach the reporter before the next round's)
        got, want = (d.dispersal[packed_order(d.dispersal)] for d in (g, c))
        for f in ("gref", "prior_time", "event_time", "x", "y", "index", "tx", "ty", "tindex"):
            assert np.array_equal(got[f], want[f]), f
