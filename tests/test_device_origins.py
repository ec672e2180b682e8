"""The origin lineages that the device writes (origins.cu) against the host's
enumeration in the reference's order: a run paused at time 0 executes nothing
and returns its origins."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M32 = 0xFFFFFFFF


def cells(syn):
    hab = syn.habitat_map(13, 9, 0.4, 20, 11)
    hab[0, :3] = 0  # empty cells at both ends of the prefix sums
    hab[-1, -4:] = 0
    return dict(kind=3, width=13, height=9, habitat=hab, dispersal=syn.dispersal_map(hab, 1.5))


def noise(coverage, sample):
    return dict(kind=5, noise_seed=3, coverage=coverage, scale=0.07, persistence=0.5, octaves=3, sample=sample,
                sigma=2.0)


CASES = {
    "grid_one": lambda syn: dict(kind=0, width=1, height=1, deme=1),
    "grid_demes": lambda syn: dict(kind=0, width=257, height=31, deme=7),
    "grid_local": lambda syn: dict(kind=1, width=1009, height=3, deme=2, meta_width=50, meta_height=2, meta_deme=3,
                                   migration_probability=0.2),
    "plane_wrapping": lambda syn: dict(kind=2, sigma=2.0, sample=(M32 - 3, M32 - 5, 37, 41)),
    "circle_0": lambda syn: dict(kind=2, sigma=2.0, radius=0, centre_x=5, centre_y=9),
    "circle_1": lambda syn: dict(kind=2, sigma=2.0, radius=1, centre_x=0, centre_y=0),
    "circle_wrapping": lambda syn: dict(kind=2, sigma=2.0, radius=100, centre_x=3, centre_y=M32 - 7),
    "cells": cells,
    "noise_none": lambda syn: noise(0.0, (10, 20, 9, 8)),
    "noise_some": lambda syn: noise(0.37, (M32 - 40, M32 - 3, 131, 77)),
    "noise_all": lambda syn: noise(1.0, (10, 20, 33, 8)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_origins_match_the_host(nb, syn, name):
    scenario = syn.to_scenario(CASES[name](syn))
    want = nb.enumerate_origins(scenario)
    with nb.Simulation(scenario, 0.5, nb.CUDA()) as sim:
        got = sim.simulate(1, pause_before=0.0)
        assert (got.n_initial, got.steps) == (len(want), 0)
        left = got.remaining if got.remaining is not None else want[:0]
        if len(want):
            # the same list handed back as resumed lineages
            again = sim.resume(want, 0.0, 1, pause_before=0.0).remaining
            assert np.array_equal(np.sort(again, order="gref"), np.sort(left, order="gref"))
    want = np.sort(want, order="gref")
    for f in ("gref", "x", "y", "index", "last_event_time"):
        assert np.array_equal(left[f], want[f]), f


def test_batch_segments(nb, syn):
    """Simulations of different sizes in one batch start from their own origins."""
    descs = [dict(kind=0, width=w, height=3, deme=d) for w, d in ((1, 1), (300, 2), (7, 5), (1, 2))]
    scenarios = [syn.to_scenario(d) for d in descs]
    one = [nb.simulate(0.05, s, 3 + k) for k, s in enumerate(scenarios)]
    many = nb.simulate_batch(scenarios, [0.05] * 4, [3, 4, 5, 6], nb.CUDA(), collect=True)
    for a, b in zip(one, many):
        assert np.array_equal(a.speciation, b.speciation)
        assert (a.n_initial, a.steps) == (b.n_initial, b.steps)


def test_batch_of_noise(nb, syn):
    """Many small samples, some of them without a habitable location."""
    scenarios = [syn.to_scenario(noise((0.0, 0.4, 1.0, 0.7)[s % 4], (M32 - 3 + 5 * s, 7 * s, 1 + s % 5, 1 + s % 9)))
                 for s in range(61)]
    got = nb.simulate_batch(scenarios, [0.05] * 61, list(range(61)), nb.CUDA(), collect=True)
    assert [g.n_initial for g in got] == [len(nb.enumerate_origins(s)) for s in scenarios]
    for s in (0, 1, 2, 3, 31, 58, 59, 60):
        one = nb.simulate(0.05, scenarios[s], s)
        assert np.array_equal(one.speciation, got[s].speciation) and one.steps == got[s].steps
    none = nb.simulate_batch(scenarios[:61:4], [0.05] * 16, list(range(16)), nb.CUDA(), collect=True)
    assert all((g.n_initial, g.steps) == (0, 0) for g in none)


@pytest.mark.parametrize("kind", ["circles", "maps"])
def test_batch_of_prefix_sums(nb, syn, kind):
    """Circles of many radii beside rectangles, and maps of many shapes: each
    simulation reads its own part of the batch's prefix sums."""
    if kind == "circles":
        descs = [dict(kind=2, sigma=2.0, radius=s % 7, centre_x=3 * s, centre_y=M32 - s) if s % 5 else
                 dict(kind=2, sigma=2.0, sample=(s, s, 1 + s, 2)) for s in range(23)]
    else:
        descs = []
        for s in range(9):
            hab = syn.habitat_map(1 + 2 * s, 1 + s % 4, 0.4, 5, 11 + s)
            hab.flat[0] = 1
            descs.append(dict(kind=3, width=hab.shape[1], height=hab.shape[0], habitat=hab,
                              dispersal=syn.dispersal_map(hab, 1.5)))
    scenarios = [syn.to_scenario(d) for d in descs]
    got = nb.simulate_batch(scenarios, [0.05] * len(descs), list(range(len(descs))), nb.CUDA(), collect=True)
    for s, g in enumerate(got):
        one = nb.simulate(0.05, scenarios[s], s)
        assert np.array_equal(one.speciation, g.speciation) and one.steps == g.steps
        assert g.n_initial == len(nb.enumerate_origins(scenarios[s]))
